// How the resident-table query kernel (table_query.cuh) splits a launch over the device.  Host code.
#pragma once
#include <algorithm>

namespace cfb {

constexpr int TQ_THREADS = 256, TQ_WARPS = TQ_THREADS / 32, TQ_PER_SM = 2;
constexpr int TQ_ROWS = 16, TQ_K = 8, TQ_COLS = 32 * TQ_K;  // a warp's tile: rows, columns per lane, columns
constexpr int TQ_CLUSTER = 4;                               // CTAs per prime at most
// How a launch splits a prime's work, tiles times queries:
//   S  CTAs in a cluster, which share the tiles: the number up to TQ_CLUSTER whose waves of resident CTAs
//      leave the least idle (their shares are equal, so a launch lasts waves / S), with a block of rows
//      for every warp.  Four at most: beside a plain rebuild that fills 96 SMs, clusters of eight find
//      fewer places in what each GPC has left (served requests with n in 513 .. 2048: p50 10.6 ms, p99
//      44; with four 5.9 and 28).
//   G  groups of queries (every G-th of the sorted sizes), each a cluster of its own that reads the
//      triangle again: as many as still run in one wave, while a warp has a tile of one query to do.
//   W  queries a warp takes of a tile at a time: all of the group's where every warp has two tiles or
//      more (the tile's entries are then read once), else two, or one where that takes fewer rounds (a
//      tile of one query lasts 0.65 of one of two).
// Without groups, and with all queries of a tile on one warp, few primes with many queries left most
// SMs idle, and small tables most warps.  us per launch without and with them (in front a CTA per
// prime and query, the form before tiles): n = 100, one prime, 256 queries 26, 894, 27; n = 16, 148
// primes, 256 queries 343, 655, 100; n = 500, 16 primes, 64 queries 402, 316, 109; n = 2048, 2 primes,
// 64 queries 1573, 2230, 218.
struct TQSplit {
    int S, G, W;
};
inline long tq_tiles(int n) {  // of a triangle of n rows: the blocks before the last, and the last
    constexpr long per = TQ_COLS / TQ_ROWS;  // blocks of rows that a column of tiles lasts
    const long m = (n - 1) / TQ_ROWS, k = m / per, r = m % per;
    return per * k * (k + 1) / 2 + r * (k + 1) + (n + TQ_COLS - 1) / TQ_COLS;
}
inline TQSplit tq_split(int B, int J, int nmax, int sms) {
    const long cap = (long)TQ_PER_SM * (sms > 0 ? sms : 1), T = tq_tiles(nmax);
    auto waves = [&](long ctas) { return (ctas + cap - 1) / cap; };
    TQSplit x{1, 1, 1};
    for (int c = 2; c <= TQ_CLUSTER && nmax >= TQ_ROWS * TQ_WARPS * c / 2; ++c)
        if (waves((long)B * c) * x.S < waves((long)B * x.S) * c) x.S = c;
    const long warps = (long)x.S * TQ_WARPS;
    x.G = (int)std::max(1l, std::min({(long)J, cap / ((long)B * x.S), T * J / warps}));
    const long Jg = (J + x.G - 1) / x.G;
    auto rounds = [&](long w) { return (T * ((Jg + w - 1) / w) + warps - 1) / warps; };
    x.W = T >= 2 * warps ? (int)Jg : 65 * rounds(1) < 100 * rounds(2) ? 1 : 2;
    return x;
}
}  // namespace cfb
