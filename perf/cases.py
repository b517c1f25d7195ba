"""The work a user of this engine has it do, as measurable cases: residues of N_bad(n, M) modulo
primes, through the public entry points of cuckoo_b200.py.

A case names an entry point ("kind"), the table size n, the choices per item d, the model, the
number of primes B and of queries J, and the prime list:

    host    Engine.residues           host buffers in and out (the CLI's batch, single.py)
    device  Engine.residues_async     device buffers on the current stream
    build   Engine.tables_async and Tables.query_async   a serving chunk built, asked once, freed
    query   Tables.query_async        queries answered from resident tables
    uneven  Uneven.launch / results   many (n, M, d) instances in one captured graph

    primes: 50 or 62 (the two fixed lists), 32 (the library CLI's primes for that table)

A program keeps one engine per device, so the cases share one; primes and query sizes are made from
the seed, resident tables and captured batches belong to a state.
"""
import functools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuckoo-failure_b200"))
import cuckoo_b200 as cb  # noqa: E402
import uneven as ub  # noqa: E402

PRIME_SPAN = 1024  # batches start at one of this many places of the fixed list


def _case(name, kind, n, B, J=1, d=3, model=0, primes=50, **more):
    return dict({"kind": kind, "n": n, "B": B, "J": J, "d": d, "model": model, "primes": primes}, **({"name": name} if name else {}), **more)


def listed():
    return [
        # the smallest useful call: one residue of a small table, launch and set-up latency
        _case("tiny_n24_b1", "host", 24, 1),
        # `single -n 200 -M 400 -d 3`: the library CLI's 32-bit primes, all in one call
        _case("single_n200_lib152", "host", 200, 152, primes=32),
        # a small parameter sweep: one table, nine (n, M) queries, the replacement model
        _case("sweep_n512_j9_b40", "host", 512, 40, J=9, model=1),
        # a serving chunk built for a new (d, n) range and asked once
        _case("build_n1000_b256", "build", 1000, 256, J=4, d=2, F=4000),
        # requests answered from a resident chunk
        _case("query_n2048_b148_j8", "query", 2048, 148, J=8, F=8192),
        # an odd size well below its transform length, a serving chunk of primes by the plain path
        _case("plain_n2500_b256_j4", "host", 2500, 256, J=4, d=4),
        # the same path with the shorter prime list below 2^62
        _case("wide_n3000_b128", "host", 3000, 128, primes=62),
        # n = 4096, M = 8192, four waves of primes (the benchmark's second configuration)
        _case("n4096_b592", "device", 4096, 592),
        # many instances of uneven size in one captured batch
        _case("uneven_24x4096", "uneven", 4096, 24, stride=16),
        # a large table on every SM, a size between transform lengths
        _case("n10000_b148", "device", 10000, 148),
        # a few primes of a deep table with several queries (the end of a prime list)
        _case("n12500_b4_j8", "host", 12500, 4, J=8),
        # a table above n = 16384: one prime per cluster of SMs
        _case("cluster_n18000_b24", "device", 18000, 24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "host", "host", "device", "device", "device", "build", "query", "uneven", "deep"])
    d, model = rng.choice([2, 3, 3, 4]), rng.choice([0, 0, 0, 1])
    if kind == "uneven":
        n = rng.choice([4096, _log_int(rng, 64, 1024)])
        return _case(None, kind, n, rng.randint(6, 24), stride=rng.randint(16, 64), model=model)
    if kind == "build":
        n = _log_int(rng, 64, 1500)
        return _case(None, kind, n, _log_int(rng, 16, 256 if n <= 1024 else 148), J=rng.randint(1, 8), d=d, model=model, F=rng.randint(2 * n, 4 * n))
    if kind == "query":
        n = _log_int(rng, 64, 2048)
        return _case(None, kind, n, _log_int(rng, 16, 256 if n <= 1024 else 148), J=_log_int(rng, 1, 32), d=d, model=model, F=rng.randint(2 * n, 4 * n))
    if kind == "deep":  # the largest tables, few primes
        if rng.random() < 0.5:
            return _case(None, "device", rng.randint(16385, 18000), rng.randint(1, 24), J=rng.randint(1, 2), d=d)
        return _case(None, "host", rng.randint(10000, 12500), rng.randint(1, 16), J=rng.randint(1, 8), d=d, model=model)
    n = _log_int(rng, 16, 10000)
    B = _log_int(rng, 1, 592 if n <= 1024 else 148)
    primes = rng.choice([50, 50, 50, 50, 62, 32 if n <= 512 else 50])
    if primes == 62:
        n = min(n, 3000)
    return _case(None, kind, n, min(B, 148) if primes != 50 else B, J=rng.choice([1, 1, 1, rng.randint(2, 9)]), d=d, model=model, primes=primes)


@functools.lru_cache(maxsize=None)
def _engine():
    return cb.Engine(0)


@functools.lru_cache(maxsize=None)
def _prime_list(bits):
    return cb.prime_range(0, PRIME_SPAN + 600, bits=bits)


def _queries(case, rng):
    """J queries: the table's own n first, then sizes below it; M between 1.5 and 4 times n."""
    n, lo = case["n"], max(case["d"], min(8, case["n"]))
    top = case.get("F") or 4 * n
    out = []
    for j in range(case["J"]):
        m = n if j == 0 else _log_int(rng, lo, n)
        out.append((m, min(top, max(m + 1, case["d"], int(m * rng.uniform(1.5, 4.0))))))
    return out


def _primes(case, rng, queries):
    B = case["B"]
    if case["primes"] == 32:  # the library CLI's primes of the table (at M = 2n), a run of them
        got = cb.lib_primes(case["n"], 2 * case["n"], case["d"], case["model"])
        at = rng.randrange(max(0, len(got) - B) + 1)
        return got[at:at + B]
    at = rng.randrange(PRIME_SPAN)
    return _prime_list(case["primes"])[at:at + B]


def _inputs(case, seed):
    rng = random.Random(seed * 1000003 + case["n"])
    q = _queries(case, rng)
    return _primes(case, rng, q), q


def _instances(case):
    """The case's own instances, within an octave of sizes; a seed chooses which of their primes are
    planned (every stride-th)."""
    return ub.instances(case["B"], seed=case["B"], n_lo=case["n"] // 2 + 1, n_hi=case["n"])


def prepare(case, seed):
    eng, kind = _engine(), case["kind"]
    s = dict(case, eng=eng)
    if kind == "uneven":
        s["handle"] = eng.uneven(_instances(case), model=case["model"], first=random.Random(seed).randrange(16), stride=case["stride"])
        return s
    primes, s["queries"] = _inputs(case, seed)
    s["list"] = np.array(primes, dtype=np.uint64)
    B, J = len(primes), len(s["queries"])
    if kind != "host":
        s["primes_dev"] = torch.tensor(primes, dtype=torch.int64, device="cuda")
        s["out"] = torch.zeros((B, J), dtype=torch.int64, device="cuda")
    if kind == "query":
        s["tables"] = eng.tables(primes, case["n"], case["F"], case["d"], model=case["model"])
    return s


def run(s):
    eng, kind, d, model = s["eng"], s["kind"], s["d"], s["model"]
    if kind == "host":
        return eng.residues(s["list"], s["n"], d, s["queries"], model=model).view(np.int64)
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "uneven":
        s["handle"].launch(stream)
        return [r.view(np.int64) for r in s["handle"].results(stream)]
    out = s["out"]
    if kind == "device":
        eng.residues_async(s["primes_dev"].data_ptr(), out.shape[0], s["n"], d, s["queries"], out.data_ptr(), stream, model=model)
    elif kind == "query":
        s["tables"].query_async(s["queries"], out.data_ptr(), stream)
    else:  # build: on the stream, asked in stream order, and freed in stream order
        t = eng.tables_async(s["list"], s["n"], s["F"], d, model=model, stream_ptr=stream)
        t.query_async(s["queries"], out.data_ptr(), stream)
        t.close()
    return out


def _table_products(n):
    """Modular products of one prime's table: two length-n convolutions a step (a forward and an
    inverse transform and the product of spectra each), and the stage factors of its entries."""
    return 2.0 * n * n * (math.log2(max(n, 2)) + 1) + 4.0 * n * n


def work(case):
    """Operations: a modular product counts as two (a multiplication and a reduction's).  Bytes: what
    a pass reads from and writes to its caller; for resident tables the rows the queries read."""
    n, B, J = case["n"], case["B"], case["J"]
    if case["kind"] == "uneven":
        prod = outs = 0.0
        for m, M, d in _instances(case):
            k = -(-cb.need(m, M, d, case["model"]) // case["stride"])
            outs += k
            prod += k * m * m / 2.0
        for (d, i), ks in ub.tables(_instances(case), lambda a, b, c: cb.need(a, b, c, case["model"]), stride=case["stride"]).items():
            prod += _table_products(max(_instances(case)[k][0] for k in ks))
        return {"bytes": 16.0 * outs, "flops": 2.0 * prod}
    sizes = [q[0] for q in _queries(case, random.Random(1))]
    rows = sum(m * m / 2.0 for m in sizes)
    io = 8.0 * B * (1 + J)
    if case["kind"] == "query":  # all queries read the same triangle: once
        return {"bytes": io + 8.0 * B * n * n / 2.0, "flops": 2.0 * B * rows}
    keep = 8.0 * B * n * n / 2.0 if case["kind"] == "build" else 0.0
    return {"bytes": io + keep, "flops": 2.0 * B * (_table_products(n) + rows)}


def _exact_nbad(nmax, queries, d, model):
    """N_bad(n, M) as whole numbers by the O(n^3) recurrence over the suffix table V[p][v]."""
    binom = math.comb

    def g(v):
        return v ** d if model else binom(v, d)

    V = [[0] * (nmax + 1) for _ in range(nmax + 1)]
    S = [[0] * (nmax + 1) for _ in range(nmax + 1)]
    for v in range(nmax):
        for vp in range(v, nmax):
            if v >= 1:
                S[vp][v] = sum(binom(vp - w - 1, vp - v) * binom(vp, w) * V[v][w] for w in range(v) if V[v][w])
        gv = g(v)
        pw = [1]
        for _ in range(nmax):
            pw.append(pw[-1] * gv)
        for p in range(v + 1, nmax + 1):
            V[p][v] = binom(p - 1, v) * pw[p] - sum(
                binom(p - q - 1, p - v - 1) * binom(p, q) * pw[p - q] * S[v][q] for q in range(1, v + 1) if S[v][q])
    out = []
    for n, M in queries:
        Q = g(M)
        tot = 0
        for q in range(1, n + 1):
            inner = sum(binom(M - w - 1, M - q) * binom(M, w) * V[q][w] for w in range(q) if V[q][w])
            tot += binom(n, q) * Q ** (n - q) * inner
        out.append(tot)
    return out


def exact(case, seed):
    if case["kind"] == "uneven" or case["n"] > 64:
        return None
    primes, queries = _inputs(case, seed)
    vals = _exact_nbad(case["n"], queries, case["d"], case["model"])
    return np.array([[v % int(p) for v in vals] for p in primes], dtype=np.int64)
