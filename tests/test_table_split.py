"""The split of a resident-table query launch (table_split.hpp) over the device: no warp is left with much
more than its share of the (tile, query) work while others have none, whatever the numbers of primes,
queries and rows."""
import ctypes
import subprocess

import pytest

import helpers as h

SRC = r"""
#include "%s/cuckoo-failure_b200/csrc/table_split.hpp"
extern "C" void split(int B, int J, int n, int sms, int* out) {
    const cfb::TQSplit x = cfb::tq_split(B, J, n, sms);
    out[0] = x.S, out[1] = x.G, out[2] = x.W, out[3] = (int)cfb::tq_tiles(n);
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    (d / "s.cpp").write_text(SRC % h.ROOT)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", str(d / "s.cpp"), "-o", str(d / "s.so")], check=True)
    L = ctypes.CDLL(str(d / "s.so"))

    def f(B, J, n, sms=148):
        out = (ctypes.c_int * 4)()
        L.split(B, J, n, sms, out)
        return list(out)

    return f


@pytest.mark.parametrize("n", [1, 16, 17, 100, 200, 500, 1000, 2048, 16384])
@pytest.mark.parametrize("B", [1, 2, 16, 64, 148, 256, 1000])
def test_shares(split, n, B):
    for J in (1, 2, 3, 8, 33, 64, 255, 256):
        S, G, W, T = split(B, J, n)
        assert T == sum(-(-min(q, n) // 256) for q in range(16, n + 16, 16))
        assert 1 <= S <= 4 and 1 <= G <= J and 1 <= W <= J
        assert G == 1 or B * G * S <= 2 * 148  # more groups than one wave holds only read the triangles again
        Jg = -(-J // G)
        longest = -(-(T * -(-Jg // W)) // (8 * S)) * W * -(-(B * G * S) // (2 * 148))  # tiles of one query, one after another
        warps = min(8 * 2 * 148, 8 * 4 * J * B)  # on the device at once, and in four CTAs a prime and query
        assert longest <= 3 * -(-(T * J * B) // warps) + 2, (S, G, W, longest)
