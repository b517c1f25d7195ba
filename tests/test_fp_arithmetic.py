"""The double-precision modular arithmetic (fparith.cuh) against whole numbers, at the edges of its
stated ranges, and the kernels' phase code in the default geometries against the oracle, with every
double-precision butterfly's bound checked (CF_CHECK_BOUNDS).  All on the CPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import cuckoo_b200 as cb
import helpers as h

PRIMES = [1125899865948161, h.oracle_primes(0, 1)[0], 4293918721, 97]  # the top of the list, a library prime, a tiny one
_dp = ctypes.POINTER(ctypes.c_double)
_up = ctypes.POINTER(ctypes.c_uint64)


@pytest.fixture(scope="module")
def fp(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("emu_fp") / "libemufp.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", os.path.join(h.EMU_DIR, "emu_fp.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.fp_products.argtypes = [_dp, _dp, ctypes.c_double, ctypes.c_long, _dp]
    L.fp_reductions.argtypes = [_dp, ctypes.c_double, ctypes.c_long, _dp, _up]
    L.fp_power_fast.argtypes = [ctypes.c_double, ctypes.c_int, ctypes.c_double]
    L.fp_power_fast.restype = ctypes.c_double
    return L


def edge_values(p, a, rng):
    """Whole numbers up to a p in size: the ends, the multiples of p / 2 and their neighbours, random ones."""
    top = int(a * p)
    v = [0, 1, -1, top, -top]
    for k in range(1, int(2 * a) + 1):
        v += [k * p // 2 + e for e in (-1, 0, 1)] + [-(k * p // 2) + e for e in (-1, 0, 1)]
    v += [int(x) for x in rng.integers(-top, top, 300, endpoint=True)]
    return sorted({x for x in v if -top <= x <= top})


@pytest.mark.parametrize("p", PRIMES)
@pytest.mark.parametrize("a,b", [(4.0, 0.5), (2.0, 1.0), (0.75, 0.75), (1.0, 1.0)])
def test_products_are_exact_and_bounded(fp, p, a, b):
    rng = np.random.default_rng(p % 1000)
    xs, ws = edge_values(p, a, rng), edge_values(p, b, rng)
    x = np.array([u for u in xs for _ in range(40)], dtype=np.float64)
    w = np.array([ws[int(i)] for i in rng.integers(0, len(ws), len(x))], dtype=np.float64)
    for k, u in enumerate((-1, 0, 1, -2)):  # each x also meets the ends of w's range
        w[k::40] = ws[u]
    out = np.zeros(len(x))
    fp.fp_products(x.ctypes.data_as(_dp), w.ctypes.data_as(_dp), float(p), len(x), out.ctypes.data_as(_dp))
    bound = (0.5 + a * b / 4) * p + 1
    for u, v, r in zip(x, w, out):
        assert r == int(r) and (int(r) - int(u) * int(v)) % p == 0 and abs(r) <= bound, (u, v, r)


@pytest.mark.parametrize("p", PRIMES)
def test_reductions(fp, p):
    xs = np.array(edge_values(p, 8.0, np.random.default_rng(5)), dtype=np.float64)
    xs = xs[np.abs(xs) < 2.0 ** 53]
    out, canon = np.zeros(len(xs)), np.zeros(len(xs), dtype=np.uint64)
    fp.fp_reductions(xs.ctypes.data_as(_dp), float(p), len(xs), out.ctypes.data_as(_dp), canon.ctypes.data_as(_up))
    for u, r, c in zip(xs, out, canon):
        assert (int(r) - int(u)) % p == 0 and abs(r) <= 0.51 * p and int(c) == int(u) % p, (u, r, c)
    for k in list(range(33)) + [1000, 16384]:
        assert int(fp.fp_power_fast(float(p // 3), k, float(p))) % p == pow(p // 3, k, p)


@pytest.mark.parametrize("lg,R,nmax,bits", [
    (14, 5, 70, 50), (11, 3, 1025, 50), (10, 3, 1024, 50), (10, 2, 600, 50), (9, 3, 512, 50), (9, 2, 257, 50), (9, 2, 512, 50),
    (8, 2, 255, 50), (8, 1, 256, 50), (8, 1, 129, 50), (7, 1, 128, 50), (7, 1, 65, 50),
    (13, 3, 90, 62), (12, 3, 80, 62), (11, 2, 1025, 62), (10, 2, 600, 62), (9, 2, 512, 62), (8, 2, 129, 62), (7, 1, 128, 62),
])
def test_default_geometries_match_oracle(fp, lg, R, nmax, bits):
    p = cb.prime_range(0, 1, bits=bits)[0]
    for model, d in ((0, 3), (1, 2)):
        qs = [(nmax, 2 * nmax + 1), (max(d, nmax // 3), nmax)]
        assert run_geo(fp, p, nmax, d, model, qs, lg, R, 0) == h.oracle_residues(p, nmax, d, qs, model)


def run_geo(fp, p, nmax, d, model, qs, lg, R, JC):
    J = len(qs)
    qn, qM = (ctypes.c_int * J)(*[q[0] for q in qs]), (ctypes.c_int * J)(*[q[1] for q in qs])
    out = (ctypes.c_uint64 * J)()
    rc = fp.emu_fp_geo(ctypes.c_uint64(p), nmax, d, model, qn, qM, J, out, lg, R, JC)
    assert rc == 0, rc
    return [int(x) for x in out]


@pytest.mark.parametrize("lg,R,bits", [(7, 1, 50), (12, 4, 50), (7, 1, 62), (12, 3, 62)])
@pytest.mark.parametrize("JC", [1, 2, 3, 7])
def test_queries_in_batches(fp, lg, R, bits, JC):
    """More queries than shared memory holds partial sums for: the batches' folds give the same residues."""
    p = cb.prime_range(2, 1, bits=bits)[0]
    n = 60
    qs = [(n - 7 * k, 2 * n + k) for k in range(7)]
    assert run_geo(fp, p, n, 3, 0, qs, lg, R, JC) == h.oracle_residues(p, n, 3, qs)
