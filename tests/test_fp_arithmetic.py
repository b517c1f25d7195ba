"""The double-precision modular arithmetic (fparith.cuh) against whole numbers, at the edges of its
stated ranges, and the kernels' phase code in the default geometries for primes below 2^50 against
the oracle, with every butterfly's bound checked (CF_CHECK_BOUNDS).  All on the CPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

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
    L.fp_power_small.argtypes = [ctypes.c_double, ctypes.c_int, ctypes.c_double]
    L.fp_power_small.restype = ctypes.c_double
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
    for k in range(33):
        assert int(fp.fp_power_small(float(p // 3), k, float(p))) % p == pow(p // 3, k, p)


@pytest.mark.parametrize("lg,R,nmax", [
    (14, 5, 70), (11, 3, 1025), (10, 3, 1024), (10, 2, 600), (9, 3, 512), (9, 2, 257), (9, 2, 512),
    (8, 2, 255), (8, 1, 256), (8, 1, 129), (7, 1, 128), (7, 1, 65),
])
def test_default_geometries_match_oracle(fp, lg, R, nmax):
    p = h.oracle_primes(0, 1)[0]
    for model, d in ((0, 3), (1, 2)):
        qs = [(nmax, 2 * nmax + 1), (max(d, nmax // 3), nmax)]
        qn, qM = (ctypes.c_int * 2)(*[q[0] for q in qs]), (ctypes.c_int * 2)(*[q[1] for q in qs])
        out = (ctypes.c_uint64 * 2)()
        rc = fp.emu_fp_geo(ctypes.c_uint64(p), nmax, d, model, qn, qM, 2, out, lg, R)
        assert rc == 0 and [int(x) for x in out] == h.oracle_residues(p, nmax, d, qs, model)
