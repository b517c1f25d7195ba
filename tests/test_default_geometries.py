"""The default geometries' phase code on the CPU, where test_fp_arithmetic.py does not run them: against the
oracle, with the transforms' bounds and the ends of shared memory and workspace checked."""
import ctypes
import os
import subprocess

import pytest

import cuckoo_b200 as cb
import helpers as h


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("emu_default") / "libemudefault.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", os.path.join(h.EMU_DIR, "emu_default.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("lg,R,n,bits", [
    (4, 1, 16, 50), (5, 1, 31, 50), (6, 1, 64, 50), (12, 3, 83, 50), (12, 4, 83, 50), (13, 4, 70, 50),
    (4, 1, 16, 62), (5, 1, 31, 62), (6, 1, 64, 62), (14, 4, 40, 62)])
@pytest.mark.parametrize("model,d", [(0, 3), (1, 2)])
def test_against_the_oracle(emu, lg, R, n, bits, model, d):
    p = cb.prime_range(3, 1, bits=bits)[0]
    qs = [(n, 2 * n + 1), (max(d, n // 3), n), (n - 1, n)]
    J = len(qs)
    qn, qM = (ctypes.c_int * J)(*[q[0] for q in qs]), (ctypes.c_int * J)(*[q[1] for q in qs])
    out = (ctypes.c_uint64 * J)()
    assert emu.emu_default(ctypes.c_uint64(p), n, d, model, qn, qM, J, out, lg, R) == 0
    assert [int(x) for x in out] == h.oracle_residues(p, n, d, qs, model)
