"""Every geometry index that tune_set took stays accepted, and each index is its own geometry."""
import pytest

import cuckoo_b200 as cb


@pytest.mark.parametrize("lg,count", [(8, 1), (10, 3), (11, 4), (12, 4), (13, 3), (14, 2), (15, 4), (16, 2)])
def test_indices(lg, count):
    v = [tuple(g.values()) for g in cb.tune_variants(lg)]
    assert len(v) >= count and len(set(v)) == len(v)


@pytest.mark.gpu
@pytest.mark.parametrize("lg,n", [(11, 1500), (12, 2500)])
def test_indices_agree(lg, n):
    primes = cb.prime_range(0, 150)
    with cb.Engine(0) as eng:
        want = eng.residues(primes, n, 3, [(n, 2 * n)])
        for k in range(len(cb.tune_variants(lg))):
            eng.tune_set(lg, k)
            assert (eng.residues(primes, n, 3, [(n, 2 * n)]) == want).all()
