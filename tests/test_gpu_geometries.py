"""The default geometry follows the number of primes (few per SM: more threads per prime): on both
sides of each length's limit, at the ends of the length's sizes, the residues equal the oracle's for
the first and the last prime and agree prime by prime between the two geometries."""
import numpy as np
import pytest
import torch

import cuckoo_b200 as cb
import helpers as h

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,per_sm", [(65, 0), (128, 0), (129, 2), (256, 2), (257, 2), (512, 2), (513, 2), (1024, 2), (1025, 0), (2049, 1)])
@pytest.mark.parametrize("model", [0, 1])
def test_few_and_many_primes_agree(n, per_sm, model):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    few = max(per_sm, 1) * sms
    primes = cb.prime_range(0, few + 1)
    d, qs = (3, [(n, 2 * n), (n // 2, n)]) if model == 0 else (2, [(n, 3 * n), (n // 3, n)])
    with cb.Engine(0) as eng:
        a = eng.residues(primes[:few], n, d, qs, model=model)
        b = eng.residues(primes, n, d, qs, model=model)  # one prime above the limit
        one = eng.residues(primes[-1:], n, d, qs, model=model)
    assert np.array_equal(a, b[:few]) and np.array_equal(one[0], b[-1])
    if n <= 1025:
        for row, p in ((a[0], primes[0]), (b[-1], primes[-1])):
            assert [int(x) for x in row] == h.oracle_residues(p, n, d, qs, model)


@pytest.mark.parametrize("n,J,bits", [(2100, 1600, 50), (1100, 3400, 50), (4100, 700, 62)])
def test_more_queries_than_one_batch(n, J, bits):
    """Launches whose queries' partial sums do not fit shared memory at once sum them in batches."""
    primes = cb.prime_range(0, 2, bits=bits)
    qs = [(n - k % n // 2, 2 * n + k % 50) for k in range(J)]
    with cb.Engine(0) as eng:
        got = eng.residues(primes, n, 3, qs)
        want = np.concatenate([eng.residues(primes, n, 3, qs[a:a + 250]) for a in range(0, J, 250)], axis=1)
        with pytest.raises(cb.EngineError) as e:
            eng.residues(primes, n, 3, qs * 8)
        assert e.value.code == cb.CF_ERR_UNSUPPORTED
    assert np.array_equal(got, want)
