"""The first launch over a freshly allocated workspace, with more primes than SMs, so several CTAs
share an SM and their warps drift apart between barriers: every residue equals the one computed in
launches of one CTA per SM.  Table words read before their writer's barrier show here (and only
here: a later launch finds the same words from the launch before)."""
import numpy as np
import pytest

import cuckoo_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count,bits", [(24, 600, 50), (200, 600, 50), (700, 600, 50), (1100, 296, 50), (2048, 256, 50), (2500, 300, 50),
                                          (1100, 296, 62)])
def test_first_launch_with_several_ctas_per_sm(n, count, bits):
    primes = cb.prime_range(0, count, bits=bits)
    queries = [(n, 2 * n), (n // 2, n)]
    with cb.Engine(0) as eng:
        first = eng.residues(primes, n, 3, queries)
    with cb.Engine(0) as eng:
        want = np.concatenate([eng.residues(primes[a:a + 100], n, 3, queries) for a in range(0, count, 100)])
    assert np.array_equal(first, want)
