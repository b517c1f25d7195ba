"""Query sums of the cluster kernels for primes below 2^62: fewer queries than a CTA has warps, as many, more,
and sizes that end before the table's, against the oracle."""
import pytest

import cuckoo_b200 as cb
import helpers as h

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lg", [15, 16])
@pytest.mark.parametrize("J", [1, 16, 17, 40])
def test_query_sums(lg, J):
    ps, n, d = cb.prime_range(7, 2, bits=62), 70, 3
    qs = [(n - j % 60, 2 * n + 3 * j) for j in range(J)]
    with cb.Engine(0) as eng:
        eng.set_transform_lg(lg)
        got = eng.residues(ps, n, d, qs)
    for p, row in zip(ps, got):
        assert [int(x) for x in row] == h.oracle_residues(p, n, d, qs)
