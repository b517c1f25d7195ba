"""Resident-table queries where a launch splits them in groups of queries, and tiles over warps by one, two
or all of a group's queries (table_split.hpp): equal to the residues of a direct build."""
import numpy as np
import pytest

import cuckoo_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count,J,model,d", [
    (3, 1, 256, 1, 1), (16, 2, 37, 0, 3), (40, 3, 5, 0, 2), (100, 1, 256, 0, 3), (100, 150, 9, 1, 2), (130, 1, 300, 0, 4),
    (257, 7, 64, 0, 3), (600, 1, 50, 1, 2), (1100, 2, 31, 0, 3), (1100, 90, 3, 0, 3),
])
def test_grouped_queries(n, count, J, model, d):
    F = 4 * n + d
    primes = cb.prime_range(3, count)
    rng = np.random.default_rng(J)
    queries = [(int(m), int(rng.integers(max(m + 1, d), F, endpoint=True))) for m in rng.integers(1, n, J, endpoint=True)]
    queries[J // 2] = (n, F)
    with cb.Engine(0) as eng:
        with eng.tables(primes, n, F, d, model=model) as tab:
            got = tab.query(queries)
        want = eng.residues(primes, n, d, queries, model=model)
    assert np.array_equal(got, want)
