"""Queries from resident tables at the edges of the query kernel's tiles (16 rows, 256 columns, pairs of
queries, 256 queries a launch, one to eight CTAs per prime): equal to the residues of a direct build."""
import numpy as np
import pytest

import cuckoo_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count,J,model,d", [
    (1, 3, 1, 1, 2), (2, 3, 2, 1, 1), (5, 3, 3, 0, 3), (16, 4, 1, 0, 3), (17, 4, 2, 1, 2), (20, 4, 3, 0, 18),
    (255, 2, 3, 0, 4), (256, 2, 1, 0, 2), (257, 2, 2, 1, 3), (258, 400, 3, 0, 3), (513, 5, 257, 0, 3), (1040, 20, 33, 1, 2),
])
def test_queries_at_tile_edges(n, count, J, model, d):
    F = max(4 * n, d + 2)
    primes = cb.prime_range(11, count)
    rng = np.random.default_rng(n)
    queries = [(n, F)]
    while len(queries) < J:
        m = int(rng.integers(1, n, endpoint=True))
        queries.append((m, int(rng.integers(max(m + 1, d), F, endpoint=True))))
    with cb.Engine(0) as eng:
        with eng.tables(primes, n, F, d, model=model) as tab:
            got = tab.query(queries)
        want = eng.residues(primes, n, d, queries, model=model)
    assert np.array_equal(got, want)
