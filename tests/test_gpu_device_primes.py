"""Primes on the device are not read by the host: those of 2^50 and above among them give the residues
of cf_residues too, which reads its primes, with queries, geometry and chunks of either kernel."""
import numpy as np
import pytest

import cuckoo_b200 as cb
import helpers as h

pytestmark = pytest.mark.gpu


def _device(eng, primes, n, queries, model=0, graph=False):
    import torch

    d_p = torch.tensor(primes, dtype=torch.int64, device="cuda")
    d_o = torch.zeros((len(primes), len(queries)), dtype=torch.int64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    if graph:
        with eng.batch_graph(d_p.data_ptr(), len(primes), n, 3, queries, d_o.data_ptr(), model=model) as g:
            g.launch(st)
            g.status(st)
    else:
        eng.residues_async(d_p.data_ptr(), len(primes), n, 3, queries, d_o.data_ptr(), st, model=model)
    return d_o.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("n,J,model", [(12, 1, 0), (40, 5, 1), (100, 2, 0), (200, 1, 1), (300, 9, 0), (700, 2, 0), (1500, 1, 0), (2500, 2, 1)])
@pytest.mark.parametrize("graph", [False, True])
def test_primes_of_both_lists(n, J, model, graph):
    primes = [p for pair in zip(cb.prime_range(0, 3), cb.prime_range(5, 3, bits=62)) for p in pair]
    queries = [(n - j, 2 * n + j) for j in range(J)]
    with cb.Engine(0) as eng:
        got = _device(eng, primes, n, queries, model, graph)
        assert np.array_equal(got, eng.residues(primes, n, 3, queries, model=model))
        if n <= 200:
            assert [[int(x) for x in r] for r in got[:2]] == [h.oracle_residues(p, n, 3, queries, model) for p in primes[:2]]


def test_all_primes_wide_in_chunks_and_clusters():
    wide = cb.prime_range(0, 40, bits=62)
    with cb.Engine(0) as eng:
        want = eng.residues(wide, 250, 3, [(250, 500)])
        assert np.array_equal(_device(eng, wide, 250, [(250, 500)]), want)
        eng.set_max_ctas(7)  # chunks share one workspace, each with its second launch
        assert np.array_equal(_device(eng, wide, 250, [(250, 500)]), want)
        eng.set_prime_bits(62)  # one launch for all
        assert np.array_equal(_device(eng, wide + cb.prime_range(0, 2), 250, [(250, 500)])[:40], want)
    for lg in (14, 15, 16):  # one CTA with 32 entries a thread, clusters of 4, of 16
        with cb.Engine(0) as eng:
            eng.set_transform_lg(lg)
            assert np.array_equal(_device(eng, [cb.prime_range(0, 1)[0], wide[0]], 120, [(120, 250)]),
                                  eng.residues([cb.prime_range(0, 1)[0], wide[0]], 120, 3, [(120, 250)]))
