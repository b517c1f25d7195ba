"""Which kernel the engine launches for a call, from its host code on a fake CUDA runtime."""
import pytest

import cuckoo_b200 as cb
import fake_device as fd


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fd.link(tmp_path_factory.mktemp("fake"))


@pytest.mark.parametrize("other", [0, 1])
def test_geometry_follows_the_engines_device(fake, other):
    """An engine counts its own device's SMs, whichever device is current when it is called."""
    with fd.on(fake) as L:
        L.fake_set_sms(0, 148)
        L.fake_set_sms(1, 40)
        primes = cb.prime_range(0, 100)
        with cb.Engine(1 - other) as eng:
            for n in (4096, 1000, 500, 200):
                threads = []
                for current in (1 - other, other):
                    L.cudaSetDevice(current)
                    eng.residues(primes, n, 3, [(n, 2 * n)])
                    dev, grid, block, _ = fd.launches(L)[-1]
                    assert dev == 1 - other and grid == 100
                    threads.append(block)
                assert threads[0] == threads[1], n


@pytest.mark.parametrize("n", [200, 500, 1000, 4096])
@pytest.mark.parametrize("B,cap", [(100, 0), (148, 0), (296, 0), (592, 0), (592, 100)])
def test_autotune_record_describes_what_ran(fake, n, B, cap):
    """The geometries of an autotuning record are those its launches had, the default's among them."""
    with fd.on(fake) as L:
        L.fake_set_sms(0, 148)
        with cb.Engine(0) as eng:
            assert L.cf_engine_set_max_ctas(eng._h, cap) == 0
            fd.launches(L)
            rec = eng.autotune(n, 2 * n, 3, B)
            ran = fd.launches(L)
            per = len(ran) // len(rec["variants"])
            assert [v["threads"] for v in rec["variants"]] == [block for _, _, block, _ in ran[::per]]
            eng.tune_set(rec["lg"], 0)
            eng.residues(cb.prime_range(0, B), n, 3, [(n, 2 * n)])
            assert fd.launches(L)[0][2] == rec["variants"][0]["threads"]
