"""Walkers to and from the caller's memory: the device rearranges the reference's layout and
large sets pass through a pinned ring in chunks of 2 MB (from 8 MB on, several host threads).
Whatever the size, what comes back is what went in, bit for bit."""
import numpy as np
import pytest

from conftest import tiny_system

pytestmark = pytest.mark.gpu


# 32 KB per walker: below, at and just past the ring's threshold, whole and ragged chunks,
# fewer and more chunks than slots; an odd shape
@pytest.mark.parametrize("nmo,nel,nw", [(64, 16, 255), (64, 16, 256), (64, 16, 257),
                                        (64, 16, 384), (64, 16, 700), (37, 5, 1601)])
@pytest.mark.parametrize("mixed", [False, True])
def test_round_trip_is_exact(nmo, nel, nw, mixed):
    from miniafqmc_b200.afqmc import AfqmcSys, AFQ_PREC_FP64, AFQ_PREC_MIXED
    if mixed and (nmo % 8 or nel % 4):
        pytest.skip("mixed form: rows of whole 16 bytes")
    s = tiny_system(complex_trial=False, complex_chol=False, nmo=nmo, nel=nel, nchol=8)
    rng = np.random.default_rng(nw)
    W, Wd = s.initial_walkers(nw)
    W = W + rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape)
    Wd = Wd + rng.normal(size=Wd.shape)
    e = AfqmcSys(s, nw, precision=AFQ_PREC_MIXED if mixed else AFQ_PREC_FP64, use_vakbl=False,
                 walkers=(W, Wd))
    for _ in range(2):
        V, Vd = e.get_walkers()
        assert np.array_equal(V, W) and np.array_equal(Vd, Wd)
        W, Wd = W[::-1].copy(), Wd[::-1].copy()
        e.set_walkers(W, Wd)
    assert np.array_equal(e.get_walkers()[0], W)
    e.close()
