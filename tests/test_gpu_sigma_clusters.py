"""Sigma on clusters of one to eight CTAs per 32 walkers: Cholesky and walker counts on both sides
of each cluster size.  Fields given by the caller; X and the hybrid weight against numpy."""
import numpy as np
import pytest

from miniafqmc_b200.synthetic import Config, make_system

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("nchol,nw", [(1, 1), (32, 33), (33, 64), (64, 700), (65, 700), (129, 31),
                                      (129, 700), (257, 40), (256, 1030), (600, 130)])
def test_sigma(nchol, nw):
    from miniafqmc_b200.afqmc import AfqmcSys
    s = make_system(Config(12, 3, nchol, 0.3, 7, dt=0.01, nwalk=nw, complex_trial=True,
                           complex_chol=True), build_vakbl=False)
    rng = np.random.default_rng(nchol + nw)
    W, Wd = s.initial_walkers(nw)
    W = W + 0.1 * (rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape))
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=(W, Wd))
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    vb = e.copy_out("vbias")
    x = rng.normal(size=(nchol, nw))
    e.sigma_from(x)
    assert np.array_equal(e.copy_out("X"), x + 1j * vb)
    terms = -1j * vb * (x + 0.5j * vb)
    assert np.all(np.abs(e.copy_out("hybridW") - terms.sum(0))
                  <= 8 * (np.sqrt(nchol) + 4) * EPS * np.abs(terms).sum(0) + 1e-300)
    e.close()
