"""One-launch propagation of small systems (FP64 form): orbital counts around the 64 rows of
a pass, up to the largest it takes, columns that do not fill the last group of eight, Taylor
orders from zero, real and complex Hamiltonians.  Reference: the chain in numpy.  Each product
carries about N roundings of its terms."""
import dataclasses

import numpy as np
import pytest

from conftest import tiny_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmo,nel,nw,order,cplx", [(5, 1, 3, 6, True), (31, 4, 2, 6, False),
                                                   (63, 5, 3, 3, True), (64, 8, 2, 6, False),
                                                   (65, 9, 2, 1, True), (111, 3, 2, 6, True),
                                                   (112, 13, 1, 0, False), (113, 4, 1, 6, False)])
def test_chain_matches_numpy(nmo, nel, nw, order, cplx):
    from miniafqmc_b200.afqmc import AfqmcSys
    s = tiny_system(complex_trial=cplx, complex_chol=cplx, nmo=nmo, nel=nel, nchol=9)
    s = dataclasses.replace(s, cfg=dataclasses.replace(s.cfg, taylor_order=order))
    rng = np.random.default_rng(nmo)
    W, Wd = s.initial_walkers(nw)
    W = W + 0.3 / np.sqrt(nmo) * (rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape))
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=(W, Wd))
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    e.sigma(3, 1)
    e.get_vHS()
    V = e.copy_out("vHS")
    e.propagate()
    got = e.get_walkers()[0]
    P = s.Propg1
    for w in range(nw):
        Vw = V[:, w].reshape(nmo, nmo)
        for sp in range(2):
            T = P @ W[w, sp]
            S = T.copy()
            size = np.abs(P) @ np.abs(W[w, sp])
            term = size
            for k in range(1, order + 1):
                T = (1j / k) * (Vw @ T)
                S = S + T
                term = np.abs(Vw) @ term / k
                size = size + term
            bound = 16 * (order + 2) * nmo * 2.0 ** -53 * (np.abs(P) @ size)
            assert np.all(np.abs(got[w, sp] - P @ S) <= bound)
    e.close()
