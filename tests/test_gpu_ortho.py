"""Householder re-orthogonalisation (FP64 form) in shared memory and, for blocks that do not
fit, in global memory; CholeskyQR (mixed form).  Column counts around the 16, 32 and 64 column
lanes, square blocks, zero and already triangular columns.  Reference: numpy's QR of the
conjugated walkers (LAPACK's Householder signs).  Both are backward stable: Q within
c N n eps cond(W) of each other."""
import numpy as np
import pytest

from miniafqmc_b200.synthetic import Config, make_system

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def system(nmo, nel, cplx):
    """Without Vakbl: (nmo nel)^2 entries per spin."""
    return make_system(Config(nmo, nel, 8, 0.3, 7, dt=0.01, nwalk=3, complex_trial=cplx,
                              complex_chol=cplx), build_vakbl=False)


@pytest.mark.parametrize("nmo,nel", [(1, 1), (5, 5), (40, 15), (40, 16), (300, 17), (33, 32),
                                     (64, 33), (190, 64), (250, 64), (64, 64)])
def test_householder_matches_lapack(nmo, nel):
    from miniafqmc_b200.afqmc import AfqmcSys
    nw = 3
    s = system(nmo, nel, True)
    rng = np.random.default_rng(nmo + nel)
    W = rng.normal(size=(nw, 2, nmo, nel)) + 1j * rng.normal(size=(nw, 2, nmo, nel))
    W[1, 0] = np.triu(W[1, 0])                       # nothing below the diagonal
    W[1, 0, np.arange(nel), np.arange(nel)] = 1.0 + np.arange(nel)   # and real pivots: H = 1
    Wd = s.initial_walkers(nw)[1]
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=(W, Wd))
    e.orthogonalize()
    Q = e.get_walkers()[0]
    for w in range(nw):
        for sp in range(2):
            want, R = np.linalg.qr(W[w, sp].conj())
            tol = 16 * nmo * nel * EPS * np.linalg.cond(W[w, sp])
            assert np.max(np.abs(Q[w, sp].conj() - want)) <= tol
            assert np.max(np.abs(Q[w, sp].conj().T @ Q[w, sp] - np.eye(nel))) <= 16 * nmo * nel * EPS
    e.close()


@pytest.mark.parametrize("nmo,nel", [(8, 8), (40, 16), (40, 20), (72, 32), (64, 36), (96, 48), (72, 64)])
def test_cholqr_spans_the_same_space(nmo, nel):
    from miniafqmc_b200.afqmc import AfqmcSys, AFQ_PREC_MIXED
    nw = 3
    s = system(nmo, nel, False)
    rng = np.random.default_rng(nmo + nel)
    W, Wd = s.initial_walkers(nw)
    W = W + 0.1 / np.sqrt(nmo) * (rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape))
    e = AfqmcSys(s, nw, precision=AFQ_PREC_MIXED, use_vakbl=False, walkers=(W, Wd))
    e.orthogonalize()
    Q = e.get_walkers()[0]
    for w in range(nw):
        for sp in range(2):
            want, R = np.linalg.qr(W[w, sp])
            d = np.diag(R) / np.abs(np.diag(R))      # positive diagonal
            cond = np.linalg.cond(W[w, sp])
            assert np.max(np.abs(Q[w, sp] - want * d)) <= 64 * nmo * nel * EPS * cond ** 2
    e.close()
