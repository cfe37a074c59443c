"""Householder re-orthogonalisation of walkers whose reflectors are the identity: real walkers
that are columns of the identity (every reflector, a molecular-orbital basis) and real square
blocks (the last reflector).  The kernel leaves such a column's turn before its barriers, so
its zero tau must still be ordered before the threads that form Q read it: every copy of a
walker among several hundred gives the same bits."""
import numpy as np
import pytest

from miniafqmc_b200.synthetic import Config, make_system

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("nel", [33, 48, 64])
@pytest.mark.parametrize("extra", [0, 40])
def test_identity_reflectors(nel, extra):
    from miniafqmc_b200.afqmc import AfqmcSys
    nmo, nw = nel + extra, 300
    s = make_system(Config(nmo, nel, 8, 0.3, 7, dt=0.01, nwalk=nw), build_vakbl=False)
    W = np.zeros((nw, 2, nmo, nel), complex)
    W[:, 0] = np.eye(nmo, nel)                       # H = 1 for every column
    rng = np.random.default_rng(nel)
    sq = rng.normal(size=(nmo, nel))
    sq[nel:] = 0.0                                   # a square real block: H = 1 for the last
    W[:, 1] = sq
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=(W, s.initial_walkers(nw)[1]))
    want = np.linalg.qr(sq)[0]
    tol = 16 * nmo * nel * EPS * np.linalg.cond(sq)
    for _ in range(5):
        e.set_walkers(W, s.initial_walkers(nw)[1])
        e.orthogonalize()
        Q = e.get_walkers()[0]
        assert np.array_equal(Q[:, 0], W[:, 0])
        assert np.all(Q[:, 1] == Q[0, 1])
        assert np.max(np.abs(Q[0, 1] - want)) <= tol
    e.close()
