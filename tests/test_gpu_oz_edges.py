"""Digit products at the edges of their chunks and splits, against long double: several Cholesky
and walker chunks of the exchange (chunks that start inside a row tile), K splits that bound the
int32 sums, Vakbl with ragged rows; and the error in the 2-norm, which a lost digit pair would
raise 20 to 100 times.  Bounds: the digits' error is 2^-56 sqrt(K) of the scales; where a column
reaches 2^-6 of them (else the FP64 pipe computes it) that is 2^-50 sqrt(K) of its largest entry, at
the sizes here below 2^-50 of the 2-norm, and the partial sums and the result round to 2^-53 a few
times: 2^-49.  A propagation chain is eight products: 2^-48."""
import dataclasses

import numpy as np
import pytest

from conftest import tiny_system

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
LD = np.clongdouble


def walkers(s, nw, seed=11):
    rng = np.random.default_rng(seed)
    W, Wd = s.initial_walkers(nw)
    return W + 0.3 / np.sqrt(s.N) * (rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape)), Wd


def norm_error(got, want):
    return float(np.linalg.norm((got - want).astype(complex)) / np.linalg.norm(want.astype(complex)))


# 200 vectors of 27: 88 vectors a chunk, which ends 72 rows into a tile; 300 walkers of 64: two
# walker chunks; 41 vectors of 33 in complex form
@pytest.mark.parametrize("nmo,nel,nchol,nw,cplx", [(33, 27, 200, 64, False), (64, 64, 40, 300, False),
                                                   (48, 33, 141, 70, True)])
def test_exchange_in_chunks(nmo, nel, nchol, nw, cplx):
    from miniafqmc_b200.afqmc import AfqmcSys
    s = tiny_system(complex_trial=cplx, complex_chol=cplx, nmo=nmo, nel=nel, nchol=nchol)
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=walkers(s, nw))
    assert e.digit_products()["exchange"]
    e.calculate_mixed_density_matrix()
    e.calculate_energy("chol")
    got = e.copy_out("energy_parts")[:, 2]
    G = e.copy_out("Gc").T.reshape(nw, 2, nel, nmo)
    assert e.digit_products_redone()["exchange"] == 0
    for w in range(0, nw, 13):
        T = [s.Lh[:, sp].astype(LD) @ G[w, sp].astype(LD).T for sp in range(2)]
        ek = sum(0.5 * (t * t.transpose(0, 2, 1)).sum() for t in T)
        size = sum((np.abs(t) ** 2).sum() for t in T)
        assert abs(got[w] - ek.real) <= 2.0 ** -49 * size
    e.close()


@pytest.mark.parametrize("nmo,nel,nchol,nw,cplx", [(64, 16, 70, 33, False), (50, 11, 130, 40, True),
                                                   (128, 32, 60, 16, False)])
def test_errors_in_the_2_norm(nmo, nel, nchol, nw, cplx):
    from miniafqmc_b200.afqmc import AfqmcSys
    s = tiny_system(complex_trial=cplx, complex_chol=cplx, nmo=nmo, nel=nel, nchol=nchol)
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=walkers(s, nw))
    assert e.digit_products()["vbias"] and e.digit_products()["coulomb"]
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    G = e.copy_out("Gc").astype(LD)
    assert norm_error(e.copy_out("vbias"), s.SpvnT.todense().astype(LD) @ G) <= 2.0 ** -49
    e.calculate_energy("chol")
    c = s.Lh.reshape(nchol, -1).astype(LD) @ G
    ej = 0.5 * (c * c).sum(0)
    size = (np.abs(c) ** 2).sum(0)
    assert np.all(np.abs(e.copy_out("energy_parts")[:, 1] - ej.real) <= 2.0 ** -48 * size)
    assert not any(e.digit_products_redone().values())
    e.close()


@pytest.mark.parametrize("nmo,nel,nw,cplx,vhs", [(130, 20, 185, False, True), (121, 5, 300, True, False)])
def test_vhs_and_propagation_in_the_2_norm(nmo, nel, nw, cplx, vhs):
    from miniafqmc_b200.afqmc import AfqmcSys
    from miniafqmc_b200.synthetic import CSR
    nchol = 96
    s = dataclasses.replace(tiny_system(complex_trial=cplx, complex_chol=cplx, nmo=nmo, nel=nel,
                                        nchol=nchol))
    rng = np.random.default_rng(4)
    A = rng.normal(size=(nmo * nmo, nchol)) * (rng.random((nmo * nmo, nchol)) < 0.7) * 2e-3
    s.Spvn = CSR.from_scipy(A if not cplx else A * (1 + 0.5j))
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=walkers(s, nw))
    on = e.digit_products()
    assert on["propagate"] and (on["vHS"] or not vhs)
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    e.sigma_from(rng.normal(size=(nchol, nw)))
    X = e.copy_out("X")
    e.get_vHS()
    V = e.copy_out("vHS")
    rows = rng.choice(nmo * nmo, 400, replace=False)
    want = s.Spvn.to_scipy()[rows].toarray().astype(LD) @ X.astype(LD)
    assert norm_error(V[rows], want) <= 2.0 ** -49
    W0 = e.get_walkers()[0]
    e.propagate()
    W1 = e.get_walkers()[0]
    P = s.Propg1.astype(LD)
    for w in (0, nw // 2, nw - 1):
        Vw = V[:, w].reshape(nmo, nmo).astype(LD)
        for sp in range(2):
            T = P @ W0[w, sp].astype(LD)
            S = T.copy()
            for k in range(1, 7):
                T = (1j / LD(k)) * (Vw @ T)
                S = S + T
            assert norm_error(W1[w, sp], P @ S) <= 2.0 ** -48
    assert not any(e.digit_products_redone().values())
    e.close()


def test_vakbl_of_ragged_rows():
    from miniafqmc_b200.afqmc import AfqmcSys
    nmo, nel, nw = 33, 5, 9                          # 2nN = 330
    s = dataclasses.replace(tiny_system(complex_trial=True, complex_chol=True, nmo=nmo, nel=nel,
                                        nchol=24))
    s.haj = np.zeros_like(s.haj)
    e = AfqmcSys(s, nw, walkers=walkers(s, nw))
    assert e.digit_products()["vakbl"]
    e.calculate_mixed_density_matrix()
    G = e.copy_out("Gc").astype(LD)
    e.calculate_energy("vakbl")
    V = s.Vakbl.todense().astype(LD)
    want = 0.5 * (G * (V @ G)).sum(0)
    size = np.linalg.norm(G.astype(complex), axis=0) * np.linalg.norm((V @ G).astype(complex), axis=0)
    assert np.all(np.abs(e.get_walker_data()[:, 0] - want) <= 2.0 ** -48 * size)
    e.close()


def test_k_splits_that_bound_the_int32_sums():
    """4nN = 17160 complex digits a row and 150 output tiles: two splits for the sums alone."""
    from miniafqmc_b200.afqmc import AfqmcSys
    from miniafqmc_b200.synthetic import CSR
    import scipy.sparse as sp
    nmo, nel, nchol, nw = 130, 33, 1200, 480
    s = dataclasses.replace(tiny_system(complex_trial=True, complex_chol=True, nmo=nmo, nel=nel,
                                        nchol=8, density=0.02))
    rng = np.random.default_rng(7)
    K = 2 * nel * nmo
    A = rng.normal(size=(nchol, K)) + 1j * rng.normal(size=(nchol, K))
    s.cfg = dataclasses.replace(s.cfg, nchol=nchol)
    s.SpvnT = CSR.from_scipy(sp.csr_matrix(A))
    s.Spvn = CSR.from_scipy(sp.csr_matrix((np.ones(nchol), (np.arange(nchol), np.arange(nchol))),
                                          shape=(nmo * nmo, nchol)).astype(complex))
    s.Lh = np.zeros((nchol, 2, nel, nmo), complex)
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=walkers(s, nw))
    assert e.digit_products()["vbias"]
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    rows, cols = np.array([0, 127, 128, 777, 1199]), np.array([0, 31, 32, 479])
    G = e.copy_out("Gc")[:, cols].astype(LD)
    assert norm_error(e.copy_out("vbias")[np.ix_(rows, cols)], A[rows].astype(LD) @ G) <= 2.0 ** -49
    e.close()


def test_short_k_bound_of_the_exchange():
    """2N = 16388 complex entries exceed the int32 sums: the exchange stays on the FP64 pipe."""
    from miniafqmc_b200.afqmc import AfqmcSys
    from miniafqmc_b200.synthetic import CSR, Config, System
    N = 8194
    one = CSR(N * N, 1, np.r_[0, np.ones(N * N, np.int32)].astype(np.int32), np.zeros(1, np.int32),
              np.ones(1, complex))
    trial = np.zeros((2, N, 1), complex)
    trial[:, 0] = 1.0
    Lh = np.full((1, 2, 1, N), 1.0 + 0.25j)
    s = System(cfg=Config(N, 1, 1, 0.1, 0, dt=0.01), h1=None, Wavefun=trial, spvn_coo=(),
               Propg1=np.zeros((N, N), complex))
    s.Spvn, s.trial, s.haj, s.Lh = one, trial, np.zeros((2, N), complex), Lh
    s.SpvnT = CSR(1, 2 * N, np.array([0, 1], np.int32), np.zeros(1, np.int32), np.ones(1, complex))
    W = np.ones((1, 2, N, 1), complex)
    e = AfqmcSys(s, 1, use_vakbl=False, walkers=(W, np.ones((1, 8), complex)))
    assert not e.digit_products()["exchange"] and e.digit_products()["coulomb"]
    e.calculate_mixed_density_matrix()
    e.calculate_energy("chol")
    want = (N * (1.0 + 0.25j)) ** 2                  # 1/2 sum over two spins of T^2, T = sum L
    assert abs(e.copy_out("energy_parts")[0, 2] - want.real) <= 1e-12 * abs(want)
    e.close()


def test_small_propagation_gives_the_separate_products_bits(monkeypatch):
    """16 walkers take the one-launch chain, 400 the separate products: the same bits for the
    walkers they share (both sum over k in order; AFQ_TUNE=0 keeps vbias and vHS alike)."""
    from miniafqmc_b200.afqmc import AfqmcSys
    monkeypatch.setenv("AFQ_TUNE", "0")
    monkeypatch.setenv("AFQ_FP64_DIGITS", "0")
    s = tiny_system(complex_trial=True, complex_chol=True, nmo=64, nel=16, nchol=40)
    W, Wd = walkers(s, 400)
    x = np.random.default_rng(5).normal(size=(40, 400))
    out = []
    for nw in (16, 400):
        e = AfqmcSys(s, nw, use_vakbl=False, walkers=(W[:nw], Wd[:nw]))
        e.calculate_mixed_density_matrix()
        e.get_vbias()
        e.sigma_from(x[:, :nw])
        e.get_vHS()
        V = e.copy_out("vHS")
        e.propagate()
        out.append((V[:, :16], e.get_walkers()[0][:16]))
        e.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


def test_reciprocal_of_the_gauss_jordan():
    """One electron: G = W / (W^T trial).  With the trial on orbital 0 and W[1] = 1, G[1] is the
    reciprocal of W[0] itself (gj_recip): within 8 roundings for every magnitude."""
    from miniafqmc_b200.afqmc import AfqmcSys
    nw = 4096
    s = dataclasses.replace(tiny_system(complex_trial=False, complex_chol=False, nmo=2, nel=1,
                                        nchol=4))
    s.trial = np.zeros((2, 2, 1), complex)
    s.trial[:, 0] = 1.0
    rng = np.random.default_rng(6)
    W = np.ones((nw, 2, 2, 1), complex)
    mag = np.exp2(rng.uniform(-900, 900, (nw, 2)))
    ratio = np.exp2(rng.uniform(-60, 60, (nw, 2)))
    sign = rng.choice([-1.0, 1.0], (2, nw, 2))
    re, im = mag * rng.uniform(1, 2, (nw, 2)), mag * np.minimum(ratio, 1.0) * rng.uniform(1, 2, (nw, 2))
    swap = rng.random((nw, 2)) < 0.5
    W[:, :, 0, 0] = np.where(swap, sign[0] * im + 1j * sign[1] * re, sign[0] * re + 1j * sign[1] * im)
    W[0, 0, 0, 0], W[1, 0, 0, 0], W[2, 0, 0, 0] = 1.0, 1j, -2.0 ** 512
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=(W, np.ones((nw, 8), complex)))
    e.calculate_mixed_density_matrix()
    G = e.copy_out("Gc").T.reshape(nw, 2, 1, 2)[:, :, 0, 1]
    want = 1.0 / W[:, :, 0, 0].astype(LD)
    assert np.all(np.abs(G - want) <= 8 * EPS * np.abs(want))
    e.close()
