"""FP64 form on the int8 tensor cores (oz_gemm.cuh): products of operands split into signed
8-bit digits against plain FP64 references (numpy, and the FP64-pipe kernels on the same
buffers).  Digits keep 55 bits below a row's power of two, so a product's error is that of an
FP64 product: bounds are a few hundred FP64 roundings of the terms summed."""
import numpy as np
import pytest

from conftest import tiny_system

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53

# tile edges: one tile, rows and columns just past a tile, several Cholesky blocks, K below,
# at and past a 64-entry slab; real and complex operands
SHAPES = [(16, 4, 12, 3, False), (33, 5, 29, 9, True), (64, 16, 64, 17, False),
          (65, 11, 70, 33, True), (24, 8, 130, 40, True), (96, 33, 40, 6, False)]


def engine(nmo, nel, nchol, nw, cplx, spread=0.3):
    from miniafqmc_b200.afqmc import AfqmcSys
    s = tiny_system(complex_trial=cplx, complex_chol=cplx, nmo=nmo, nel=nel, nchol=nchol)
    rng = np.random.default_rng(nmo + nw)
    W, Wd = s.initial_walkers(nw)
    W = W + spread / np.sqrt(nmo) * (rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape))
    return s, AfqmcSys(s, nw, use_vakbl=False, walkers=(W, Wd))


def gc(e):
    """Gc [nw][2][n][N] as the device holds it."""
    return e.copy_out("Gc").T.reshape(e.nw, 2, e.n, e.N)


def exchange(Lh, G):
    T = np.einsum("csak,wsbk->swcab", Lh, G, optimize=True)
    return 0.5 * np.einsum("swcab,swcba->w", T, T), np.einsum("swcab,swcba->w", abs(T), abs(T))


@pytest.mark.parametrize("nmo,nel,nchol,nw,cplx", SHAPES)
def test_exchange_matches_fp64(nmo, nel, nchol, nw, cplx):
    s, e = engine(nmo, nel, nchol, nw, cplx)
    e.calculate_mixed_density_matrix()
    e.calculate_energy("chol")
    got = e.copy_out("energy_parts")[:, 2]
    want, size = exchange(s.Lh, gc(e))
    # T carries 2 nmo roundings of its terms, twice in the product
    assert np.all(np.abs(got - want.real) <= 64 * nmo * EPS * size)
    e.close()


def test_exchange_of_a_non_finite_walker_stays_its_own():
    s, e = engine(33, 5, 29, 9, False)
    W, Wd = e.get_walkers()
    W[4, 1, 7, 2] = np.nan
    e.set_walkers(W, Wd)
    e.calculate_mixed_density_matrix()
    e.calculate_energy("chol")
    got = e.copy_out("energy_parts")[:, 2]
    assert np.isnan(got[4])
    keep = np.arange(9) != 4
    want, size = exchange(s.Lh, gc(e)[keep])
    assert np.all(np.abs(got[keep] - want.real) <= 64 * 33 * EPS * size)
    e.close()
