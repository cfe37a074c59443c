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


def stages(nmo, nel, nchol, nw, cplx, **kw):
    s, e = engine(nmo, nel, nchol, nw, cplx, **kw)
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    e.sigma_from(np.random.default_rng(3).normal(size=(nchol, nw)))
    return s, e


@pytest.mark.parametrize("nmo,nel,nchol,nw,cplx", SHAPES)
def test_vbias_and_coulomb_match_fp64(nmo, nel, nchol, nw, cplx):
    """Products with G over K splits (a K of one slab up to several slabs per split)."""
    s, e = stages(nmo, nel, nchol, nw, cplx)
    G = e.copy_out("Gc")
    A = s.SpvnT.todense()
    size = np.abs(A) @ np.abs(G)
    big = np.abs(A).max(1)[:, None] * np.abs(G).max(0)[None] * np.sqrt(A.shape[1])
    assert np.all(np.abs(e.copy_out("vbias") - A @ G) <= 64 * EPS * (np.sqrt(A.shape[1]) * size + big))
    e.calculate_energy("chol")
    L = s.Lh.reshape(nchol, -1)
    c, csize = L @ G, np.abs(L) @ np.abs(G)
    ej = 0.5 * (c * c).sum(0).real
    assert np.all(np.abs(e.copy_out("energy_parts")[:, 1] - ej)
                  <= 256 * np.sqrt(A.shape[1]) * EPS * (csize ** 2).sum(0))
    e.close()


# large enough for the digit products by the rules of oz.cu: tile edges in every direction,
# real and complex Hamiltonians, one and two row tiles, odd electron and walker counts
@pytest.mark.parametrize("nmo,nel,nchol,nw,cplx", [(130, 9, 96, 131, False), (67, 21, 150, 83, True),
                                                   (128, 16, 64, 80, False)])
def test_vhs_and_propagation_match_fp64(nmo, nel, nchol, nw, cplx):
    s, e = stages(nmo, nel, nchol, nw, cplx)
    X = e.copy_out("X")
    e.get_vHS()
    V = e.copy_out("vHS")
    A = s.Spvn.todense()
    big = np.abs(A).max(1)[:, None] * np.abs(X).max(0)[None] * np.sqrt(nchol)
    assert np.all(np.abs(V - A @ X) <= 64 * EPS * (np.sqrt(nchol) * (np.abs(A) @ np.abs(X)) + big))
    W0 = e.get_walkers()[0]
    e.propagate()
    W1 = e.get_walkers()[0]
    P = s.Propg1
    for w in range(0, nw, 7):
        Vw = V[:, w].reshape(nmo, nmo)
        for sp in range(2):
            T = P @ W0[w, sp]
            S = T.copy()
            for k in range(1, 7):
                T = (1j / k) * (Vw @ T)
                S = S + T
            want = P @ S
            assert np.max(np.abs(W1[w, sp] - want)) <= 1e-13 * np.max(np.abs(want))
    e.close()


# the caller-owned buffers' path from its threshold on: several walker and Cholesky chunks,
# chunks that end inside a row tile, n up to 96, real and complex factors, and the largest n
@pytest.mark.parametrize("nmo,nel,nchol,nw,cplx", [(33, 20, 900, 131, False), (40, 40, 150, 61, True),
                                                   (96, 96, 70, 33, False), (61, 3, 800, 700, True)])
def test_exchange_of_buffers_matches_fp64(nmo, nel, nchol, nw, cplx):
    import torch
    from miniafqmc_b200.afqmc import load_library
    g = torch.Generator("cuda").manual_seed(nmo)

    def rand(*shape, imag=True):
        x = torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)
        y = torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)
        return torch.complex(x, y if imag else torch.zeros_like(y))

    L, G = rand(nchol, 2, nel, nmo, imag=cplx), rand(nw, 2, nel, nmo)
    G[1] *= 1e-200   # a row scale of its own per walker; T T underflows to zero
    G[2, 1, 0, 0] = float("inf")
    ek = torch.empty(nw, dtype=torch.complex128, device="cuda")
    lib = load_library()
    for _ in range(2):
        ek.fill_(7.0)
        st = lib.afq_exchange_energy_noalloc(L.data_ptr(), G.data_ptr(), nmo, nel, nchol, nw,
                                             ek.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert st == 0
    want = torch.zeros(nw, dtype=torch.complex128, device="cuda")
    size = torch.zeros(nw, dtype=torch.float64, device="cuda")
    for s in range(2):
        for c in range(nchol):
            T = torch.einsum("ak,wbk->wab", L[c, s], G[:, s])
            want += 0.5 * (T * T.transpose(1, 2)).sum((1, 2))
            size += (T.abs() ** 2).sum((1, 2))
    got, want, size = ek.cpu().numpy(), want.cpu().numpy(), size.cpu().numpy()
    assert not np.isfinite(got[2])
    keep = np.arange(nw) != 2
    assert np.all(np.abs(got[keep] - want[keep]) <= 64 * nmo * EPS * size[keep])
