"""Mixed-form exchange over many Cholesky blocks: the persistent kernel walks the tiles in
groups of half the SMs' M tiles, so block counts below, at and past one and two groups and a
ragged last group must all be covered.  Reference: the exchange of the same density matrices
in FP64 (numpy).  Each operand carries 16 significant bits (bf16 hi + lo, the lo * lo product
dropped), so a block's T is within 2^-15 of the sum of its terms' magnitudes, and T enters
twice."""
import numpy as np
import pytest

from conftest import tiny_system

pytestmark = pytest.mark.gpu


# 2n = 24, 32, 64 and 128: 10, 8, 4 and 2 Cholesky vectors per tile
@pytest.mark.parametrize("nmo,nel,nchol,nw", [(16, 12, 16, 5), (32, 16, 600, 9), (32, 16, 592, 3),
                                              (32, 32, 608, 4), (64, 64, 304, 3),
                                              # other widths, per-tile kernel: walkers in
                                              # batches of eight, half circles of pairs
                                              (32, 4, 80, 37), (40, 8, 40, 17), (40, 20, 32, 7),
                                              (56, 28, 16, 10), (64, 36, 8, 5), (48, 44, 8, 3),
                                              (64, 60, 8, 3)])
def test_exchange_covers_every_block(nmo, nel, nchol, nw):
    from miniafqmc_b200.afqmc import AfqmcSys, AFQ_PREC_MIXED
    s = tiny_system(complex_trial=False, complex_chol=False, nmo=nmo, nel=nel, nchol=nchol)
    rng = np.random.default_rng(nchol)
    W, Wd = s.initial_walkers(nw)
    if nel < nmo:
        W = W + 0.3 / np.sqrt(nmo) * (rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape))
    e = AfqmcSys(s, nw, precision=AFQ_PREC_MIXED, use_vakbl=False, walkers=(W, Wd))
    e.calculate_mixed_density_matrix()
    e.calculate_energy("chol")
    got = e.copy_out("energy_parts")[:, 2]
    G = e.copy_out("Gc").T.reshape(nw, 2, nel, nmo)
    T = np.einsum("csak,wsbk->swcab", s.Lh, G, optimize=True)
    M = np.einsum("csak,wsbk->swcab", abs(s.Lh), abs(G.real) + abs(G.imag), optimize=True)
    want = 0.5 * np.einsum("swcab,swcba->w", T, T).real
    size = np.einsum("swcab,swcba->w", M, M)
    assert np.all(np.abs(got - want) <= 2.0 ** -14 * size)
    # a block left out or counted twice shows even where terms cancel
    per = np.abs(0.5 * np.einsum("swcab,swcba->wc", T, T).real)
    assert np.all(np.abs(got - want) < 0.5 * np.median(per, axis=1))
    e.close()
