"""Panel Gauss-Jordan (gj.cuh) in the density matrix of both forms: sizes around the panel of
eight pivots and the 32 rows of a warp, pivoting across panels, singular and non-finite
walkers.  Reference: numpy's inverse and determinant in FP64.  Backward stable with partial
pivoting: errors within c n^2 eps times the condition number (FP64), within the bf16 split's
2^-14 of the terms summed (mixed)."""
import numpy as np
import pytest

from conftest import tiny_system

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def walkers(s, nw, seed):
    """Walkers whose overlap matrices are full and need row exchanges."""
    rng = np.random.default_rng(seed)
    W, Wd = s.initial_walkers(nw)
    W = rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape) + 0.2 * W
    return W, Wd


def reference(s, W):
    T1 = np.einsum("wsia,sib->wsab", W, s.trial)
    return T1, np.linalg.det(T1), np.linalg.solve(T1, np.swapaxes(W, 2, 3))


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 40, 47, 48, 63, 64])
def test_fp64_density_matrix(n):
    from miniafqmc_b200.afqmc import AfqmcSys
    N, nw = n + 5, 5
    s = tiny_system(nmo=N, nel=n, nchol=6)
    W, Wd = walkers(s, nw, n)
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=(W, Wd))
    e.calculate_mixed_density_matrix()
    G, D = e.copy_out("Gc").T.reshape(nw, 2, n, N), e.get_walker_data()[:, 2:4]
    T1, det, want = reference(s, W)
    cond = np.linalg.cond(T1)
    tol = 64 * n * n * EPS * cond
    assert np.all(np.abs(D - det) <= tol * np.abs(det))
    err = np.abs(G - want).max((2, 3)) / np.abs(want).max((2, 3))
    assert np.all(err <= tol)
    e.calculate_overlaps(save_old=True)   # the determinant alone
    D2 = e.get_walker_data()
    assert np.all(np.abs(D2[:, 2:4] - det) <= tol * np.abs(det))
    assert np.array_equal(D2[:, 6:8], D)
    assert np.all(e.copy_out("info") == 0)
    e.close()


@pytest.mark.parametrize("n", [4, 8, 12, 32, 36, 48, 64])
def test_mixed_density_matrix(n):
    from miniafqmc_b200.afqmc import AfqmcSys, AFQ_PREC_MIXED
    N, nw = (n + 15) // 8 * 8, 5
    s = tiny_system(complex_trial=False, complex_chol=False, nmo=N, nel=n, nchol=8)
    W, Wd = walkers(s, nw, n)
    e = AfqmcSys(s, nw, precision=AFQ_PREC_MIXED, use_vakbl=False, walkers=(W, Wd))
    e.calculate_mixed_density_matrix()
    G = e.copy_out("Gc").T.reshape(nw, 2, n, N)
    T1, det, want = reference(s, W)
    terms = np.abs(np.linalg.inv(T1)) @ np.swapaxes(np.abs(W), 2, 3)
    # T1 itself carries the split's error: a relative perturbation of the inverse by cond(T1)
    tol = 2.0 ** -14 * (1 + np.linalg.cond(T1))[:, :, None, None]
    assert np.all(np.abs(G - want) <= tol * terms.max((2, 3), keepdims=True))
    e.close()


def test_singular_and_non_finite_walkers_stay_their_own():
    from miniafqmc_b200.afqmc import AfqmcSys
    n, N, nw = 19, 24, 6
    s = tiny_system(nmo=N, nel=n, nchol=6)
    W, Wd = walkers(s, nw, 3)
    W[1, 0, :, 11] = 0.0              # an exactly zero row of T1, past the first panel
    W[2, 1, 3, 9] = np.nan
    W[4] *= 1e-180                    # products of pivots below the normal range, row by row finite
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=(W, Wd))
    e.calculate_mixed_density_matrix()
    G, D, info = (e.copy_out("Gc").T.reshape(nw, 2, n, N), e.get_walker_data()[:, 2:4],
                  e.copy_out("info"))
    assert D[1, 0] == 0 and info[1, 0] == 1 and np.all(G[1, 0] == 0)
    assert info[1, 1] == 0 and np.all(np.isfinite(G[1, 1]))
    assert np.isnan(D[2, 1]) and np.isfinite(D[2, 0])
    T1, det, want = reference(s, W[[0, 3, 4, 5]])
    err = np.abs(G[[0, 3, 4, 5]] - want).max((2, 3)) / np.abs(want).max((2, 3))
    assert np.all(err <= 64 * n * n * EPS * np.linalg.cond(T1))
    e.close()
