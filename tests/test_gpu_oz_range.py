"""FP64 form, results that 55-bit fixed-point rows do not hold: operand rows whose large entries
meet only zeros of the other operand (every output comes from entries 1e-13 of the row's
largest), infinities, scales at the ends of the range, and pipeline waits that run out.  The
product's columns stay unmarked (oz_gemm.cuh) and the FP64 pipe computes them: the results carry
FP64's rounding of the terms, as without digits.  References: numpy in long double."""
import dataclasses

import numpy as np
import pytest

from conftest import tiny_system

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
LD = np.clongdouble
TINY = 1e-13
WAIT_CLOCKS = 300   # far below one bulk copy: every work wait runs out


def csr(dense):
    from miniafqmc_b200.synthetic import CSR
    return CSR.from_scipy(dense)


def graded_system(nmo=64, nel=16, nchol=64, k0=5):
    """Half-rotated operands that are large at orbital k0 alone."""
    s = dataclasses.replace(tiny_system(complex_trial=False, complex_chol=False, nmo=nmo, nel=nel,
                                        nchol=nchol))
    scale = np.full(nmo, TINY)
    scale[k0] = 1.0
    rng = np.random.default_rng(5)
    s.Lh = (rng.normal(size=s.Lh.shape) * scale).astype(complex)
    s.SpvnT = csr(0.1 * s.Lh.reshape(nchol, -1))
    m = 2 * nel * nmo
    s.Vakbl = csr(rng.normal(size=(m, m)) * np.tile(scale, 2 * nel))
    s.haj = np.zeros_like(s.haj)
    return s


def walkers(s, nw, seed=3):
    rng = np.random.default_rng(seed)
    W, Wd = s.initial_walkers(nw)
    return W + 0.3 / np.sqrt(s.N) * (rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape)), Wd


def test_products_with_g_of_graded_rows():
    from miniafqmc_b200.afqmc import AfqmcSys
    s, nw, k0 = graded_system(), 24, 5
    W, Wd = walkers(s, nw)
    W[:, :, k0, :] = 0.0                             # G is zero at k0
    e = AfqmcSys(s, nw, walkers=(W, Wd))
    on = e.digit_products()
    assert on["vbias"] and on["coulomb"] and on["vakbl"] and on["exchange"]
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    Gc = e.copy_out("Gc")
    assert np.all(Gc.reshape(2 * s.n, s.N, nw)[:, k0] == 0)
    G = Gc.astype(LD)

    def close(got, A, extra=1.0):
        want, size = A @ G, np.abs(A) @ np.abs(G)
        bound = 64 * np.sqrt(A.shape[1]) * EPS * extra
        assert np.all(np.abs(got - want) <= bound * size)

    A = s.SpvnT.todense().astype(LD)
    close(e.copy_out("vbias"), A)
    e.calculate_energy("chol")
    parts = e.copy_out("energy_parts")
    L = s.Lh.astype(LD)
    c, csize = L.reshape(s.nchol, -1) @ G, np.abs(L.reshape(s.nchol, -1)) @ np.abs(G)
    assert np.all(np.abs(parts[:, 1] - 0.5 * (c * c).sum(0).real)
                  <= 256 * np.sqrt(A.shape[1]) * EPS * (csize ** 2).sum(0))
    Gw = G.T.reshape(nw, 2, s.n, s.N)
    for w in range(0, nw, 5):
        ek = size = 0.0
        for sp in range(2):
            T = L[:, sp] @ Gw[w, sp].T
            ek += 0.5 * (T * T.transpose(0, 2, 1)).sum().real
            size += (np.abs(T) ** 2).sum()
        assert abs(parts[w, 2] - ek) <= 64 * s.N * EPS * size
    E = e.calculate_energy("vakbl")
    V = s.Vakbl.todense().astype(LD)
    e2, size = 0.5 * (G * (V @ G)).sum(0), (np.abs(G) * (np.abs(V) @ np.abs(G))).sum(0)
    loc = e.get_walker_data()[:, 0]
    assert np.all(np.abs(loc - e2) <= 64 * np.sqrt(A.shape[1]) * EPS * size)
    redone = e.digit_products_redone()
    assert redone["vbias"] == redone["coulomb"] == redone["vakbl"] == redone["exchange"] == nw
    assert redone["vHS"] == 0
    # ordinary walkers on the same handle: the digit products again
    e.set_walkers(*walkers(s, nw))
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    G = e.copy_out("Gc").astype(LD)
    close(e.copy_out("vbias"), A)
    assert e.digit_products_redone()["vbias"] == nw
    e.close()


def test_vhs_of_graded_rows():
    from miniafqmc_b200.afqmc import AfqmcSys
    nmo, nel, nchol, nw, c0 = 130, 9, 96, 131, 7
    s = dataclasses.replace(tiny_system(complex_trial=False, complex_chol=False, nmo=nmo, nel=nel,
                                        nchol=nchol))
    rng = np.random.default_rng(6)
    A = rng.normal(size=(nmo * nmo, nchol)) * (rng.random((nmo * nmo, nchol)) < 0.7) * TINY
    A[:, c0] = 1.0
    s.Spvn = csr(A)
    T = s.SpvnT.todense()
    T[c0] = 0.0
    s.SpvnT = csr(T)
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=walkers(s, nw))
    assert e.digit_products()["vHS"]
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    x = rng.normal(size=(nchol, nw))
    x[c0] = 0.0
    e.sigma_from(x)
    X = e.copy_out("X")
    assert np.all(X[c0] == 0)
    e.get_vHS()
    V = e.copy_out("vHS")
    assert e.digit_products_redone()["vHS"] == nw
    rows = rng.choice(nmo * nmo, 500, replace=False)
    want = A[rows].astype(LD) @ X.astype(LD)
    size = np.abs(A[rows]) @ np.abs(X)
    assert np.all(np.abs(V[rows] - want) <= 64 * np.sqrt(nchol) * EPS * size)
    e.close()


def test_propagation_past_a_large_entry_of_vhs():
    """vHS couples orbital p to orbital q by 1e12; no walker reaches q."""
    from miniafqmc_b200.afqmc import AfqmcSys
    nmo, nel, nchol, nw, p, q = 128, 20, 64, 160, 9, 40
    s = dataclasses.replace(tiny_system(complex_trial=False, complex_chol=False, nmo=nmo, nel=nel,
                                        nchol=nchol))
    A = s.Spvn.todense().reshape(nmo, nmo, nchol)
    A[q], A[:, q] = 0.0, 0.0
    A[p, q, 0] = 1e12
    s.Spvn = csr(A.reshape(nmo * nmo, nchol))
    s.Propg1 = np.eye(nmo, dtype=complex)
    W, Wd = walkers(s, nw)
    W[:, :, q, :] = 0.0
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=(W, Wd))
    assert e.digit_products()["propagate"]
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    e.sigma_from(np.random.default_rng(8).normal(size=(nchol, nw)))
    e.get_vHS()
    V = e.copy_out("vHS")
    for _ in range(2):
        W0 = e.get_walkers()[0]
        e.propagate()
        W1 = e.get_walkers()[0]
        for w in range(0, nw, 31):
            for sp in range(2):
                T = W0[w, sp]
                S = T.copy()
                for k in range(1, 7):
                    T = (1j / k) * (V[:, w].reshape(nmo, nmo) @ T)
                    S = S + T
                assert np.max(np.abs(W1[w, sp] - S)) <= 1e-13 * np.max(np.abs(S))
    assert e.digit_products_redone()["propagate"] == 2 * nw
    e.close()


def exchange_of_buffers(L, G):
    import torch
    from miniafqmc_b200.afqmc import load_library
    nchol, _, nel, nmo = L.shape
    nw = G.shape[0]
    ek = torch.full((nw,), 7.0, dtype=torch.complex128, device="cuda")
    st = load_library().afq_exchange_energy_noalloc(
        L.data_ptr(), G.data_ptr(), nmo, nel, nchol, nw, ek.data_ptr(),
        torch.cuda.current_stream().cuda_stream)
    assert st == 0
    return ek.cpu().numpy()


def exchange_reference(L, G):
    L, G = L.cpu().numpy().astype(LD), G.cpu().numpy().astype(LD)
    ek, size = np.zeros(G.shape[0], LD), np.zeros(G.shape[0])
    for w in range(G.shape[0]):
        for s in range(2):
            T = L[:, s] @ G[w, s].T
            ek[w] += 0.5 * (T * T.transpose(0, 2, 1)).sum()
            size[w] += float((np.abs(T) ** 2).sum())
    return ek, size


def buffers(cplx, nmo=41, nel=20, nchol=120, nw=60):
    import torch
    g = torch.Generator("cuda").manual_seed(nmo)
    rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    Lr = rand(nchol, 2, nel, nmo)
    L = torch.complex(Lr, rand(nchol, 2, nel, nmo) if cplx else torch.zeros_like(Lr))
    return L, torch.complex(rand(nw, 2, nel, nmo), rand(nw, 2, nel, nmo))


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("kind", ["plain", "graded", "scaled"])
def test_exchange_of_buffers_of_any_scaling(kind, cplx):
    L, G = buffers(cplx)
    up = 1.0
    if kind == "graded":       # all walkers but one meet only the small entries
        L[..., 1:] *= TINY
        G[1:, ..., 0] = 0.0
    elif kind == "scaled":     # past the digit products' range, the products within FP64's
        up = 2.0 ** 950
    want, size = exchange_reference(L, G)
    got = exchange_of_buffers(L * up, G / up)
    assert np.all(np.abs(got - want) <= 64 * L.shape[3] * EPS * size)


def test_infinity_is_the_fp64_pipes(monkeypatch):
    from miniafqmc_b200.afqmc import AfqmcSys
    s = dataclasses.replace(tiny_system(complex_trial=False, complex_chol=False, nmo=64, nel=16,
                                        nchol=64))
    A = np.random.default_rng(9).normal(size=(64, 2 * 16 * 64))
    A[3, 77] = np.inf
    s.SpvnT = csr(A)
    nw = 24
    wk = walkers(s, nw)
    out = []
    for digits in ("1", "0"):
        monkeypatch.setenv("AFQ_FP64_DIGITS", digits)
        e = AfqmcSys(s, nw, use_vakbl=False, walkers=wk)
        assert e.digit_products()["vbias"] == (digits == "1")
        e.calculate_mixed_density_matrix()
        e.get_vbias()
        out.append(e.copy_out("vbias"))
        e.close()
    assert np.array_equal(out[0], out[1], equal_nan=True)
    assert not np.any(np.isfinite(out[0][3])) and np.all(np.isfinite(np.delete(out[0], 3, 0)))


def test_waits_that_run_out_are_reported_and_the_fp64_pipe_computes():
    from miniafqmc_b200.afqmc import AfqmcError, AfqmcSys, load_library
    lib = load_library()
    s = tiny_system(complex_trial=False, complex_chol=False, nmo=128, nel=20, nchol=64)
    nw = 160
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=walkers(s, nw))
    on = e.digit_products()
    assert on["vbias"] and on["exchange"] and on["propagate"]
    x = np.random.default_rng(8).normal(size=(64, nw))
    W0 = e.get_walkers()
    L, G = buffers(True)
    wantb, sizeb = exchange_reference(L, G)

    def step():
        e.set_walkers(*W0)
        e.calculate_mixed_density_matrix()
        e.get_vbias()
        e.sigma_from(x)
        e.get_vHS()
        e.propagate()
        W = e.get_walkers()[0]
        e.calculate_mixed_density_matrix()
        return {"vbias": e.copy_out("vbias"), "W": W, "E": np.array([e.calculate_energy("chol")])}

    want = step()
    e.synchronize()
    before = e.digit_products_redone()
    assert lib.afq_set_tc_wait_limit(0, WAIT_CLOCKS) == 0
    try:
        got = step()
        gotb = exchange_of_buffers(L, G)
        with pytest.raises(AfqmcError) as ei:
            e.synchronize()
    finally:
        assert lib.afq_set_tc_wait_limit(0, 0) == 0
    assert ei.value.status == 3 and "timed out" in str(ei.value)
    for k in want:
        assert np.max(np.abs(got[k] - want[k])) <= 2e-12 * np.max(np.abs(want[k])), k
    assert np.all(np.abs(gotb - wantb) <= 64 * L.shape[3] * EPS * sizeb)
    after = e.digit_products_redone()
    assert after["vbias"] > before["vbias"] and after["propagate"] > before["propagate"]
    got = step()
    e.synchronize()                                   # reported once, then cleared
    assert e.digit_products_redone() == after
    for k in want:
        assert np.array_equal(got[k], want[k]), k
    e.close()
