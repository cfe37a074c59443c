"""FP64 form with the digit products switched off (AFQ_FP64_DIGITS=0): the products on the FP64
pipe that sizes without a digit form and handles short of memory run.  Against the digit
products on the same walkers, and with the set-up tuner's shapes against its rules (the same
bits: every shape sums an output in the same order)."""
import numpy as np
import pytest

from conftest import system, tiny_system

pytestmark = pytest.mark.gpu


def run(s, nw, wk, use_vakbl):
    from miniafqmc_b200.afqmc import AfqmcSys
    e = AfqmcSys(s, nw, use_vakbl=use_vakbl, walkers=wk)
    for k in range(1, 6):
        e.substep(4, k, 5)
    e.calculate_mixed_density_matrix()
    out = {"E": np.array([e.calculate_energy("chol")]), "parts": e.copy_out("energy_parts")}
    if use_vakbl:
        out["Evakbl"] = np.array([e.calculate_energy("vakbl")])
    e.get_vbias()
    out["vbias"], (out["W"], d) = e.copy_out("vbias"), e.get_walkers()
    out["weight"], out["overlap"] = d[:, 1], d[:, 2:4]
    res = out, e.digit_products(), e.sparse_paths()
    e.close()
    return res


def walkers(s, nw):
    rng = np.random.default_rng(nw)
    W, Wd = s.initial_walkers(nw)
    return W + 0.2 / np.sqrt(s.N) * (rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape)), Wd


@pytest.mark.parametrize("case", ["C1", "dense", "complex"])
def test_digit_products_agree_with_the_fp64_pipe(case, monkeypatch):
    s, nw, vak = {"C1": (system("C1"), 16, True),
                  "dense": (system("C1", density=0.3, nchol=128), 40, True),
                  "complex": (tiny_system(nmo=130, nel=24, nchol=160), 130, False)}[case]
    wk = walkers(s, nw)
    a, on, _ = run(s, nw, wk, vak)
    assert on["vbias"] and on["exchange"] and on["vakbl"] == vak
    monkeypatch.setenv("AFQ_FP64_DIGITS", "0")
    b, off, pb = run(s, nw, wk, vak)
    assert not any(off.values())
    for k in a:   # five substeps: an FP64 rounding grows by less than three digits
        assert np.max(np.abs(a[k] - b[k])) <= 2e-12 * np.max(np.abs(b[k])), k
    monkeypatch.setenv("AFQ_TUNE", "0")
    c, _, pc = run(s, nw, wk, vak)
    same = [v["path"] for v in pb.values()] == [v["path"] for v in pc.values()]
    for k in b:
        if same:
            assert np.array_equal(b[k], c[k]), k
        else:
            assert np.max(np.abs(b[k] - c[k])) <= 2e-12 * np.max(np.abs(b[k])), k
