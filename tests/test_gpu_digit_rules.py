"""Where the FP64 form's digit products are taken (oz.cu): on both sides of each rule of size,
the results against the FP64 pipe's on the same walkers."""
import dataclasses

import numpy as np
import pytest

from conftest import tiny_system

pytestmark = pytest.mark.gpu


def run(s, nw, monkeypatch, digits, taylor=6):
    from miniafqmc_b200.afqmc import AfqmcSys
    monkeypatch.setenv("AFQ_FP64_DIGITS", "1" if digits else "0")
    rng = np.random.default_rng(nw)
    W, Wd = s.initial_walkers(nw)
    W = W + 0.2 / np.sqrt(s.N) * (rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape))
    e = AfqmcSys(s, nw, use_vakbl=False, walkers=(W, Wd))
    on = e.digit_products()
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    out = {"vbias": e.copy_out("vbias")}
    e.sigma_from(rng.normal(size=(s.nchol, nw)))
    e.get_vHS()
    e.propagate()
    out["W"] = e.get_walkers()[0]
    e.calculate_mixed_density_matrix()
    e.calculate_energy("chol")
    out["parts"] = e.copy_out("energy_parts")
    assert not any(e.digit_products_redone().values())
    e.close()
    return out, on


@pytest.mark.parametrize("nmo,nel,nchol,nw,on", [
    (32, 3, 24, 5, {"vbias": False, "exchange": True}),              # K = 192; 32 x 32 blocks
    (32, 4, 24, 5, {"vbias": True, "exchange": True}),               # K = 256
    (32, 8, 24, 40, {"vbias": True, "exchange": False}),             # short blocks
    (32, 10, 24, 40, {"vbias": True, "exchange": True}),             # n^2 N = 3200
    (31, 31, 8, 40, {"vbias": True, "exchange": False}),             # K below 32
    (64, 4, 40, 60, {"exchange": True}),                             # small blocks, few of them
    (64, 4, 80, 160, {"exchange": False}),                           # and many
    (17, 1, 40, 30, {"vbias": False, "exchange": True}),             # blocks of one
    (64, 16, 8, 700, {"propagate": False}),                          # two slabs of padding
    (121, 2, 8, 986, {"propagate": True}),
    (130, 30, 8, 30, {"propagate": False}),                          # half of the tiles padding
    (130, 64, 8, 175, {"propagate": True}),
    (192, 32, 8, 30, {"propagate": True}),
    (30, 14, 8, 332, {"propagate": False}),                          # one launch or eight
    (11, 5, 8, 721, {"propagate": False}),
])
def test_rules_of_size(nmo, nel, nchol, nw, on, monkeypatch):
    s = tiny_system(complex_trial=False, complex_chol=False, nmo=nmo, nel=nel, nchol=nchol)
    a, ra = run(s, nw, monkeypatch, True)
    b, rb = run(s, nw, monkeypatch, False)
    assert {k: ra[k] for k in on} == on and not any(rb.values())
    for k in a:
        assert np.max(np.abs(a[k] - b[k])) <= 2e-12 * np.max(np.abs(b[k])), k


def test_sparse_operand_rule(monkeypatch):
    """SpvnT of 2% (K = 2048: 43 nonzeros a row): CSR for few walkers, digits for many."""
    from miniafqmc_b200.synthetic import CSR
    s = dataclasses.replace(tiny_system(complex_trial=False, complex_chol=False, nmo=64, nel=16,
                                        nchol=64))
    rng = np.random.default_rng(2)
    s.SpvnT = CSR.from_scipy(rng.normal(size=(64, 2048)) * (rng.random((64, 2048)) < 0.022))
    for nw, on in ((16, False), (200, True)):
        a, ra = run(s, nw, monkeypatch, True)
        b, _ = run(s, nw, monkeypatch, False)
        assert ra["vbias"] == on
        assert np.max(np.abs(a["vbias"] - b["vbias"])) <= 2e-12 * np.max(np.abs(b["vbias"]))
