"""Split-K vbias / Coulomb product of the mixed form at a K of 4096, where the estimate of waves and
slices (mixed.cu) takes 256-column tiles for these counts: ragged rows and columns, an odd walker
count.  Reference: FP64 product with the form's own density matrix; operands carry 16 significant
bits, so each result is within 2^-14 of its sum of absolute terms."""
import numpy as np
import pytest

from miniafqmc_b200.synthetic import Config, make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchol,nw", [(640, 256), (632, 255), (584, 200), (640, 384)])
def test_vbias_of_wide_tiles(nchol, nw):
    from miniafqmc_b200.afqmc import AfqmcSys, AFQ_PREC_MIXED
    nmo, nel = 128, 16
    s = make_system(Config(nmo, nel, nchol, 0.02, 7, dt=0.01, nwalk=nw, complex_trial=False,
                           complex_chol=False), build_vakbl=False)
    rng = np.random.default_rng(nchol + nw)
    W, Wd = s.initial_walkers(nw)
    W = W + 0.1 / np.sqrt(nmo) * (rng.normal(size=W.shape) + 1j * rng.normal(size=W.shape))
    e = AfqmcSys(s, nw, precision=AFQ_PREC_MIXED, use_vakbl=False, walkers=(W, Wd))
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    G, got = e.copy_out("Gc"), e.copy_out("vbias")
    e.close()
    F = s.SpvnT.to_scipy()
    assert np.all(np.abs(got - F @ G) <= 2.0 ** -14 * (np.abs(F) @ np.abs(G)))
