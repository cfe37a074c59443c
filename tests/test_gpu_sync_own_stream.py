"""afq_synchronize of an FP64 handle waits for the handle's own stream, not for work that the
caller has queued on the default stream."""
import pytest

from conftest import tiny_system

pytestmark = pytest.mark.gpu


def test_synchronize_leaves_the_default_stream_alone():
    import torch
    from miniafqmc_b200.afqmc import AfqmcSys
    s = tiny_system(nmo=64, nel=16, nchol=64)
    e = AfqmcSys(s, 8, use_vakbl=False)
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    assert e.digit_products()["vbias"]
    e.synchronize()
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    torch.cuda._sleep(1_000_000_000)     # about half a second
    done.record()
    e.calculate_mixed_density_matrix()
    e.get_vbias()
    e.synchronize()
    assert not done.query()
    torch.cuda.synchronize()
    e.close()
