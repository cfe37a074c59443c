"""The digits and workspaces of an FP64 handle take at most a sixth of the device memory that is
free at set-up, however many products run on them, so a further handle finds nearly the room it
did without them; products that do not fit run on the FP64 pipe."""
import pytest

from conftest import tiny_system

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_digits_leave_the_memory_to_others(monkeypatch):
    import torch
    from miniafqmc_b200.afqmc import AfqmcSys
    s = tiny_system(complex_trial=False, complex_chol=False, nmo=128, nel=32, nchol=256)
    nw = 256
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    AfqmcSys(s, nw, use_vakbl=False).close()     # the library's kernels and static arrays
    torch.cuda.empty_cache()
    hold = torch.empty(free() - 1200 * MB, dtype=torch.uint8, device="cuda")
    used = {}
    for digits in ("1", "0"):
        monkeypatch.setenv("AFQ_FP64_DIGITS", digits)
        before = free()
        e = AfqmcSys(s, nw, use_vakbl=False)
        used[digits] = before - free()
        if digits == "1":
            on, at_setup = e.digit_products(), before
            e.substep(1, 1, 5)
            e.synchronize()
        e.close()
    del hold
    torch.cuda.empty_cache()
    assert any(on.values()) and not all(on[k] for k in ("vbias", "coulomb", "exchange", "propagate"))
    # small buffers share 32 MB blocks
    assert used["1"] - used["0"] <= at_setup / 6 + 32 * MB
