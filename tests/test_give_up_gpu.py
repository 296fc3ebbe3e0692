"""A dedispersion kernel whose bounded wait for its own copies gives up: the call ends,
says so in d_err, and leaves the context and the plan usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["AUTO", "PAT4", "PAT2"])
@pytest.mark.parametrize("ndm", [48, 700])  # split and whole CTAs of the band-wise kernel
def test_a_wait_that_gives_up_is_flagged(vf, O, variant, ndm):
    import torch
    off, _ = O.delay_table(np.linspace(0, 20.0, ndm).astype(np.float32), 384.0, 0.25, 1e-3, 256)
    nt = 700
    fb = torch.randn((256, (nt + int(off.max()) + 15) // 16 * 16), device="cuda")
    plan = vf.DedispPlan(off)
    plan.set_variant(vf.F32, getattr(vf, "DD_" + variant))
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    want, _ = plan(fb, nt, d_err=err, stats=False)
    want = want.clone()
    assert int(err.item()) == 0
    plan.set_give_up(True)
    plan(fb, nt, d_err=err, stats=False)
    assert int(err.item()) == 8
    plan.set_give_up(False)
    err.zero_()
    got, _ = plan(fb, nt, d_err=err, stats=False)
    assert int(err.item()) == 0 and torch.equal(got, want)
