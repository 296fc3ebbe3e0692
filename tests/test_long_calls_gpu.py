"""Calls of more samples than a grid's second dimension has tiles for: they run the same
kernel as short ones, which shows in the bits, since the order of a sample's sums
depends on the kernel and not on the call's length."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndm,nt,nch", [(8, 128 * 65535 + 1000, 40),    # streaming kernel, 128 samples a CTA
                                        (17, 288 * 65535 + 1000, 40)])  # band-wise kernel, tiles of 288
def test_long_calls_sum_like_short_ones(vf, O, ndm, nt, nch):
    import torch
    off, _ = O.delay_table(np.linspace(0, 1.6, ndm).astype(np.float32), 384.0, 64.0 / nch, 1e-3, nch)
    plan = vf.DedispPlan(off)
    rows = (nt + plan.max_delay + 15) // 16 * 16
    if torch.cuda.mem_get_info()[0] < 4 * (nch * rows + ndm * nt) + (2 << 30):
        pytest.skip("needs the device memory")
    fb = torch.empty((nch, rows), device="cuda").normal_(generator=torch.Generator("cuda").manual_seed(1))
    out, st = plan(fb, nt)
    for t0, n in ((0, 3000), (nt // 2 // 16 * 16, 3000), (nt - 2001, 2001)):
        cut, _ = plan(fb, n, row0=t0, nrows_valid=rows - t0, stats=False)
        assert torch.equal(out[:, t0:t0 + n], cut), t0
    mx, arg = out.max(dim=1)
    assert torch.equal(st["argmax"].long(), arg)
