"""Dedispersion from rings no longer than they must be: the smallest power of two
that holds the valid rows, which start anywhere on it.  NaN (int8: -128) fills the
ring's other rows and guards behind the last channel; a value is a sum of nchan FP32
terms, <= 1e-5 of the rms as for the other kernels."""
import numpy as np
import pytest

from test_band_gpu import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [0, 1, 2])
@pytest.mark.parametrize("ndm,nch,nt,dm_max,row0", [
    (17, 64, 1, 1.0, 71), (17, 64, 7, 20.0, 1039), (40, 96, 300, 30.0, 510), (60, 64, 97, 4.0, 127), (400, 64, 20, 60.0, 3)])
def test_smallest_ring(vf, O, ndm, nch, nt, dm_max, row0, storage):
    import torch
    from vfrb_oracle import delay_table
    off, _ = delay_table(np.linspace(0, dm_max, ndm).astype(np.float32), 384.0, 64.0 / nch, 0.001, nch)
    R = max((4, 8, 16)[storage], 1 << (nt + int(off.max()) - 1).bit_length())
    off, ring, fb, rows = _case(ndm, nch, nt, dm_max, 7, storage, row0, R)
    assert ring.shape == (nch, R) and rows <= R
    kw = {}
    if storage:
        kw = dict(uniform_scale=0.5)
        fb = fb * 0.5
    ref = O.dedisperse(fb, off, nt)
    guarded = torch.full(((nch + 8) * R,), -128 if storage == 2 else float("nan"), dtype=torch.from_numpy(ring).dtype,
                         device="cuda")
    x = guarded[4 * R:(nch + 4) * R].view(nch, R)
    x.copy_(torch.from_numpy(ring))
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    got, _ = vf.DedispPlan(off)(x, nt, storage=storage, row0=row0, row_mask=R - 1, nrows_valid=rows, d_err=err,
                                stats=False, **kw)
    assert int(err.item()) == 0
    assert np.max(np.abs(got.cpu().numpy() - ref)) <= 1e-5 * np.sqrt(np.mean(ref ** 2))
