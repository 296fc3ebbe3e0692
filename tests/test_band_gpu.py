"""The automatic choice's own dedispersion kernels -- streaming for few trials,
band-wise for equally spaced ones -- against the FP64 oracle: every storage form with and without channel
weights, sizes at the edges of its tiles and trial groups, ring wrap, rows
outside the valid ones (NaN there must not reach an output), batched statistics.

Tolerances: a series value is a sum of nchan FP32 terms in a few levels (runs,
chunks, bands): <= 1e-5 of the rms, as for the other kernels; the weighted
forms round each product once, 6e-8 of a term, far below that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(ndm, nch, nt, dm_max, seed, storage, row0, R):
    """Ring [nch][R] with the valid rows from row0 on, NaN (int8: -128) elsewhere, and the FP64 rows."""
    from vfrb_oracle import delay_table
    rng = np.random.default_rng(seed)
    dms = np.linspace(0, dm_max, ndm).astype(np.float32)
    off, _ = delay_table(dms, 384.0, 64.0 / nch, 0.001, nch)
    rows = nt + int(off.max())
    fb = rng.standard_normal((rows, nch)).astype(np.float32) * 3.0
    if R == 0:
        R = (row0 + rows + 15) // 16 * 16 + 16
    if storage == 2:
        ring = np.full((nch, R), -128, np.int8)
        fb = np.clip(np.round(fb * 16), -127, 127).astype(np.int8)
    else:
        dt = np.float16 if storage == 1 else np.float32
        ring = np.full((nch, R), np.nan, dt)
        fb = fb.astype(dt)
    ring[:, (row0 + np.arange(rows)) % R] = fb.T
    return off, ring, fb.astype(np.float64), rows


@pytest.mark.parametrize("storage,weighted", [(0, False), (1, False), (1, True), (2, False), (2, True)])
@pytest.mark.parametrize("ndm,nch,nt,dm_max,row0,R", [
    (1, 64, 1, 3.0, 0, 0),            # streaming: one trial, one sample
    (16, 333, 1290, 40.0, 900, 2048), # streaming: most trials, a ragged channel count, the ring wraps
    (17, 64, 1, 3.0, 0, 0),           # one sample; the last group overlaps the one before
    (50, 320, 449, 30.0, 0, 0),       # last group overlaps the one before; one past an FP16 tile
    (97, 256, 1500, 90.0, 5, 0),      # a start off the alignment
    (33, 512, 960, 8.0, 1900, 2048),  # the ring wraps
    (48, 96, 481, 400.0, 0, 0),       # many rows per trial: bands of a few channels
    (400, 128, 289, 60.0, 3, 0),      # eight groups to a CTA
    (700, 64, 700, 40.0, 0, 0),       # sixteen groups to a CTA
])
def test_automatic_kernels_match_fp64(vf, O, ndm, nch, nt, dm_max, row0, R, storage, weighted):
    import torch
    off, ring, fb, rows = _case(ndm, nch, nt, dm_max, ndm + nt, storage, row0, R)
    w = np.random.default_rng(5).uniform(0.5, 2.0, nch).astype(np.float32) if weighted else None
    kw = {}
    if storage and weighted:
        kw = dict(chan_scale=torch.from_numpy(w).cuda())
        fb = fb * w[None, :].astype(np.float64)
    elif storage:
        kw = dict(uniform_scale=0.5)
        fb = fb * 0.5
    ref = O.dedisperse(fb, off, nt)
    rms = np.sqrt(np.mean(ref ** 2))
    plan = vf.DedispPlan(off)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.full((ndm, nt + 3), 7.0, device="cuda")  # padded rows: nothing past nt is written
    got, st = plan(torch.from_numpy(ring).cuda(), nt, storage=storage, row0=row0, row_mask=R - 1 if R else 0xFFFFFFFF,
                   nrows_valid=rows, out=out, d_err=err, stats=nt > 1, **kw)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    x = got.cpu().numpy()
    assert (x[:, nt:] == 7.0).all()
    e = np.max(np.abs(x[:, :nt] - ref)) / rms
    print(f"storage {storage} weighted {weighted}: err/rms {e:.2e}")
    assert e <= 1e-5
    if nt > 1:
        want = O.calcstats_dm(x[:, :nt])
        assert np.array_equal(st["frb"].cpu().numpy(), want["frb"])
        assert np.array_equal(st["argmax"].cpu().numpy(), want["argmax"])
        assert np.allclose(st["peak"].cpu().numpy(), want["peak"], rtol=1e-5)
        assert np.allclose(st["sigma"].cpu().numpy(), want["sigma"], rtol=1e-6)


def test_band_kernel_is_the_automatic_choice_and_agrees_with_the_others(vf, O):
    """AUTO against the pattern, register and staged kernels on the same input."""
    import torch
    off, ring, _, rows = _case(70, 320, 1500, 8.0, 3, 0, 0, 0)
    plan = vf.DedispPlan(off)
    x = torch.from_numpy(ring).cuda()
    base, _ = plan(x, 1500, nrows_valid=rows)
    rms = float(base.pow(2).mean().sqrt())
    for v in (vf.DD_STAGED, vf.DD_REG4, vf.DD_PAT4, vf.DD_PAT2, vf.DD_DIRECT):
        plan.set_variant(0, v)
        other, _ = plan(x, 1500, nrows_valid=rows)
        assert float((other - base).abs().max()) <= 1e-5 * rms
    # an infinity in one sample reaches exactly the sums that take it
    x[7, 900] = float("inf")
    plan.set_variant(0, vf.DD_AUTO)
    got, _ = plan(x, 1500, nrows_valid=rows)
    hit = torch.isinf(got).cpu().numpy()
    want = np.zeros_like(hit)
    for d in range(70):
        t = 900 - off[d, 7]
        if 0 <= t < 1500:
            want[d, t] = True
    assert np.array_equal(hit, want) and bool(torch.isfinite(got[~torch.from_numpy(want).cuda()]).all())


@pytest.mark.parametrize("ndm,nt,row0", [(1, 33, 0), (2, 5000, 1800), (64, 700, 7), (65, 300, 0)])
def test_sigma_form_sizes(vf, O, ndm, nt, row0):
    """Sigma form at the sizes where its kernel or samples per lane change, off
    the alignment and across the ring's end: mean <= 1e-5 of the rms, sigma <=
    1e-5 relative (FP32 sums of squares, as before)."""
    import torch
    R = 8192 if row0 > 1000 else 0
    if R:
        row0 = R - row0
    off, ring, fb, rows = _case(ndm, 200, nt, 30.0, 9, 0, row0, R)
    ave, sig = O.dedisperse_sigma(fb, off, nt)
    out = torch.full((2, ndm, nt), 7.0, device="cuda")
    vf.DedispPlan(off)(torch.from_numpy(ring).cuda(), nt, row0=row0, row_mask=R - 1 if R else 0xFFFFFFFF,
                       nrows_valid=rows, out=out[0], sigma_out=out[1], stats=False)
    got = out.cpu().numpy()
    assert np.max(np.abs(got[0] - ave)) <= 1e-5 * np.sqrt(np.mean(ave ** 2))
    assert np.max(np.abs(got[1] - sig) / sig) <= 1e-5
