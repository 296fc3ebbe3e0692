"""Results at the sizes where a stage call changes its kernel, on both sides of each line,
against the FP64 oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(rows, nch, seed):
    return np.random.default_rng(seed).standard_normal((rows, nch)).astype(np.float32) * 2.0 + 5.0


@pytest.mark.parametrize("rows,ncol", [(7, 2), (1000, 16), (1023, 1023), (1024, 1024), (1025, 1025), (2048, 1024),
                                       (2500, 1024), (2500, 1025), (9000, 4096)])
def test_chan_stats_lines(vf, O, rows, ncol):
    """Blocks of 1024 rows, all whole, and every other kind.  FP64 sums of values of
    order 10, stored as float: 1e-6."""
    import torch
    nch, nblk = 41, -(-rows // ncol)
    if rows - (nblk - 1) * ncol == 1:
        nblk -= 1  # (a last block of one row has no variance)
    x = _rows(rows, nch, rows + ncol)
    x[rows // 2, 3] = 1e4
    a, s, o = vf.chan_stats(torch.from_numpy(np.ascontiguousarray(x.T)).cuda(), rows, ncol, nblk)
    a_r, s_r, o_r = O.calcstats_chan(x.astype(np.float64), ncol, nblk)
    assert np.allclose(a.cpu().numpy(), a_r, rtol=1e-6, atol=0)
    assert np.allclose(s.cpu().numpy(), s_r, rtol=1e-6, atol=1e-9)
    assert np.array_equal(o.cpu().numpy(), o_r)


@pytest.mark.parametrize("rows,ncol,nch", [(6, 2, 70), (446, 223, 300), (448, 224, 300), (300, 223, 64), (700, 224, 65),
                                           (223, 5000, 257), (224, 5000, 256)])
def test_chan_sk_lines(vf, O, rows, ncol, nch):
    """Spectral kurtosis of blocks shorter and longer than a CTA's sets of rows want,
    ragged last blocks and channel groups: FP64, stored as float.  SK - 1 is a small
    difference of terms of order 1 times (m nsum + 1) / (m - 1): 1e-6 of the terms."""
    import torch
    x = _rows(rows, nch, rows)
    n = -(-rows // ncol)
    got = vf.chan_sk(torch.from_numpy(x).cuda(), ncol, n, 20).cpu().numpy()
    for k in range(n):
        b = x[k * ncol:(k + 1) * ncol].astype(np.float64)
        m = len(b)
        if m == 1:
            continue
        f = (m * 20 + 1) / (m - 1)
        assert np.allclose(got[k], f * (m * (b * b).sum(0) / b.sum(0) ** 2 - 1), rtol=1e-6, atol=1e-12 * f)


@pytest.mark.parametrize("rows", [2, 5, 255, 256, 257, 1024, 1025, 1028, 2047, 2048, 2049, 2052, 6144, 6145, 6148, 8191,
                                  8192, 8196])
@pytest.mark.parametrize("row0", [0, 3])
def test_subtract_bp_full_lines(vf, O, rows, row0):
    """Whole-block bandpass in registers, in quads and in shared memory, at the edges of
    each, with the rows aligned or not: one float rounding of the values."""
    import torch
    nch = 128
    x = _rows(rows, nch, rows) - 5.0  # (the reference's first mean divides by the channels)
    x[rows // 3, 2] += 50.0  # clipped
    buf = torch.full((nch, (row0 + rows + 7) // 4 * 4), 7.0, device="cuda")
    buf[:, row0:row0 + rows] = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    vf.subtract_bp_full(buf, nrows=rows, row0=row0)
    ref = O.subtract_bp_full(x.astype(np.float64))
    got = buf.cpu().numpy()
    assert (got[:, :row0] == 7.0).all() and (got[:, row0 + rows:] == 7.0).all()
    want = ref.T
    assert np.array_equal(np.isnan(got[:, row0:row0 + rows]), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.max(np.abs(got[:, row0:row0 + rows] - want)[ok], initial=0.0) <= 1e-6 * np.abs(x).max()


@pytest.mark.parametrize("nch,rows", [(2, 167), (2, 168), (3, 5000), (64, 5375), (64, 5376), (192, 16127), (192, 16128),
                                      (193, 16300), (193, 2**19)])
@pytest.mark.parametrize("row0", [0, 5])
def test_subtract_zero_lines(vf, O, nch, rows, row0):
    """Zero-DM with a thread per row for many rows beside the channels, and with clusters:
    one float rounding of the values."""
    import torch
    x = _rows(rows, nch, rows + nch)
    x[rows // 3] += 20.0  # a broadband row
    x[rows // 2, 1] += 500.0  # clipped
    buf = torch.full((nch, (row0 + rows + 7) // 4 * 4), 7.0, device="cuda")
    buf[:, row0:row0 + rows] = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    vf.subtract_zero(buf, nrows=rows, row0=row0)
    got = buf.cpu().numpy()
    assert (got[:, :row0] == 7.0).all() and (got[:, row0 + rows:] == 7.0).all()
    assert np.max(np.abs(got[:, row0:row0 + rows] - O.subtract_zero(x).T)) <= 1e-6 * np.abs(x).max()


@pytest.mark.parametrize("nch,rows", [(1, 1), (2, 33), (12, 1000), (13, 1000), (12, 32 * 65535), (12, 32 * 65535 + 1), (64, 64),
                                      (65, 129)])
def test_transpose_lines(vf, nch, rows):
    """Small and large tiles, and the rows that a grid of the small ones has: equal bits."""
    import torch
    x = torch.randn((nch, rows + 3), device="cuda")
    assert torch.equal(vf.fb_to_time_major(x, nrows=rows, row0=2), x[:, 2:2 + rows].t())


@pytest.mark.parametrize("nt", [1, 2, 100, 191, 192, 193])
@pytest.mark.parametrize("width", [1, 2, 64])
def test_boxcar_short_series(vf, O, nt, width):
    """Series around the shortest that go through tiles, with sums that are exact."""
    import torch
    x = np.round(np.random.default_rng(nt).standard_normal((33, nt)) * 64).astype(np.float32) / 64
    x[5, nt // 2:nt // 2 + 7] += 3.0
    x[0] = 0.5  # equal samples: the smaller width, then the earlier start
    ave, sig = x.mean(axis=1).astype(np.float32), np.maximum(x.std(axis=1), 0.25).astype(np.float32)
    best, start, w = O.boxcar_best(x, ave, sig, width)
    snr, s0, w0 = vf.boxcar(torch.from_numpy(x).cuda(), torch.from_numpy(ave).cuda(), torch.from_numpy(sig).cuda(), width)
    assert np.array_equal(w0.cpu().numpy(), w) and np.array_equal(s0.cpu().numpy(), start)
    assert np.allclose(snr.cpu().numpy(), best, rtol=1e-6, atol=1e-9)
