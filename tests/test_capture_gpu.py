"""Stage calls recorded into a CUDA graph and replayed on new input give the bits of the
plain call: the kernels with clusters, with overlapping launches, and the short ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _replayed(call, refill, outs):
    import torch
    call()  # (tables to the device, limits of shared memory)
    refill(1)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    refill(2)
    g.replay()
    torch.cuda.synchronize()
    got = [o.clone() for o in outs]
    refill(2)
    call()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, outs))


@pytest.mark.parametrize("ndm,storage", [(3, 0), (48, 0), (48, 1), (300, 2)])
def test_dedispersion(vf, O, ndm, storage):
    import torch
    off, _ = O.delay_table(np.linspace(0, 30.0, ndm).astype(np.float32), 384.0, 0.25, 1e-3, 256)
    nt, dt = 900, (torch.float32, torch.float16, torch.int8)[storage]
    plan = vf.DedispPlan(off)
    fb = torch.empty((256, (nt + plan.max_delay + 15) // 16 * 16), dtype=dt, device="cuda")
    out = torch.zeros((ndm, nt), device="cuda")
    assert plan.kernel(storage)[0] == (vf.DD_FEW if ndm == 3 else vf.DD_BAND)

    def refill(seed):
        fb.copy_((torch.randn(fb.shape, generator=torch.Generator().manual_seed(seed)) * 20).to(dt))

    _replayed(lambda: plan(fb, nt, storage=storage, uniform_scale=0.5 if storage else 0.0, stats=False, out=out), refill,
              [out])


@pytest.mark.parametrize("rows", [16, 200])  # a cluster per row, and a CTA per row
def test_channeliser_and_statistics(vf, rows):
    import torch
    L = vf.layout(nave=4, muoslowfreq=384.0)
    n = rows * 4 * 12500 // 5000 + 2
    frames = torch.empty(n * 10064, dtype=torch.uint8, device="cuda")
    s0 = torch.arange(n, dtype=torch.int64, device="cuda") * 10064 + 32
    s1 = s0 + 5032
    fb = torch.zeros((rows, L.nchanout), device="cuda")
    cm = torch.zeros((L.nchanout, (rows + 15) // 16 * 16), device="cuda")

    def refill(seed):
        frames.copy_(torch.randint(0, 256, frames.shape, dtype=torch.uint8, generator=torch.Generator().manual_seed(seed)))

    def call():
        vf.channelise(frames, s0, s1, 0, rows, L, out=fb)
        vf.bandpass(fb, out=cm)
        vf.subtract_zero(cm, nrows=rows)
        vf.subtract_bp_full(cm, nrows=rows)

    _replayed(call, refill, [fb, cm])
