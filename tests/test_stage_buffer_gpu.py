"""Pageable pushes whose size grows and shrinks within a stream, so that each staging
buffer is replaced while the other is in use: the same bits as one page-locked push."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_pageable_pushes_of_growing_size(vf):
    import torch
    from vlite_frb_b200 import synth
    buf = synth.make_vdif(synth.StreamSpec(duration=2.0, seed=5, pulses=[synth.Pulse(0.7, 6.0, 2.0, 40.0)]))
    raw = np.ascontiguousarray(buf.numpy())

    def run(pieces, stage=False):
        plan = vf.Plan(np.arange(0, 20.5, 0.5, dtype=np.float32), nave=2, muoslowfreq=384.0, mode=vf.MODE_STREAM,
                       outputs=vf.OUT_DEDISP, chunk_seconds=0.5)
        if stage:
            plan.stage_stream(0)
        for p in pieces:
            plan.push(0, p)
            if stage:
                plan.stage_stream(0)  # (again: nothing to do)
        plan.push(0, None)
        res = plan.drain()
        plan.close()
        return np.concatenate([r["dd"] for r in res], axis=1)

    want = run([torch.from_numpy(raw).pin_memory()])
    sizes = [5032, 5032 * 9 + 100, 5032 * 16 - 100, 5032 * 17, 5032 * 3, 5032 * 400 + 7, 5032 * 2, 5032 * 20000]
    at, pieces = 0, []
    while at < raw.size:
        n = sizes[len(pieces) % len(sizes)]
        pieces.append(raw[at:at + n].copy())
        at += n
    assert len(pieces) > len(sizes)
    got = run(pieces)
    assert got.shape == want.shape and np.array_equal(got, want)
    assert np.array_equal(run(pieces, stage=True), want)


def test_staging_ahead_refuses_other_streams(vf):
    plan = vf.Plan(np.arange(0, 2.0, 0.5, dtype=np.float32), nave=2, muoslowfreq=384.0, mode=vf.MODE_STREAM,
                   outputs=vf.OUT_DEDISP, chunk_seconds=0.5)
    plan.stage_stream(0)
    for s in (-1, 1):
        with pytest.raises(vf.VfrbError):
            plan.stage_stream(s)
    plan.close()
