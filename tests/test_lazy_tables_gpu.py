"""The pattern and register kernels' tables of a plan whose automatic kernel needs none:
made when a variant is first chosen, by whichever thread comes first and beside a
capture under way."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(vf, O):
    import torch
    off, _ = O.delay_table(np.linspace(0, 20.0, 96).astype(np.float32), 384.0, 0.25, 1e-3, 256)
    fb = torch.empty((256, 1600), device="cuda").normal_(generator=torch.Generator("cuda").manual_seed(3))
    return off, fb, 1600 - int(off.max()) - 16


def _series(vf, plan, variant, fb, nt):
    plan.set_variant(vf.F32, variant)
    return plan(fb, nt, stats=False)[0].cpu()


def test_choosing_a_variant_inside_a_capture(vf, O):
    import torch
    off, fb, nt = _case(vf, O)
    want = _series(vf, vf.DedispPlan(off), vf.DD_PAT4, fb, nt)
    plan = vf.DedispPlan(off)
    out = torch.zeros((96, nt), device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.set_variant(vf.F32, vf.DD_PAT4)
        plan(fb, nt, stats=False, out=out)
    g.replay()
    assert torch.equal(out.cpu(), want)


def test_threads_that_choose_variants_at_once(vf, O):
    import torch
    off, fb, nt = _case(vf, O)
    variants = [vf.DD_REG4, vf.DD_REG2, vf.DD_PAT4, vf.DD_PAT2]
    one = vf.DedispPlan(off)
    want = [_series(vf, one, v, fb, nt) for v in variants]
    auto = vf.DedispPlan(off)(fb, nt, stats=False)[0].cpu()
    assert len({w.numpy().tobytes() for w in want}) > 1  # the kernels' sums differ in their order
    for _ in range(5):
        plan = vf.DedispPlan(off)
        gate, errors = threading.Barrier(8), []

        def choose(i):
            try:
                torch.cuda.set_device(0)
                gate.wait()
                plan.set_variant(vf.F16, variants[i % 4])  # (the FP32 calls meanwhile stay automatic)
                with torch.cuda.stream(torch.cuda.Stream()):
                    if not torch.equal(plan(fb, nt, stats=False)[0].cpu(), auto):
                        errors.append("automatic call")
            except Exception as e:  # noqa: BLE001
                errors.append(repr(e))

        th = [threading.Thread(target=choose, args=(i,)) for i in range(8)]
        [t.start() for t in th]
        [t.join() for t in th]
        assert not errors
        for v, w in zip(variants, want):
            assert torch.equal(_series(vf, plan, v, fb, nt), w)
