"""Which kernel a dedispersion call runs, asked of the plan and shown by its launches:
the automatic choice's own kernels at the edges of their ranges, and explicit ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _launched(f):
    import torch
    from torch.profiler import ProfilerActivity, profile
    f()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    return [e.name for e in p.events() if "vfrb::" in e.name]


@pytest.mark.parametrize("ndm,spacing,sigma,storage,want,name", [
    (1, "even", False, 0, "FEW", "k_dedisp_few"), (16, "even", False, 1, "FEW", "k_dedisp_few"),
    (16, "uneven", False, 2, "FEW", "k_dedisp_few"), (17, "even", False, 0, "BAND", "k_dedisp_band"),
    (90, "even", False, 1, "BAND", "k_dedisp_band"), (201, "even", False, 2, "BAND", "k_dedisp_band"),
    (64, "even", True, 0, "FEW", "k_dedisp_few"), (65, "even", True, 0, "STAGED", "k_dedisperse"),
    (40, "uneven", False, 0, None, "k_dedisp_pat"), (40, "uneven", False, 2, "STAGED", "k_dedisperse"),
    (48, "even PAT2", False, 0, "PAT2", "k_dedisp_pat"), (48, "even REG4", False, 0, "REG4", "k_dedisp_reg")])
def test_the_query_names_the_kernel_that_runs(vf, O, ndm, spacing, sigma, storage, want, name):
    import torch
    rng = np.random.default_rng(2)
    dms = np.linspace(0, 20.0, ndm) if "even" == spacing[:4] else np.sort(rng.uniform(0, 10.0, ndm))
    off, _ = O.delay_table(dms.astype(np.float32), 384.0, 0.25, 1e-3, 256)
    nt = 600
    plan = vf.DedispPlan(off)
    if " " in spacing:
        plan.set_variant(storage, getattr(vf, "DD_" + spacing.split()[1]))
    dt = (torch.float32, torch.float16, torch.int8)[storage]
    fb = torch.ones((256, (nt + plan.max_delay + 15) // 16 * 16), device="cuda").to(dt)
    kw = dict(storage=storage, stats=False, out=torch.empty((ndm, nt), device="cuda"))
    if storage:
        kw["uniform_scale"] = 1.0
    if sigma:
        kw["sigma_out"] = torch.empty((ndm, nt), device="cuda")
    kernel, launches = plan.kernel(storage, sigma)
    ran = _launched(lambda: plan(fb, nt, **kw))
    if want is None:  # the variant that the plan reports for such calls
        assert kernel == plan.variant(storage) and kernel in (vf.DD_PAT4, vf.DD_PAT2)
    else:
        assert kernel == getattr(vf, "DD_" + want)
    assert len(ran) == launches and all("vfrb::" + name + "<" in n or "vfrb::" + name + "(" in n for n in ran), ran
