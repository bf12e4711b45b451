"""The FP64 batched step with every split of the levels over CTAs that small grids lead to (1 to 8 levels a
CTA, a last CTA with fewer, tracer counts whose batches do and do not chain from level to level),
against the plain FP64 step.  Both are FP64 and differ in operation order and contraction only: 1e-11
normwise, the bound of the FP64 variant's other comparisons."""
import numpy as np
import pytest

from cases import case, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("glevel,rlevel,kall,ntr", [(3, 0, 4, 1), (4, 0, 9, 4), (4, 1, 12, 3), (5, 0, 21, 8), (5, 1, 44, 2),
                                                    (6, 0, 13, 5)])
def test_fast64_step_equals_plain_step(built, glevel, rlevel, kall, ntr):
    import torch
    from icoatmosbenchmark_v1_b200 import api
    c = case(glevel, rlevel, kall, ntr)
    g, f = c["grid"], c["fields"]
    dev = lambda d: {k: torch.as_tensor(v, device="cuda").contiguous() for k, v in d.items()}  # noqa: E731
    ctx = api.IcoAdv(glevel, rlevel, kall - 2)
    try:
        ctx.set_grid(g)
        G = {k: v.copy() for k, v in c["state"].items()}
        ctx.advect_step(c["dt"], G["rhog"], G["rhog_pl"], G["rhogq"], G["rhogq_pl"], f["rhogvx"], f["rhogvx_pl"],
                        f["rhogvy"], f["rhogvy_pl"], f["rhogvz"], f["rhogvz_pl"], f["rhogw"], f["rhogw_pl"])
        a, fd = dev(c["state"]), dev(f)
        for shape in (0, 5):
            b = {k: torch.full_like(v, float("nan")) for k, v in a.items()}
            ctx.fast_set_shape(shape)
            ctx.advect_fast64_dev(c["dt"], a, b, fd)
            torch.cuda.synchronize()
            for k in G:
                got = b[k].cpu().numpy()
                if k.endswith("_pl"):  # the ring slots and the centre
                    assert np.isfinite(got).all()
                assert rel_err(got, G[k]) <= 1e-11, (shape, k)
    finally:
        ctx.close()
