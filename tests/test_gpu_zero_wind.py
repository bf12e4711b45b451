"""Vertical wind of exactly zero through interior faces.  The vertical limiter takes a face's inflow side from
the sign of its Courant number -w dt / (rho dz), which w = +0.0 makes -0.0 and w = -0.0 makes +0.0.  The plain
step is compared with the oracle bit for bit, its adjoint at 1e-11 normwise and the FP64 batched step with the
plain one at 1e-11, the bounds of their other comparisons."""
import numpy as np
import pytest

from cases import case, rel_err
from test_gpu_adjoint import STATE, WIND, _close, _ctx, _noisy

pytestmark = pytest.mark.gpu

WHERE = ("lower", "upper", "single", "scattered")


def _zeroed(f, where, zero):
    """The fields with rhogw (and its pole values) set to `zero` at some half levels."""
    rng = np.random.default_rng(3)
    out = dict(f)
    for k in ("rhogw", "rhogw_pl"):
        w = out[k] = f[k].copy()
        K = w.shape[1]  # (lall, K, gall): half level h lies below level h, faces 1 .. K - 1
        if where == "lower":
            w[:, :K // 2] = zero
        elif where == "upper":
            w[:, K // 2:] = zero
        elif where == "single":
            w[:, 2::4] = zero
        else:
            w[rng.random(w.shape) < 0.3] = zero
    return out


def _step(ctx, dt, G, f):
    ctx.advect_step(dt, G["rhog"], G["rhog_pl"], G["rhogq"], G["rhogq_pl"], f["rhogvx"], f["rhogvx_pl"], f["rhogvy"],
                    f["rhogvy_pl"], f["rhogvz"], f["rhogvz_pl"], f["rhogw"], f["rhogw_pl"])


@pytest.mark.parametrize("zero", [0.0, -0.0])
@pytest.mark.parametrize("where", WHERE)
@pytest.mark.parametrize("glevel,rlevel,kall,ntr", [(4, 0, 12, 3), (5, 1, 9, 2)])
def test_plain_step_equals_oracle(built, glevel, rlevel, kall, ntr, where, zero):
    from oracle import oracle as O
    c = case(glevel, rlevel, kall, ntr)
    g, f = c["grid"], _zeroed(c["fields"], where, zero)
    S = {k: v.copy() for k, v in c["state"].items()}
    G = {k: v.copy() for k, v in c["state"].items()}
    ctx = _ctx(g)
    try:
        for _ in range(2):
            O.step(c["dims"], g.have_sgp, c["topo"], c["dt"], S, f, g.arrays, nthreads=8)
            _step(ctx, c["dt"], G, f)
    finally:
        ctx.close()
    for k in S:
        np.testing.assert_array_equal(G[k], S[k], err_msg=k)


@pytest.mark.parametrize("zero", [0.0, -0.0])
@pytest.mark.parametrize("where", WHERE)
def test_adjoint_equals_oracle(built, where, zero):
    from oracle import oracle as O
    c = case(4, 0, 12, 3)
    g, f = c["grid"], _zeroed(c["fields"], where, zero)
    S0 = _noisy(c["state"])
    rng = np.random.default_rng(8)
    w = {k: rng.standard_normal(v.shape) for k, v in S0.items()}
    ref = {k: v.copy() for k, v in w.items()}
    ref_w = {k: np.zeros_like(f[k]) for k in WIND}
    O.step_adjoint(c["dims"], g.have_sgp, c["topo"], c["dt"], S0, f, g.arrays, ref, ref_w)
    got = {k: v.copy() for k, v in w.items()}
    got_w = {k: np.zeros_like(f[k]) for k in WIND}
    ctx = _ctx(g)
    try:
        ctx.advect_step_adjoint(c["dt"], S0, f, got, got_w)
    finally:
        ctx.close()
    for k in STATE:
        _close(got[k], ref[k], 1e-11, k)
    for k in WIND:
        _close(got_w[k], ref_w[k], 1e-11, k)


@pytest.mark.parametrize("zero", [0.0, -0.0])
@pytest.mark.parametrize("where", WHERE)
def test_fast64_step_equals_plain_step(built, where, zero):
    import torch
    c = case(4, 0, 12, 3)
    g, f = c["grid"], _zeroed(c["fields"], where, zero)
    ctx = _ctx(g)
    try:
        G = {k: v.copy() for k, v in c["state"].items()}
        _step(ctx, c["dt"], G, f)
        a = {k: torch.as_tensor(v, device="cuda").contiguous() for k, v in c["state"].items()}
        fd = {k: torch.as_tensor(v, device="cuda").contiguous() for k, v in f.items()}
        b = {k: torch.empty_like(v) for k, v in a.items()}
        ctx.advect_fast64_dev(c["dt"], a, b, fd)
        torch.cuda.synchronize()
        for k in G:
            assert rel_err(b[k].cpu().numpy(), G[k]) <= 1e-11, k
    finally:
        ctx.close()
