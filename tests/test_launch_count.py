"""launch_count against the kernels that really start, counted by the fake CUDA runtime: the three kernels and the halo
fills, with and without pole arrays, the plain step and its adjoint."""
from test_cuda_errors import child  # noqa: F401

COUNT = r"""
g = Grid(2, 0, 6)
out = {}

def count(name, ctx, call, *args):
    fake.fake_reset()
    n0 = ctx.launch_count
    call(*args)
    out[name] = [ctx.launch_count - n0, calls("cudaLaunchKernel")]

def entries(tag, ctx, L):
    K, G = ctx.sizes.kall, ctx.sizes.gall
    r = lambda *lead: np.ones(lead + (L, K, G))
    p = lambda *lead: np.ones(lead + (2, K, 6))
    count(tag + "flux", ctx, ctx.horizontal_flux, r(6), p(), r(3, 3), p(3), r(), p(), r(), p(), r(), p(), r(), p(), 1.0)
    lim = [r(6), p(), r(), p(), r(), p(), r(6), p(), r(3), p(), r(2), p(2)]
    count(tag + "limiter, Qout given", ctx, ctx.horizontal_limiter_thuburn, *lim, r(2), p(2))
    if tag == "grid ":
        count(tag + "limiter", ctx, ctx.horizontal_limiter_thuburn, *lim, None, None)
    count(tag + "vertical limiter", ctx, ctx.vertical_limiter_thuburn, r(), p(), r(), p(), r(), p(), r(2), p(2))
    return r, p

geo = g.geometry()
for poles in (False, True):
    ctx = api.IcoAdv.regions(g.gall_1d, g.kall, g.kmin, g.kmax, 1, poles, g.have_sgp[:1])
    ctx.set_geometry(*[geo[k] if k.endswith("_pl") else np.ascontiguousarray(geo[k][..., :1, :])
                       for k in ("GRD_xr", "GRD_xr_pl", "GMTR_p", "GMTR_p_pl", "GMTR_t", "GMTR_t_pl", "GMTR_a", "GMTR_a_pl")])
    entries("regions, poles " if poles else "regions ", ctx, 1)
    ctx.close()
ctx = api.IcoAdv(2, 0, 4)
ctx.set_grid(g)
r, p = entries("grid ", ctx, ctx.sizes.lall)
count("fill", ctx, ctx.COMM_data_transfer, r(3), p(3))
count("fill with poles", ctx, ctx.COMM_var, r(3), p(3))
state = lambda n: dict(rhog=r(), rhog_pl=p(), rhogq=r(n), rhogq_pl=p(n))
fields = {k: (p() if k.endswith("_pl") else r()) for k in api.FIELD_KEYS}
wind = lambda: {k: (p() if k.endswith("_pl") else r()) for k in api.WIND_KEYS}
for n in (1, 9):
    s = state(n)
    count(f"step, {n}", ctx, ctx.advect_step, 1.0, *[s[k] for k in api.STATE_KEYS], *[fields[k] for k in api.FIELD_KEYS])
    count(f"adjoint, {n}", ctx, ctx.advect_step_adjoint, 1.0, s, fields, state(n), wind())
print(json.dumps(out))
"""


def test_launch_count_is_what_was_launched(child):  # noqa: F811
    out = child(COUNT)
    assert len(out) == 16
    wrong = {k: v for k, v in out.items() if v[0] != v[1] or v[1] < 1}
    assert not wrong, wrong
