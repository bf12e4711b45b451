"""How horizontal_flux cuts a grid's levels into runs, one block each: a grid whose levels fit one wave (4 blocks on
each of 148 SMs) in runs of at most 12 takes that split, every other grid runs of 8.  Read off the launch that a
fake CUDA runtime sees; regions of 18 x 18 cells are three blocks each."""
import numpy as np
import pytest

from test_cuda_errors import child  # noqa: F401

FLUX = r"""
lall, kall = int(sys.argv[2]), int(sys.argv[3])
ctx = api.IcoAdv.regions(18, kall, 1 if kall < 3 else 2, max(kall - 1, 1), lall, False, np.zeros(lall, np.int32))
z = lambda *s: np.zeros(s)
ctx.set_geometry(*[z(*lead, lall, 324) if pl is None else z(*pl) for name, reg, pole in api.IcoAdv.GRID_KEYS[1:]
                   for lead, pl in ((reg, None), ((), pole))])
r = lambda *lead: z(*lead, lall, kall, 324)
p = lambda *lead: z(*lead, 2, kall, 6)
ctx.horizontal_flux(r(6), p(), r(3, 3), p(3), r(), p(), r(), p(), r(), p(), r(), p(), 1.0)
print(json.dumps(fake.fake_blocks()))
"""


@pytest.mark.parametrize("lall,kall,runs", [(10, 42, 14),   # 30 blocks a run: 19 runs fit a wave, so 3 levels
                                            (100, 12, 1),   # 300: one run fits
                                            (100, 13, 2),   # one run of 13 is too long: 8 + 5
                                            (197, 12, 1),   # 591, the largest grid with a run that fits
                                            (198, 5, 1),    # 594: none does
                                            (198, 8, 1), (198, 9, 2), (198, 12, 2), (198, 17, 3)])
def test_runs_of_levels(child, lall, kall, runs):  # noqa: F811
    assert child(FLUX, lall, kall) == 3 * lall * runs


@pytest.mark.gpu
@pytest.mark.parametrize("kall", [6, 9])
def test_grid_of_more_than_one_wave_equals_oracle(built, kall):
    """Fewer levels than a run of 8, and one more; the operations are the oracle's, so the tolerance is zero."""
    from cases import case
    from icoatmosbenchmark_v1_b200 import api
    c = case(7, 0, kall)
    f, ref = c["fields"], [c[k] for k in ("flx", "flx_pl", "xc", "xc_pl")]
    out = [np.full_like(a, np.nan) for a in ref]
    out[1][..., 0] = out[3][..., 0] = 0.0  # the centres' slots, which no face has
    ctx = api.IcoAdv(7, 0, kall - 2)
    try:
        ctx.set_grid(c["grid"])
        ctx.horizontal_flux(*out, *[f[k] for k in ("rhog", "rhog_pl") + api.WIND_KEYS], c["dt"])
    finally:
        ctx.close()
    for got, want in zip(out, ref):
        np.testing.assert_array_equal(got, want)
