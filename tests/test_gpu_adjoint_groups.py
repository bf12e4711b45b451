"""The step's adjoint where its launches can go wrong: tracer counts past a group of 8, regions of 1 to
32 cells a side (both tile widths, partial tiles, regions of boundary cells only) and the smallest
level counts, against the oracle's adjoint.  1e-11 normwise, the bound of the other adjoint
comparisons: both sides sum the same terms, in another order."""
import numpy as np
import pytest

from cases import case
from test_gpu_adjoint import STATE, WIND, _close, _ctx, _noisy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("glevel,rlevel,kall,ntr", [(1, 1, 4, 2), (2, 0, 5, 9), (3, 1, 7, 8), (4, 0, 4, 17), (5, 0, 6, 10)])
def test_step_adjoint_groups_and_tiles(built, glevel, rlevel, kall, ntr):
    from oracle import oracle as O
    c = case(glevel, rlevel, kall, ntr)
    g, f = c["grid"], c["fields"]
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
