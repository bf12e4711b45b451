"""The transposed flux kernels where a thread takes a full block of levels and the last block a few
(grids large enough for 8 levels a thread, level counts that 8 does not divide), against the oracle's
adjoint.  1e-11 normwise, the bound of the other adjoint comparisons: the same terms, in another order."""
import numpy as np
import pytest

from cases import case
from test_gpu_adjoint import STATE, WIND, _close, _ctx, _noisy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("glevel,rlevel,kall", [(5, 0, 60), (5, 1, 45), (6, 0, 13)])
def test_step_adjoint_level_blocks(built, glevel, rlevel, kall):
    from oracle import oracle as O
    c = case(glevel, rlevel, kall, 1)
    g, f = c["grid"], c["fields"]
    S0 = _noisy(c["state"])
    rng = np.random.default_rng(11)
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
