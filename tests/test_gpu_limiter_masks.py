"""The horizontal limiter's Qout takes a shorter form where every mask around a cell is 0 or 1 and
agrees with its Courant numbers.  Both forms, in one call, against the oracle: the masks of the step,
masks that contradict the Courant numbers (an outflow mask on an inflow face, whose bound is +-BIG),
and fractional ones.  The operations are the oracle's, so the tolerance is zero."""
import numpy as np
import pytest

from cases import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("glevel,rlevel,kall", [(5, 0, 6), (3, 1, 5)])
@pytest.mark.parametrize("masks", ["flipped", "fractional"])
def test_qout_with_masks_of_every_kind(built, glevel, rlevel, kall, masks):
    from icoatmosbenchmark_v1_b200 import api
    from oracle import oracle as O
    c = case(glevel, rlevel, kall)
    g = c["grid"]
    rng = np.random.default_rng(3)
    cm, cm_pl = c["cm"].copy(), c["cm_pl"].copy()
    some = rng.random(cm.shape) < 0.05
    cm[some] = 1.0 - cm[some] if masks == "flipped" else rng.random(int(some.sum()))
    args = (c["dims"], g.have_sgp, c["qa"], c["qa_pl"], c["q"], c["q_pl"], c["d"], c["d_pl"], c["ch"], c["ch_pl"], cm,
            cm_pl)
    ra, rap, rqo, rqop = O.horizontal_limiter(*args, topo=c["topo"])
    qa, qa_pl = c["qa"].copy(), c["qa_pl"].copy()
    qo, qop = np.zeros_like(rqo), np.zeros_like(rqop)
    ctx = api.IcoAdv(glevel, rlevel, kall - 2)
    try:
        ctx.horizontal_limiter_thuburn(qa, qa_pl, c["q"], c["q_pl"], c["d"], c["d_pl"], c["ch"], c["ch_pl"], cm, cm_pl,
                                       qo, qop)
    finally:
        ctx.close()
    for got, ref in ((qa, ra), (qa_pl, rap), (qo, rqo), (qop, rqop)):
        np.testing.assert_array_equal(got, ref)
