"""The plain FP64 step where its launches can go wrong: regions of 1 to 64 cells a side (partial
tiles of both tile widths, regions with nothing but boundary cells), the smallest and largest
level counts, and tracer counts on both sides of a pair and of a group.  The step keeps the
reference's operation sequence, so the tolerance against the oracle is zero."""
import numpy as np
import pytest

from cases import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("glevel,rlevel,kall,ntr", [(1, 1, 4, 1), (1, 0, 5, 2), (2, 1, 6, 3), (3, 2, 7, 9), (4, 0, 4, 8),
                                                    (4, 1, 13, 17), (5, 0, 9, 16), (6, 0, 5, 3), (3, 0, 128, 2)])
def test_plain_step_every_tile_form(built, glevel, rlevel, kall, ntr):
    from icoatmosbenchmark_v1_b200 import api
    from oracle import oracle as O
    c = case(glevel, rlevel, kall, ntr)
    g, f = c["grid"], c["fields"]
    S = {k: v.copy() for k, v in c["state"].items()}
    G = {k: v.copy() for k, v in c["state"].items()}
    ctx = api.IcoAdv(glevel, rlevel, kall - 2)
    try:
        ctx.set_grid(g)
        for _ in range(2):
            O.step(c["dims"], g.have_sgp, c["topo"], c["dt"], S, f, g.arrays, nthreads=8)
            ctx.advect_step(c["dt"], G["rhog"], G["rhog_pl"], G["rhogq"], G["rhogq_pl"], f["rhogvx"], f["rhogvx_pl"],
                            f["rhogvy"], f["rhogvy_pl"], f["rhogvz"], f["rhogvz_pl"], f["rhogw"], f["rhogw_pl"])
        for k in S:
            np.testing.assert_array_equal(G[k], S[k], err_msg=k)
    finally:
        ctx.close()
