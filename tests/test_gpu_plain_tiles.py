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


def test_plain_step_quotients_at_every_magnitude(built):
    """The step forms several quotients from one reciprocal where that is exact and divides where it
    is not: mixing ratios of 1e-309 (subnormal), 1e-300, 1e-240 and 1e250, and a zero tracer, against
    the oracle's divisions, bit for bit."""
    from icoatmosbenchmark_v1_b200 import api
    from oracle import oracle as O
    c = case(4, 0, 8, 5)
    g, f = c["grid"], c["fields"]
    scale = np.array([1e-309, 1e-300, 1e-240, 1e250, 0.0]).reshape(5, 1, 1, 1)
    S = {k: v * scale if k.startswith("rhogq") else v.copy() for k, v in c["state"].items()}
    G = {k: v.copy() for k, v in S.items()}
    ctx = api.IcoAdv(4, 0, 6)
    try:
        ctx.set_grid(g)
        O.step(c["dims"], g.have_sgp, c["topo"], c["dt"], S, f, g.arrays, nthreads=8)
        ctx.advect_step(c["dt"], G["rhog"], G["rhog_pl"], G["rhogq"], G["rhogq_pl"], f["rhogvx"], f["rhogvx_pl"],
                        f["rhogvy"], f["rhogvy_pl"], f["rhogvz"], f["rhogvz_pl"], f["rhogw"], f["rhogw_pl"])
        for k in S:
            np.testing.assert_array_equal(G[k], S[k], err_msg=k)
    finally:
        ctx.close()
