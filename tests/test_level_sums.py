"""The (0,0) mode of the pressure from the level sums of W: rows of whole
16-byte vectors and not, sums from W2 itself and from the forward x
transform's tiles (W2 of more than 5.2 MB and rows that fill a level's tiles, or
in the generic form nearly so; and rows that do not), levels past the tiled z
solve, walls and periodic z, against the oracle."""
import numpy as np
import pytest

from conftest import rel
from gpu_elmm_b200 import lib as L
from gpu_elmm_b200.config import (BC_FREESLIP, BC_NOSLIP, BC_PERIODIC, PREC_FP64, PREC_MIXED, grid_of, make_config)
from gpu_elmm_b200.workloads import interiors, log_profile_state
from oracle import Oracle

pytestmark = pytest.mark.gpu

P = BC_PERIODIC
# the mixed path's pressure: each stage's projection turns the rounding of
# the stored velocity deviations (at most 0.4 m/s) over one cell into pressure
# through its coefficient 2 alpha dt, and the pressure sums the stages' increments
P_MIXED_ABS = 2.0 ** -24 * 0.4 * sum(1.0 / (2.0 * a * 0.02) for a in (4.0 / 15.0, 1.0 / 15.0, 1.0 / 6.0))


# the double integral of the levels' divergence: changes of unit roundoff in
# the oracle's own velocity change its pressure by 0.3 to 1.2e-15 nz^2 of it
P_FP64_REL = 4 * 1.2e-15

BOTTOM, TOP, PERIODIC = (BC_NOSLIP, BC_FREESLIP), (BC_FREESLIP, BC_NOSLIP), (P, P)


@pytest.mark.parametrize("n,z", [((8, 6, 5), BOTTOM), ((8, 6, 5), PERIODIC), ((9, 5, 4), TOP), ((64, 72, 6), BOTTOM),
                                 ((20, 75, 5), PERIODIC), ((12, 10, 220), PERIODIC), ((12, 10, 300), BOTTOM),
                                 ((4, 4, 440), TOP), ((64, 72, 300), BOTTOM), ((81, 75, 220), PERIODIC),
                                 ((75, 64, 280), TOP), ((64, 64, 176), BOTTOM), ((64, 128, 130), PERIODIC), ((256, 125, 45), BOTTOM),
                                 ((75, 250, 80), TOP)])
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
def test_step_follows_the_oracle(n, z, precision):
    btype = (P, P, P, P) + z
    cfg = make_config(*n, btype=btype, precision=precision)
    g = grid_of(cfg)
    o = Oracle(make_config(*n, btype=btype))
    o.set_state(*log_profile_state(g, seed=n[2]))
    o.project(1.0)
    d = L.Domain(cfg)
    d.upload(*o.state())
    o.step(1)
    d.step(1)
    for a, b, name in zip(interiors(g, *d.download()), interiors(g, *o.state()), "UVWP"):
        if name != "P":
            assert rel(a, b) < (1e-12 if precision == PREC_FP64 else 1e-5), name
        elif precision == PREC_FP64:
            assert rel(a, b) < max(1e-11, P_FP64_REL * n[2] ** 2)
        else:
            # two roundings of W meet in a level's flux: its own and the level's below
            assert float(np.abs(a - b).max()) < 2 * P_MIXED_ABS * max(1.0, n[2] / 64)


# Both kinds of x transform that leave the sums of their tiles.  A row of W
# repeats (1, e, -1, e) with 1 + e = 1 in FP32:
# the mean e / 2 of a level survives only if every value is widened before it
# is added.  Away from the walls, where the rest of the divergence is, the
# pressure rises by its solution's e / 2 a level; the bound is the FP32
# rounding of a level's value, at most nz / 2 such rises from the mean.
@pytest.mark.parametrize("n", [(256, 256, 40), (300, 128, 40)])
def test_tile_sums_keep_every_bit(n):
    nx, ny, nz = n
    e = 2.0 ** -26
    rise = []
    for precision in (PREC_FP64, PREC_MIXED):
        cfg = make_config(*n, precision=precision, btype=(P, P, P, P) + BOTTOM)
        g = grid_of(cfg)
        st = [np.zeros(s) for s in (g.shape_u(), g.shape_v(), g.shape_w(), g.shape_p())]
        st[2][3:-3, 3:-3, 3:-3] = np.tile([1.0, e, -1.0, e], nx // 4)
        d = L.Domain(cfg)
        d.upload(*st)
        d.project(1.0)
        rise.append(np.diff(d.download()[3][2:-2, 2:-2, 2:-2].mean((1, 2)))[nz // 2 - 5:nz // 2 + 4])
        d.close()
    assert rel(rise[0], np.full(9, e / 2)) < 1e-9
    assert rel(rise[1], rise[0]) < 2 * nz / 2 * 2.0 ** -24
