"""Short columns of the marching kernels: depths around the chunk lengths of
2 to 16 planes that small grids take, with the wall model at the bottom, the
top or both (the packed wall planes of the mixed path), uniform and stretched
z, even and odd rows, against the oracle (its transforms take the factors 2, 3
and 5)."""
import pytest

from conftest import rel
from gpu_elmm_b200 import lib as L
from gpu_elmm_b200.config import (BC_FREESLIP, BC_NOSLIP, BC_PERIODIC, PREC_FP64, PREC_MIXED, grid_of, make_config)
from gpu_elmm_b200.workloads import interiors, log_profile_state, stretched_zw
from oracle import Oracle

pytestmark = pytest.mark.gpu

P = BC_PERIODIC
WALLS = {"bottom": (BC_NOSLIP, BC_FREESLIP), "top": (BC_FREESLIP, BC_NOSLIP), "both": (BC_NOSLIP, BC_NOSLIP)}


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("stretched", [False, True])
@pytest.mark.parametrize("walls", sorted(WALLS))
@pytest.mark.parametrize("n", [(36, 10, 4), (15, 9, 5), (45, 8, 17)])
def test_columns_and_wall_planes(n, walls, stretched, precision):
    btype = (P, P, P, P) + WALLS[walls]
    zW = stretched_zw(n[2], 0.5, 1.1) if stretched else None
    cfg = make_config(*n, btype=btype, precision=precision, zW=zW)
    g = grid_of(cfg)
    o = Oracle(make_config(*n, btype=btype, zW=zW))
    o.set_state(*log_profile_state(g, seed=n[0], zW=zW))
    o.project(1.0)
    d = L.Domain(cfg)
    d.upload(*o.state())
    o.step(2)
    d.step(2)
    for a, b, name in zip(interiors(g, *d.download())[:3], interiors(g, *o.state())[:3], "UVW"):
        assert rel(a, b) < (1e-12 if precision == PREC_FP64 else 1e-5), name
