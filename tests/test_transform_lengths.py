"""The transforms of lengths without a register FFT: one, two and three
passes, odd lengths and lengths that leave a remainder of rows, columns or
16-byte vectors, and the register FFTs of 80 to 512, against the oracle."""
import numpy as np
import pytest

from conftest import rel
from gpu_elmm_b200 import lib as L
from gpu_elmm_b200.config import PREC_FP64, PREC_MIXED, grid_of, make_config
from gpu_elmm_b200.workloads import interiors, log_profile_state
from oracle import Oracle

pytestmark = pytest.mark.gpu


# lengths of 1 (4, 5, 16), 2 (18 = 6 x 3, 27, 45, 75, 250 -> 3) and 3 (270,
# 500, 900) passes; FP64 sums of n terms: 1e-12, FP32: 1e-5 (as the other
# Poisson checks of this repository)
@pytest.mark.parametrize("precision, tol", [(PREC_FP64, 1e-12), (PREC_MIXED, 1e-5)])
@pytest.mark.parametrize("n", [(4, 5, 6), (16, 18, 5), (27, 45, 7), (75, 20, 4), (250, 12, 5), (512, 270, 4),
                               (6, 500, 4), (900, 10, 4), (80, 144, 5), (144, 80, 5), (160, 240, 4), (240, 160, 4),
                               (288, 320, 4), (320, 288, 4), (400, 432, 4), (432, 400, 4), (480, 512, 4), (512, 480, 4)])
def test_poisson_of_every_pass_count(n, precision, tol):
    cfg = make_config(*n, sgstype=0)
    g = grid_of(cfg)
    r = np.random.default_rng(n[0]).standard_normal((n[2], n[1], n[0]))
    RHS = np.zeros(g.shape_rhs())
    RHS[1:-1, 1:-1, 1:-1] = r - r.mean()
    want = Oracle(cfg).poisson(RHS)
    ps = L.PoissonSolver(n, L=tuple(float(x) for x in n), precision=precision)
    Phi = np.zeros(g.shape_p())
    ps.execute(Phi, RHS)
    assert rel(Phi[2:-2, 2:-2, 2:-2], want[2:-2, 2:-2, 2:-2]) < tol


# the mixed path's pressure: each stage's projection turns the rounding of
# the stored velocity deviations (at most 0.4 m/s: the perturbations and the
# profile's spread within a level) over one cell into pressure through its
# coefficient 2 alpha dt, and the pressure sums the stages' increments
P_MIXED_ABS = 2.0 ** -24 * 0.4 * sum(1.0 / (2.0 * a * 0.02) for a in (4.0 / 15.0, 1.0 / 15.0, 1.0 / 6.0))


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("n", [(50, 36, 8), (75, 30, 6), (20, 100, 5), (144, 15, 4)])
def test_step_through_the_divergence(n, precision):
    cfg = make_config(*n, precision=precision)
    g = grid_of(cfg)
    o = Oracle(make_config(*n))
    o.set_state(*log_profile_state(g, seed=n[1]))
    o.project(1.0)
    d = L.Domain(cfg)
    d.upload(*o.state())
    o.step(1)
    d.step(1)
    for a, b, name in zip(interiors(g, *d.download()), interiors(g, *o.state()), "UVWP"):
        if name != "P":
            assert rel(a, b) < (1e-12 if precision == PREC_FP64 else 1e-5), name
        elif precision == PREC_FP64:
            assert rel(a, b) < 1e-11
        else:
            assert float(np.abs(a - b).max()) < P_MIXED_ABS


# The form of the y transform at the ends of the FP64 rule (192, 288 and 320 in
# registers, 240, 384 and 400 not), with an x length of each form beside it; 1e-12
# as above
@pytest.mark.parametrize("n", [(32, 192, 4), (36, 288, 4), (48, 320, 4), (32, 240, 5), (36, 384, 4), (45, 400, 4)])
def test_fp64_y_forms(n):
    test_poisson_of_every_pass_count(n, PREC_FP64, 1e-12)


# A given right-hand side on large domains (W2 of more than 5.2 MB): register x
# tiles across levels, and generic ones that start anew at each level with a
# last tile that is not full; bounds as above
@pytest.mark.parametrize("precision, tol", [(PREC_FP64, 1e-12), (PREC_MIXED, 1e-5)])
@pytest.mark.parametrize("n", [(256, 125, 45), (300, 270, 18)])
def test_poisson_with_tiles_per_level(n, precision, tol):
    test_poisson_of_every_pass_count(n, precision, tol)
