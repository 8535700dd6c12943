"""Workloads of ordinary size over several steps against the CPU oracle, each
field with a bound of its own: the small channel, a dispersion request, a
convective boundary layer on odd lengths, and an array of cubes.

U, V, W, the temperature's deviation and the scalar: 1e-12 and 1e-11 (FP64, as
in the other parity tests; 1e-11 and P 1e-10 among bodies) or 1e-5 (mixed) of the
largest value.  The mixed pressure: each stage's projection turns the rounding
of the stored velocity (of a deviation of at most 0.4 m/s, or of the full
velocity among bodies) over one cell, the tallest on a stretched grid, into
pressure through its coefficient 2 alpha dt, twice (a value's own and its neighbour's); the next projection takes
it back with the pressure gradient, so that a sum over one step's stages bounds
it after any number of steps; a stratification adds the rounding of its own
pressure."""
import os

import numpy as np
import pytest

from conftest import rel
from gpu_elmm_b200 import lib as L
from gpu_elmm_b200.config import FIELD_SCALAR, FIELD_TEMPERATURE, PREC_FP64, PREC_MIXED, grid_of, make_config
from gpu_elmm_b200.workloads import (interior, interiors, log_profile_state, puff_state, stretched_zw,
                                     temperature_state)
import oracle as orc
from oracle import Oracle

pytestmark = pytest.mark.gpu

STAGES = sum(1.0 / (2.0 * a * 0.02) for a in (4.0 / 15.0, 1.0 / 15.0, 1.0 / 6.0))
SMALL, DISPERSION, CONVECTIVE = (64, 64, 32), (128, 128, 64), (135, 135, 75)


@pytest.fixture(scope="module", autouse=True)
def _all_cores():
    orc.set_threads(os.cpu_count() or 1)
    yield


def _check(g, d, o, precision, vel, cell=1.0, solids=False):
    a, b = interiors(g, *d.download()), interiors(g, *o.state())
    fp64 = precision == PREC_FP64
    for x, y, name in zip(a, b, "UVW"):
        assert rel(x, y) < ((1e-11 if solids else 1e-12) if fp64 else 1e-5), name
    if fp64:
        assert rel(a[3], b[3]) < (1e-10 if solids else 1e-11)
    else:
        bound = 2 * 2.0 ** -24 * vel * cell * STAGES + 4 * 2.0 ** -24 * np.abs(b[3]).max()
        assert float(np.abs(a[3] - b[3]).max()) < bound


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("n, steps, kw", [
    (SMALL, 40, {}), (DISPERSION, 6, dict(num_scalars=1, point_sources=[(1, (42.5, 63.5, 15.5), 1.0)])),
    (CONVECTIVE, 4, dict(buoyancy=True, heat_flux=(0.1, 0.0)))], ids=["small", "dispersion", "convective"])
def test_steps_follow_the_oracle(n, steps, kw, precision):
    cfg = make_config(*n, precision=precision, **kw)
    g = grid_of(cfg)
    o = Oracle(make_config(*n, **kw))
    d = L.Domain(cfg)
    st = log_profile_state(g, seed=n[0])
    o.set_state(*st)
    T0, S0 = temperature_state(g, seed=n[0]), puff_state(g, (43, 64, 16))
    if "buoyancy" in kw:
        o.set_field(FIELD_TEMPERATURE, T0)
        d.upload_temperature(T0)
    if "num_scalars" in kw:
        o.set_field(FIELD_SCALAR, S0)
        d.upload_scalar(1, S0)
    o.project(1.0)
    d.upload(*o.state())
    d.project(1.0)
    o.step(steps)
    d.step(steps)
    _check(g, d, o, precision, 0.4)
    m, tol = (g.Prnx, g.Prny, g.Prnz), 1e-11 if precision == PREC_FP64 else 1e-5
    if "buoyancy" in kw:
        assert rel(interior(d.temperature(), -2, m) - 295.0, interior(o.get_field(FIELD_TEMPERATURE), -2, m) - 295.0) < tol
    if "num_scalars" in kw:
        assert rel(interior(d.scalar(1), -2, m), interior(o.get_field(FIELD_SCALAR), -2, m)) < tol
    d.close()


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
def test_cubes_follow_the_oracle(precision):
    """2 x 2 cubes of 16 cells on a stretched grid under a mean pressure gradient, 20 steps."""
    from gpu_elmm_b200.solids import build_solids, cube_array
    from gpu_elmm_b200.workloads import CUBES_PR_GRADIENT_X
    n, zw = (96, 96, 48), stretched_zw(48)
    kw = dict(zW=zw, pr_gradient_x=CUBES_PR_GRADIENT_X)
    cfg = make_config(*n, precision=precision, **kw)
    g = grid_of(cfg)
    sol = build_solids(cfg, cube_array(2, 16.0, 48.0, float(zw[16]), offset=16.0, depth=5.0))
    o = Oracle(make_config(*n, **kw))
    o.set_state(*log_profile_state(g, seed=4, zW=zw))
    o.project(1.0)
    d = L.Domain(cfg)
    d.upload(*o.state())
    o.set_solids(sol)
    d.set_solids(sol)
    o.step(20)
    d.step(20)
    vel = float(max(np.abs(x).max() for x in o.state()[:3]))
    _check(g, d, o, precision, vel, cell=float(np.diff(zw).max()), solids=True)
    d.close()
