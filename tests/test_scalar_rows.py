"""The scalar stage's rows and columns: widths of whole warps and pairs, one
past and one short of them, odd widths (the per-cell stage on both paths), odd
row counts, columns shorter and longer than a chunk, against the oracle."""
import pytest

from conftest import rel
from gpu_elmm_b200 import lib as L
from gpu_elmm_b200.config import FIELD_TEMPERATURE, PREC_FP64, PREC_MIXED, grid_of, make_config
from gpu_elmm_b200.workloads import interior, interiors, log_profile_state, puff_state, temperature_state
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("n", [(30, 9, 5), (32, 5, 18), (36, 8, 40), (45, 10, 6), (64, 5, 70), (75, 6, 34), (4, 4, 16)])
def test_scalar_rows(n, precision):
    kw = dict(buoyancy=True, num_scalars=1, point_sources=[(1, (0.5, 1.5, 0.5), 1.0)])
    cfg = make_config(*n, precision=precision, **kw)
    g = grid_of(cfg)
    st, T0, S0 = log_profile_state(g, seed=n[0]), temperature_state(g, seed=n[1]), puff_state(g, (2, 2, 2))
    o = Oracle(make_config(*n, **kw))
    o.set_state(*st)
    o.set_field(FIELD_TEMPERATURE, T0)
    o.set_field(16, S0)
    o.project(1.0)
    d = L.Domain(cfg)
    d.upload(*o.state())
    d.upload_temperature(T0)
    d.upload_scalar(1, S0)
    o.step(2)
    d.step(2)
    # the mixed path's bound of the other tests: FP32 rounding of the fields
    # and of their increments
    tol = 1e-11 if precision == PREC_FP64 else 1e-5
    m = (g.Prnx, g.Prny, g.Prnz)
    assert rel(interior(d.temperature(), -2, m) - 295.0, interior(o.get_field(12), -2, m) - 295.0) < tol
    assert rel(interior(d.scalar(1), -2, m), interior(o.get_field(16), -2, m)) < tol
    for a, b, name in zip(interiors(g, *d.download())[:3], interiors(g, *o.state())[:3], "UVW"):
        assert rel(a, b) < tol, name
    d.close()
