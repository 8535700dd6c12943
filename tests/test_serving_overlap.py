"""Requests admitted beside a running chunk: their memory is zeroed, filled and
projected while other requests' steps keep the GPU busy, and every one of them
ends well."""
import pytest

from gpu_elmm_b200.serve import Server, request_inputs, run_arrivals
from gpu_elmm_b200.workloads import dispersion_request, poisson_arrivals

pytestmark = pytest.mark.gpu


def test_requests_admitted_beside_a_chunk():
    reqs = [dict(dispersion_request(0, q), steps=600) for q in range(10)]
    inputs = [request_inputs(r) for r in reqs]
    srv = Server(precision=1, budget_bytes=40 << 30, max_active=64, chunk_steps=50, device=0)
    done, _ = run_arrivals(srv, reqs, poisson_arrivals(0, 20.0, len(reqs)), inputs)  # raises for a failed request
    srv.close()
    assert len(done) == len(reqs)
