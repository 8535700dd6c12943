"""Requests admitted beside a running chunk: their memory is zeroed, filled and
projected while other requests' steps keep the GPU busy, and every one of them
returns what it returns alone, bit for bit (a field whose zeroing or upload
came late would change its slices even where it stays finite)."""
import numpy as np
import pytest

from gpu_elmm_b200.serve import Server, request_inputs, run_arrivals
from gpu_elmm_b200.workloads import dispersion_request, poisson_arrivals
from test_serving import _alone

pytestmark = pytest.mark.gpu


def test_requests_admitted_beside_a_chunk():
    reqs = [dict(dispersion_request(0, q), steps=600) for q in range(10)]
    inputs = [request_inputs(r) for r in reqs]
    srv = Server(precision=1, budget_bytes=40 << 30, max_active=64, chunk_steps=50, device=0)
    done, _ = run_arrivals(srv, reqs, poisson_arrivals(0, 20.0, len(reqs)), inputs)  # raises for a failed request
    srv.close()
    assert len(done) == len(reqs)
    for q, _, slices in done:
        assert all(np.array_equal(a, b) for a, b in zip(slices, _alone(reqs[q], 1))), reqs[q]["n"]
