"""Served FP64 solves whose factorisation takes digits."""
import numpy as np
import pytest

from peeeeeeeeeeeeeeeeeeec_gb300.mesh import SynthMesh
from test_gpu_server import GB, run

pytestmark = pytest.mark.gpu


def test_tight_budget_changes_no_digits(gpu_lib):
    """5714 unknowns, whose digits exceed the 64 MiB of scratch in a request's
    estimate: a budget that holds the request without them gives the same bits."""
    with SynthMesh.box(1.3, 0.9, 0.55, 26, 18, 11) as m:
        n = m.n_edges + m.n_nodes
        r = [dict(mesh=0, frequency=3e7, k_hat=np.array([[0.0, 0.0, 1.0]]), e_hat=np.array([[1.0, 0.0, 0.0]]),
                  mixed=False)]
        budget = (72 << 20) + 32 * n * n + 8 * (m.n_edges ** 2 + m.n_nodes ** 2) + 200 * n
        (xa, ra), = run([m], r, 8 * GB, 1)
        (xb, rb), = run([m], r, budget, 1)
        assert ra["status"] == 0 and rb["status"] == 0
        assert np.array_equal(xa, xb)
