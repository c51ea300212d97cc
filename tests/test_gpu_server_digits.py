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


def test_served_plate_meets_the_gate(gpu_lib):
    """1541 unknowns of a square plate, whose pivot candidates tie: the served FP64 solve
    keeps its digits (its pivots stay inside), against the drop-in factorisation."""
    from helpers import ComplexLU
    from test_gpu_server import host_mna, plane_wave_rhs
    with SynthMesh.plate(1.1, 1.1, 22, 22) as m:
        k, e, f = np.array([0.6, 0.0, 0.8]), np.array([0.0, 1.0, 0.0]), 4.7e7
        r = [dict(mesh=0, frequency=f, k_hat=k[None], e_hat=e[None], mixed=False)]
        (x, res), = run([m], r, 8 * GB, 1)
        assert res["status"] == 0 and res["backward_error"] <= 1e-10
        Z, b = host_mna(gpu_lib, m, f), plane_wave_rhs(m, f, k, e)
        x = x.reshape(-1)
        assert np.max(np.abs(Z @ x - b) / (np.abs(Z) @ np.abs(x) + np.abs(b))) <= 1e-10
        lu = ComplexLU(gpu_lib, Z)
        s, y = lu.solve(b)
        lu.free()
        # both backward stable in FP64: N u of the largest entry times the condition
        cond = np.linalg.cond(Z / np.abs(Z).max(axis=1)[:, None])
        assert s == 0 and np.max(np.abs(x - y)) <= len(b) * 2.0 ** -53 * cond * np.max(np.abs(y))
