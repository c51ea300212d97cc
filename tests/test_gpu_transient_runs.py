"""Every number of runs that a batch takes steps them as single runs do (the
step kernels are instantiated for 1, 2, 3, 4, 6 and 8 runs, one or two rows a warp)."""
import ctypes as C

import numpy as np
import pytest

from conftest import golden
from helpers import inductance, potential
from peeeeeeeeeeeeeeeeeeec_gb300.mesh import SynthMesh
from test_gpu_transient import I_TOL, V_TOL, DeviceTransient, werr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", range(1, 9))
def test_batch_of_n_runs(gpu_lib, n):
    """86 unknowns (56 edge rows, 30 node rows; rows shorter than the unrolled
    loops): the same sums in the same order whatever the batch, so the same bits."""
    f, g = golden("box421"), golden("transient_box421")
    ne, nv = f["L"].shape[0], f["P"].shape[0]
    srcs = [(1e5 * (1 + k), 1500.0 + 100 * k, 1.0e6, 0.0, k, 29 - k) for k in range(n)]
    t = DeviceTransient(gpu_lib, f["L"], f["P"], f["edges"], g["R"], 2, 1e-7)
    try:
        X = np.zeros((n, ne + nv))
        dX = t.put(X)
        col = lambda k: (C.c_double * n)(*[s[k] for s in srcs])
        sz = lambda k: (C.c_size_t * n)(*[s[k] for s in srcs])
        assert gpu_lib.peec_gb300_transient_lightning_batch(t.h, n, col(0), col(1), col(2), col(3), sz(4), sz(5), 0, 40,
                                                            dX, None, 0, None, 0, None) == 0
        gpu_lib.peec_gb300_copy_to_host(X.ctypes.data, dX, X.nbytes)
        for r, src in enumerate(srcs):
            s, I, V, _ = t.run(src, 40)
            assert s == 0
            assert np.array_equal(X[r, :ne], I) and np.array_equal(X[r, ne:], V)
    finally:
        t.close()


@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 12), (4, 4), (1, 25), (1, 26)])
def test_inverse_at_block_edges(gpu_lib, oracle, nx, ny):
    """8, 63, 65, 128 and 133 unknowns: whole and ragged 64-row blocks of the
    substitution that forms the inverse."""
    with SynthMesh.plate(0.05 * nx, 0.05 * ny, nx, ny) as m:
        _, L = inductance(gpu_lib, m)
        _, P = potential(gpu_lib, m)
        edges = np.ascontiguousarray(m.edges())
        R = 1e-3 * np.ones(m.n_edges)
        src = (102900.0, 1500.0, 1.0e6, 0.0, 0, m.n_nodes - 1)
        t = DeviceTransient(gpu_lib, L, P, edges, R, 2, 1e-7)
        try:
            s, I, V, _ = t.run(src, 20)
            so, Io, Vo, _ = oracle.transient_lightning(L, P, edges, R, 2, 1e-7, src, 20, probe_nodes=range(m.n_nodes),
                                                       probe_edges=range(m.n_edges))
            assert s == 0 and so == 0
            assert werr(I, Io) < I_TOL and werr(V, Vo) < V_TOL
        finally:
            t.close()
