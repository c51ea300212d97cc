"""Entries of Lp and P with translated copies of the same regions share one
evaluation of the far rule; against every entry by itself, on meshes where all,
some and none of the regions repeat."""
import numpy as np
import pytest

from helpers import elem_rel_err, inductance, potential
from peeeeeeeeeeeeeeeeeeec_gb300.mesh import SynthMesh

pytestmark = pytest.mark.gpu


def grid(kind, nx, ny):
    """Plate of nx x ny quads about 5 cm wide."""
    rng = np.random.default_rng(nx * 100 + ny)
    x, y = 0.05 * np.arange(nx + 1), 0.047 * np.arange(ny + 1)
    if kind == "graded":  # the right half's cells differ from the left's and from one another
        x = np.where(x > x[nx // 2], x + 0.3 * np.maximum(x - x[nx // 2], 0) ** 2, x)
    xyz = np.zeros(((nx + 1) * (ny + 1), 3))
    xyz[:, 0], xyz[:, 1] = np.tile(x, ny + 1), np.repeat(y, nx + 1)
    if kind == "jittered":
        xyz += rng.uniform(-0.004, 0.004, xyz.shape)
    if kind == "turned":
        q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
        xyz = xyz @ q.T + [1.0, -2.0, 0.5]
    i, j = np.meshgrid(np.arange(nx), np.arange(ny))
    p = (j * (nx + 1) + i).ravel()
    return xyz, np.stack([p, p + 1, p + nx + 2, p + nx + 1], 1)


@pytest.mark.parametrize("far_order", [2, 4, 6])
@pytest.mark.parametrize("kind", ["regular", "graded", "jittered", "turned"])
@pytest.mark.parametrize("nx,ny", [(3, 2), (12, 11), (31, 7)])
def test_shared_far_entries(gpu_lib, kind, nx, ny, far_order):
    xyz, quads = grid(kind, nx, ny)
    with SynthMesh.from_arrays(xyz, quads) as m:
        prev = gpu_lib.peec_gb300_set_near_reuse(0)
        try:
            own = [f(gpu_lib, m, far_order=far_order) for f in (inductance, potential)]
            gpu_lib.peec_gb300_set_near_reuse(1)
            shared = [f(gpu_lib, m, far_order=far_order) for f in (inductance, potential)]
        finally:
            gpu_lib.peec_gb300_set_near_reuse(prev)
    # the points are held as float pairs: 2^-49 of the largest coordinate, four of
    # them in a difference of two points and of two results, against a distance
    # of at least half a patch (a quarter of a cell); 64 roundings of 2^-48
    bound = 8 * 2.0 ** -49 * np.abs(xyz).max() / (0.5 * 0.01) + 64 * 2.0 ** -48
    for (s0, a), (s1, b) in zip(own, shared):
        assert s0 == 0 and s1 == 0
        assert elem_rel_err(b, a) < bound
        assert np.array_equal(b, b.T) and np.array_equal(a == 0, b == 0)

