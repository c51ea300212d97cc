"""Meshes far from their origin: the reuse of translated copies where a coordinate's
rounding is no longer small beside a patch."""
import os
import subprocess
import sys

import numpy as np
import pytest

from helpers import inductance, potential
from peeeeeeeeeeeeeeeeeeec_gb300.mesh import SynthMesh

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))

_PROBE = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, {repo!r})
from peeeeeeeeeeeeeeeeeeec_gb300 import abi
from peeeeeeeeeeeeeeeeeeec_gb300.mesh import SynthMesh
lib = abi.load_gpu_lib()
ulp = 2.0 ** -24                      # of a coordinate of 2^28
h = 2.0 ** 20 * ulp
with SynthMesh.plate(1.0, 1.0, 1, 1) as m:
    for r in range(4):
        x, d = 2.0 ** 28 + 64 * h * r, (3 if r % 2 == 0 else -3) * ulp
        quad = [x, 0, 0, x + h, 2 * h, 0, x + 2 * h, 0, 0, x + h + d, -2 * h, 0]
        assert m.dual.node_patches[r].count == 1
        for t in range(12):
            m.dual.node_patches[r].patches[0].points[t] = quad[t]
    o, st = abi.PotentialOptions(), abi.PeecAssemblyStats()
    lib.potential_options_default(C.byref(o), 1)
    p = lib.peec_gb300_device_alloc(16 * 8)
    assert lib.peec_gb300_potential_device(C.byref(m.mesh), C.byref(m.dual), C.byref(o), p, C.byref(st)) == 0
    P = np.zeros((4, 4))
    assert lib.peec_gb300_copy_to_host(P.ctypes.data, p, P.nbytes) == 0
assert np.all(np.isfinite(P))
print(int(st.near_pairs), int(st.near_pairs_evaluated))
"""


def test_copies_whose_longest_edge_differs():
    """Four patches that agree to 6 ulps of their coordinates (2^28 beside edges of
    2^-4): the first triangle has two equal longest edges, in the second the longer of
    two edges (by 1.2e-6) is another one in every second patch.  A copy that would
    bisect another edge than its representative is integrated by itself, by levels
    as by the depth-first form, which compares the lengths at every node."""
    res = {}
    for mode in ("1", "0"):
        env = dict(os.environ, PEEC_GB300_NEAR_LEVELS=mode)
        r = subprocess.run([sys.executable, "-c", _PROBE.format(repo=os.path.dirname(HERE))], env=env,
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        res[mode] = r.stdout.split()
    assert res["0"] == ["4", "2"]
    assert res["1"] == res["0"]


@pytest.mark.parametrize("offset", [0.0, 2.0 ** 10, 2.0 ** 20])
def test_shared_entries_far_from_the_origin(gpu_lib, offset):
    """A plate of 12 x 11 cells whose node coordinates are off by up to two ulps of
    the largest one: entries of regions at least five cells apart with and without reuse.
    Points are held as float pairs of distances from the mesh's middle, 2^-49 of its
    half extent, four of them in a difference of two points and of two results; the
    corrected sharing of copies within 8 ulps of the extent adds 16 2^-52 of it."""
    nx, ny, h = 12, 11, 0.05
    rng = np.random.default_rng(21)
    i, j = np.meshgrid(np.arange(nx + 1), np.arange(ny + 1))
    xyz = np.zeros((i.size, 3))
    xyz[:, 0], xyz[:, 1] = offset + h * i.ravel(), offset + h * j.ravel()
    xyz[:, :2] += rng.integers(-2, 3, (i.size, 2)) * np.spacing(np.abs(xyz).max())
    a, b = np.meshgrid(np.arange(nx), np.arange(ny))
    p = (b * (nx + 1) + a).ravel()
    got = {}
    with SynthMesh.from_arrays(xyz, np.stack([p, p + 1, p + nx + 2, p + nx + 1], 1)) as m:
        ends = xyz[m.edges()].mean(axis=1)
        before = gpu_lib.peec_gb300_set_near_reuse(0)
        try:
            for on in (0, 1):
                gpu_lib.peec_gb300_set_near_reuse(on)
                got[on] = [f(gpu_lib, m) for f in (inductance, potential)]
        finally:
            gpu_lib.peec_gb300_set_near_reuse(before)
    for (s0, own), (s1, shared), at in zip(got[0], got[1], (ends, xyz)):
        assert s0 == 0 and s1 == 0
        apart = np.linalg.norm(at[:, None] - at[None], axis=-1)
        far = (apart > 5.5 * h) & (own != 0)
        bound = (8 * 2.0 ** -49 * 0.5 * nx * h + 16 * 2.0 ** -52 * nx * h) / (4 * h) + 64 * 2.0 ** -48
        assert np.max(abs(shared - own)[far] / abs(own)[far]) < bound


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_a_non_finite_corner_names_its_own_entry(gpu_lib, capfd, value):
    """Points are taken from the mesh's middle: an infinite corner must not spoil the
    other patches' points.  The entry that is named is the one of the FP64 rule."""
    named = []
    before = gpu_lib.peec_gb300_set_far_precision(1)
    try:
        for mode in (0, 1):
            gpu_lib.peec_gb300_set_far_precision(mode)
            with SynthMesh.plate(2.0, 1.0, 8, 4) as m:
                m.dual.node_patches[30].patches[0].points[0] = value
                capfd.readouterr()
                assert potential(gpu_lib, m)[0] != 0
                named.append([x for x in capfd.readouterr().err.splitlines() if "failed" in x])
    finally:
        gpu_lib.peec_gb300_set_far_precision(before)
    assert named[0] and named[0] == named[1]
