"""Meshes far from their origin: the reuse of translated copies where a coordinate's
rounding is no longer small beside a patch."""
import os
import subprocess
import sys

import numpy as np
import pytest

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
