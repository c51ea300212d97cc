"""The cluster FP64 panel against the lean and the cooperative panel: the same
pivots and the same factors bit for bit, at the edges of its warps and CTAs, on
columns with equal magnitudes, zeros, and entries far from 1."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_PROBE = r"""
import hashlib, sys
import numpy as np
sys.path.insert(0, {repo!r}); sys.path.insert(0, {tests!r})
from helpers import ComplexLU, RealLU
from peeeeeeeeeeeeeeeeeeec_gb300 import abi
lib = abi.load_gpu_lib()
h = hashlib.sha256()
rng = np.random.default_rng(11)
for n in (2, 31, 33, 129, 513, 1100):
    for kind in ("normal", "ties", "zeros", "sizes"):
        a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        if kind == "ties":  # few distinct magnitudes
            a = np.round(a.real) + 1j * np.round(a.imag) + 4 * np.eye(n)
        if kind == "zeros":
            a = a * (rng.random((n, n)) < 0.1) + np.eye(n)
        if kind == "sizes":
            a = a * np.logspace(-140, 140, n)[:, None]
        c = a if kind != "sizes" else a * np.logspace(135, -135, n)[:, None]
        f = ComplexLU(lib, np.ascontiguousarray(c))
        h.update(b"%d" % f.status)
        if f.status == 0:
            lu, piv, rs, cs = f.factors()
            h.update(lu.tobytes()); h.update(piv.tobytes()); f.free()
        r = RealLU(lib, np.ascontiguousarray(a.real), tol=1e-300)
        h.update(b"%d" % r.status)
        if r.status == 0:
            lu, piv = r.factors()
            h.update(lu.tobytes()); h.update(piv.tobytes()); r.free()
    print(n, h.hexdigest())
"""


def test_cluster_lean_and_grid_panels_agree():
    here = os.path.dirname(os.path.abspath(__file__))
    code = _PROBE.format(repo=os.path.dirname(here), tests=here)
    out = {}
    for mode in ("", "lean", "coop"):
        env = dict(os.environ)
        env.pop("PEEC_GB300_PANEL", None)
        if mode:
            env["PEEC_GB300_PANEL"] = mode
        r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        out[mode] = r.stdout.strip()
    assert out[""] == out["lean"] == out["coop"]
