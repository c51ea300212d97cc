"""Performance cases: what users of the library have it do, each through its
public entry points (include/*.h, called with ctypes as any host program calls
the C ABI).

A case is one of these jobs:

  assemble    Lp and P of a mesh into device memory, quasi-static, with the
              FP64-accurate far rule (precision 1) or the FP32 one of the
              mixed path (precision 2)
  retarded    Lp, P with the kernel exp(-jkR)/R and the harmonic matrix
  real_lu     real LU and solve of a device-resident MNA matrix
  dropin      complex_lu_factorize / complex_lu_solve_multiple on host arrays,
              as an unchanged reference driver calls them
  plain       harmonic solve with every matrix in device memory: MNA fill,
              plane waves, FP64 complex LU, solve
  mixed       the same system by the mixed-precision solve (1e-10 gate)
  sweep       one mesh's frequency sweep on a plan that the program keeps
  lightning   steps of the stage-1 transient on a resident system, one or
              more runs stepped together
  lightning_new   the same from a new system: create, step, destroy

Meshes are boxes and plates of quadrilateral cells; every seed scales the
sides by a few per cent and draws its own frequencies, waves and sources.
The assembly jobs take the library's Mesh / DualMesh structs.  The solver
jobs take Lp and P as given matrices: here the 1/R kernel between edge
centres (node positions) with the self term of a square cell, so that their
inputs come from the seed alone.
"""
import ctypes as C
import math

import numpy as np
import torch

from peeeeeeeeeeeeeeeeeeec_gb300 import abi
from peeeeeeeeeeeeeeeeeeec_gb300.mesh import SynthMesh

C0 = 299792458.0
MU0 = 4e-7 * math.pi
EPS0 = 1.0 / (MU0 * C0 * C0)
DT = 1e-7          # time step of the lightning runs
TOL = 1e-10        # backward-error gate of the mixed paths
MAX_ITER = 30


def listed():
    return [
        # the smallest job: a 1 m plate of 16 x 16 cells, launch-bound
        {"name": "assemble_plate16", "job": "assemble", "shape": "plate", "nx": 16, "ny": 16, "nz": 0, "precision": 1},
        # the headline box (2 x 1 x 0.5 m at 5 cm), assembled for the FP64 path
        {"name": "assemble_box", "job": "assemble", "shape": "box", "nx": 40, "ny": 20, "nz": 10, "precision": 1},
        # an uneven box assembled for the mixed path (FP32 far rule)
        {"name": "assemble_box_fp32", "job": "assemble", "shape": "box", "nx": 33, "ny": 17, "nz": 9, "precision": 2},
        # retarded harmonic matrix of the box at 10 cm
        {"name": "retarded_box", "job": "retarded", "shape": "box", "nx": 20, "ny": 10, "nz": 5},
        # real MNA of the 16 x 16 plate (833 unknowns), one injection
        {"name": "real_lu_plate16", "job": "real_lu", "shape": "plate", "nx": 16, "ny": 16, "nz": 0},
        # host arrays through complex_lu.h, 2102 unknowns, four excitations
        {"name": "dropin_box_half", "job": "dropin", "shape": "box", "nx": 20, "ny": 10, "nz": 5, "nrhs": 4},
        # the headline solve on the FP64 path: 8402 unknowns, one plane wave
        {"name": "plain_box", "job": "plain", "shape": "box", "nx": 40, "ny": 20, "nz": 10, "nrhs": 1},
        # the same on the mixed path
        {"name": "mixed_box", "job": "mixed", "shape": "box", "nx": 40, "ny": 20, "nz": 10, "nrhs": 1},
        # a served RCS request: a plate with the most plane waves of a request
        {"name": "mixed_plate_rcs", "job": "mixed", "shape": "plate", "nx": 39, "ny": 31, "nz": 0, "nrhs": 64},
        # frequency sweep of a small mesh, four plane waves a frequency
        {"name": "sweep_plate", "job": "sweep", "shape": "plate", "nx": 17, "ny": 14, "nz": 0, "nrhs": 4, "nfreq": 8},
        # lightning on the headline box: three strikes stepped together
        {"name": "lightning_box", "job": "lightning", "shape": "box", "nx": 40, "ny": 20, "nz": 10, "nrun": 3, "steps": 48},
        # lightning on a mesh seen for the first time (system built in the pass)
        {"name": "lightning_new_box", "job": "lightning_new", "shape": "box", "nx": 23, "ny": 13, "nz": 8, "nrun": 1,
         "steps": 48},
    ]


# Cells of the smallest and the largest mesh each job draws.
RANGES = {
    "assemble": (100, 2800), "retarded": (60, 900), "real_lu": (100, 1400), "dropin": (100, 1000),
    "plain": (170, 2800), "mixed": (170, 2800), "sweep": (100, 700), "lightning": (100, 2800),
    "lightning_new": (100, 1400),
}


def draw(rng):
    job = rng.choice(sorted(RANGES))
    lo, hi = RANGES[job]
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    while True:
        a, b = rng.uniform(0.3, 1.0), rng.uniform(0.3, 1.0)
        if rng.random() < 0.5:  # plate: nx ny cells
            h = math.sqrt(a / cells)
            c = {"job": job, "shape": "plate", "nx": max(2, round(1 / h)), "ny": max(2, round(a / h)), "nz": 0}
            count = c["nx"] * c["ny"]
        else:  # box: 2 (nx ny + ny nz + nz nx) cells
            h = math.sqrt(2 * (a + a * b + b) / cells)
            c = {"job": job, "shape": "box", "nx": max(1, round(1 / h)), "ny": max(1, round(a / h)),
                 "nz": max(1, round(b / h))}
            count = 2 * (c["nx"] * c["ny"] + c["ny"] * c["nz"] + c["nz"] * c["nx"])
        if count <= hi:
            break
    if job == "assemble":
        c["precision"] = rng.choice([1, 2])
    if job in ("dropin", "plain", "sweep"):
        c["nrhs"] = rng.randint(1, 4)
    if job == "mixed":
        c["nrhs"] = rng.randint(1, 64)
    if job == "sweep":
        c["nfreq"] = rng.randint(4, 12)
    if job == "lightning":
        c["nrun"], c["steps"] = rng.randint(1, 8), rng.randint(16, 64)
    if job == "lightning_new":
        c["nrun"], c["steps"] = 1, rng.randint(16, 64)
    return c


# ---------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------
def counts(case):
    """(edges, nodes) of the case's mesh."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["shape"] == "plate":
        return nx * (ny + 1) + ny * (nx + 1), (nx + 1) * (ny + 1)
    cells = 2 * (nx * ny + ny * nz + nz * nx)
    return 2 * cells, cells + 2


def sides(case, rng):
    """Side lengths in metres: 5 cm cells, each side scaled by up to 4 per cent."""
    n = [case["nx"], case["ny"], case["nz"]]
    return [0.05 * k * (1.0 + 0.04 * rng.uniform(-1, 1)) for k in n]


def surface(case, size):
    """Node positions and edges (node pairs) of the plate or closed box."""
    n = [case["nx"], case["ny"], case["nz"]]
    faces = []  # integer corner coordinates of every cell

    def face(u, v, w, at):
        i, j = np.meshgrid(np.arange(n[u]), np.arange(n[v]), indexing="ij")
        i, j = i.ravel(), j.ravel()
        q = np.zeros((i.size, 4, 3), dtype=np.int64)
        for k, (di, dj) in enumerate(((0, 0), (1, 0), (1, 1), (0, 1))):
            q[:, k, u], q[:, k, v], q[:, k, w] = i + di, j + dj, at
        faces.append(q)

    face(0, 1, 2, 0)
    if case["shape"] == "box":
        face(0, 1, 2, n[2])
        for at in (0, n[1]):
            face(0, 2, 1, at)
        for at in (0, n[0]):
            face(1, 2, 0, at)
    q = np.concatenate(faces)
    key = (q[..., 0] * (n[1] + 1) + q[..., 1]) * (n[2] + 1) + q[..., 2]
    _, first, node = np.unique(key, return_index=True, return_inverse=True)
    node = node.reshape(-1, 4)
    step = [s / k if k else 0.0 for s, k in zip(size, n)]
    xyz = q.reshape(-1, 3)[first] * np.array(step)
    pairs = np.concatenate([node[:, [k, (k + 1) % 4]] for k in range(4)])
    pairs = np.unique(np.sort(pairs, axis=1), axis=0)
    return xyz, pairs.astype(np.int32)


def inverse_distance(points, soft):
    """1 / sqrt(|p - q|^2 + soft^2) between all points, FP64 on the device."""
    p = torch.from_numpy(points).cuda()
    r2 = torch.full((p.shape[0], p.shape[0]), soft * soft, dtype=torch.float64, device="cuda")
    for k in range(3):
        r2 += (p[:, None, k] - p[None, :, k]).square()
    return r2.rsqrt_()


def waves(rng, count):
    """Propagation directions and transverse unit polarisations (count x 3)."""
    th, ph = np.arccos(rng.uniform(-1, 1, count)), rng.uniform(0, 2 * math.pi, count)
    k = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], 1)
    a = np.where(np.abs(k[:, 2:]) < 0.9, [[0.0, 0.0, 1.0]], [[1.0, 0.0, 0.0]])
    e = np.cross(k, a)
    return np.ascontiguousarray(k), np.ascontiguousarray(e / np.linalg.norm(e, axis=1)[:, None])


def inputs(case, seed):
    """Everything a solver job is given, from the seed alone."""
    rng = np.random.default_rng(seed)
    size = sides(case, rng)
    xyz, edges = surface(case, size)
    d = {"ne": len(edges), "nv": len(xyz), "edges": edges}
    d["vectors"] = np.ascontiguousarray(xyz[edges[:, 1]] - xyz[edges[:, 0]])
    d["centers"] = np.ascontiguousarray(0.5 * (xyz[edges[:, 1]] + xyz[edges[:, 0]]))
    soft = 0.336 * 0.05  # the mean of 1/R over a square cell of side h is 2.97 / h
    vec = torch.from_numpy(d["vectors"]).cuda()
    dot = torch.zeros((d["ne"], d["ne"]), dtype=torch.float64, device="cuda")
    for k in range(3):
        dot += vec[:, None, k] * vec[None, :, k]
    d["L"] = dot.mul_(inverse_distance(d["centers"], soft)).mul_(MU0 / (4 * math.pi))
    d["P"] = inverse_distance(xyz, soft).mul_(1 / (4 * math.pi * EPS0))
    d["frequency"] = float(rng.uniform(1e6, 100e6))
    if "nrhs" in case:
        d["k_hat"], d["e_hat"] = waves(rng, case["nrhs"])
    if "nfreq" in case:
        f = np.logspace(6.5, 8, case["nfreq"]) * rng.uniform(0.95, 1.05, case["nfreq"])
        d["frequencies"] = np.ascontiguousarray(f)
    if case["job"].startswith("lightning"):
        r = case["nrun"]
        nodes = np.stack([rng.choice(len(xyz), 2, replace=False) for _ in range(r)])
        d["strike"], d["ret"] = nodes[:, 0], nodes[:, 1]
        # 10/350 us first strokes of 50 to 150 kA
        d["K"], d["alpha"], d["beta"] = 105139.0 * rng.uniform(0.5, 1.5, r), np.full(r, 2127.18), np.full(r, 246066.0)
        d["delay"] = np.zeros(r)
        d["probe_nodes"] = nodes.ravel().astype(np.int32)
        d["probe_edges"] = rng.integers(0, len(edges), 4).astype(np.int32)
    if case["job"] == "real_lu":
        d["M"] = transient_matrix(d)[0]
        b = np.zeros(d["ne"] + d["nv"])
        i, j = rng.choice(d["nv"], 2, replace=False)
        b[d["ne"] + i], b[d["ne"] + j] = 1.0, -1.0
        d["b"] = torch.from_numpy(b).cuda()
    return d


def incidence(d):
    """A (edges x nodes): -1 at the tail, +1 at the head."""
    A = torch.zeros((d["ne"], d["nv"]), dtype=torch.float64, device="cuda")
    e = torch.from_numpy(d["edges"]).long().cuda()
    A.scatter_(1, e, torch.tensor([[-1.0, 1.0]], dtype=torch.float64, device="cuda").expand(d["ne"], 2))
    return A


def transient_matrix(d, theta=0.5, dt=DT):
    """[L/dt, theta A S; -theta A^T, F/dt] (perfect conductor), A S and F."""
    A, P, ne = incidence(d), d["P"], d["ne"]
    F = 1.0 / P.diagonal()
    e = torch.from_numpy(d["edges"]).long().cuda()
    AS = (P[e[:, 1]] - P[e[:, 0]]) * F
    M = torch.empty((ne + d["nv"],) * 2, dtype=torch.float64, device="cuda")
    M[:ne, :ne], M[:ne, ne:], M[ne:, :ne], M[ne:, ne:] = d["L"] / dt, theta * AS, -theta * A.T, torch.diag(F / dt)
    return M, A, AS, F


# ---------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------
def ok(status, what):
    if status != 0:
        raise RuntimeError("%s: status %d: %s" % (what, status, abi.load_gpu_lib().peec_gb300_last_error().decode()))


def dbl(a):
    return a.ctypes.data_as(abi.c_double_p)


def empty(*shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, device="cuda")


class Handle:
    """A sweep plan or a transient system, destroyed with its owner."""

    def __init__(self, handle, destroy):
        self.handle, self.destroy = handle, destroy

    def __del__(self):
        if self.handle:
            self.destroy(self.handle)


class HostFactor:
    """A complex_lu.h factorisation on the host, freed when it and the views
    of its arrays are gone."""

    def __init__(self, lib):
        self.lib, self.f = lib, abi.ComplexLUFactorization()
        lib.complex_lu_init(C.byref(self.f))

    def view(self, pointer, shape, ctype, dtype):
        array = (ctype * math.prod(shape)).from_address(C.cast(pointer, C.c_void_p).value)
        array.owner = self
        return np.frombuffer(array, dtype=dtype).reshape(shape)

    def __del__(self):
        self.lib.complex_lu_free(C.byref(self.f))


def prepare(case, seed):
    lib, job = abi.load_gpu_lib(), case["job"]
    s = {"case": dict(case), "lib": lib}
    ne, nv = counts(case)
    n = ne + nv
    if job in ("assemble", "retarded"):
        rng = np.random.default_rng(seed)
        lx, ly, lz = sides(case, rng)
        s["mesh"] = (SynthMesh.plate(lx, ly, case["nx"], case["ny"]) if case["shape"] == "plate" else
                     SynthMesh.box(lx, ly, lz, case["nx"], case["ny"], case["nz"]))
        s["lo"], s["po"] = abi.InductanceOptions(), abi.PotentialOptions()
        lib.inductance_options_default(C.byref(s["lo"]), 1)
        lib.potential_options_default(C.byref(s["po"]), 1)
        kind = torch.complex128 if job == "retarded" else torch.float64
        s["L"], s["P"] = empty(ne, ne, dtype=kind), empty(nv, nv, dtype=kind)
        if job == "retarded":
            s["frequency"] = float(rng.uniform(20e6, 100e6))
            s["edges"] = torch.from_numpy(s["mesh"].edges()).cuda()
            s["Z"] = empty(n, n, dtype=kind)
        torch.cuda.synchronize()
        return s
    d = inputs(case, seed)
    for k in ("ne", "nv", "frequency", "k_hat", "e_hat", "frequencies", "K", "alpha", "beta", "delay"):
        if k in d:
            s[k] = d[k]
    if job == "real_lu":
        s["M"], s["b"] = d["M"], d["b"]
        s["lu"], s["x"] = empty(n, n), empty(n)
        s["piv"], s["perm"] = empty(n, dtype=torch.int64), empty(n, dtype=torch.int32)
    elif job == "dropin":
        s["Z"], s["B"] = host_system(d)
        s["X"] = np.zeros_like(s["B"])
        s["opt"] = abi.ComplexLUOptions()
        lib.complex_lu_options_default(C.byref(s["opt"]), 1)
    else:
        s["L"], s["P"] = d["L"], d["P"]
        s["edges"] = torch.from_numpy(d["edges"]).cuda()
        s["centers"], s["vectors"] = torch.from_numpy(d["centers"]).cuda(), torch.from_numpy(d["vectors"]).cuda()
    if job in ("plain", "mixed"):
        s["Z"] = empty(n, n, dtype=torch.complex128)
        s["B"] = empty(case["nrhs"], n, dtype=torch.complex128)
        s["X"] = empty(case["nrhs"], n, dtype=torch.complex128)
        s["piv"], s["perm"] = empty(n, dtype=torch.int64), empty(n, dtype=torch.int32)
        s["rows"], s["cols"] = empty(n), empty(n)
        s["k"] = [(C.c_double * 3)(*v) for v in d["k_hat"]]
        s["e"] = [(C.c_double * 3)(*v) for v in d["e_hat"]]
    torch.cuda.synchronize()  # the inputs are complete before the library's own stream reads them
    if job == "sweep":
        s["X"] = empty(case["nfreq"], case["nrhs"], n, dtype=torch.complex128)
        s["eta"], s["fallback"] = np.zeros(case["nfreq"]), np.zeros(case["nfreq"], dtype=np.int32)
        s["plan"] = Handle(lib.peec_gb300_sweep_create(
            s["L"].data_ptr(), s["P"].data_ptr(), s["edges"].data_ptr(), None, s["centers"].data_ptr(),
            s["vectors"].data_ptr(), ne, nv, case["nrhs"], dbl(s["k_hat"]), dbl(s["e_hat"]), None),
            lib.peec_gb300_sweep_destroy)
    if job.startswith("lightning"):
        s["state"] = torch.zeros((case["nrun"], n), dtype=torch.float64, device="cuda")
        s["rest"] = torch.zeros_like(s["state"])
        s["probe_nodes"] = torch.from_numpy(d["probe_nodes"]).cuda()
        s["probe_edges"] = torch.from_numpy(d["probe_edges"]).cuda()
        s["probes"] = empty(case["steps"], case["nrun"], len(d["probe_nodes"]) + len(d["probe_edges"]))
        s["strike"] = (C.c_size_t * case["nrun"])(*[int(v) for v in d["strike"]])
        s["ret"] = (C.c_size_t * case["nrun"])(*[int(v) for v in d["ret"]])
        torch.cuda.synchronize()
        if job == "lightning":
            s["system"] = new_system(s)
    return s


def new_system(s):
    h = C.c_void_p()
    ok(s["lib"].peec_gb300_transient_create(s["L"].data_ptr(), s["P"].data_ptr(), s["edges"].data_ptr(), None, s["ne"],
                                            s["nv"], 2, DT, C.byref(h)), "transient system")
    return Handle(h, s["lib"].peec_gb300_transient_destroy)


def run_assemble(s):
    lib, m = s["lib"], s["mesh"]
    before = lib.peec_gb300_set_far_precision(s["case"]["precision"])
    try:
        ok(lib.peec_gb300_inductance_device(C.byref(m.mesh), C.byref(m.dual), C.byref(s["lo"]), s["L"].data_ptr(),
                                            None), "Lp")
        ok(lib.peec_gb300_potential_device(C.byref(m.mesh), C.byref(m.dual), C.byref(s["po"]), s["P"].data_ptr(),
                                           None), "P")
    finally:
        lib.peec_gb300_set_far_precision(before)
    return {"L": s["L"], "P": s["P"]}


def run_retarded(s):
    lib, m = s["lib"], s["mesh"]
    k = 2 * math.pi * s["frequency"] / C0
    ok(lib.peec_gb300_inductance_retarded_device(C.byref(m.mesh), C.byref(m.dual), C.byref(s["lo"]), k,
                                                 s["L"].data_ptr(), None), "retarded Lp")
    ok(lib.peec_gb300_potential_retarded_device(C.byref(m.mesh), C.byref(m.dual), C.byref(s["po"]), k,
                                                s["P"].data_ptr(), None), "retarded P")
    ok(lib.peec_gb300_harmonic_build_retarded_device(s["L"].data_ptr(), s["P"].data_ptr(), s["edges"].data_ptr(), None,
                                                     m.n_edges, m.n_nodes, s["frequency"], s["Z"].data_ptr()), "fill")
    return {"L": s["L"], "P": s["P"], "Z": s["Z"]}


def run_real_lu(s):
    lib, n = s["lib"], s["ne"] + s["nv"]
    scale, column = C.c_double(), C.c_int()
    ok(lib.peec_gb300_copy_device(s["lu"].data_ptr(), s["M"].data_ptr(), n * n * 8), "copy")
    ok(lib.peec_gb300_lu_factor_device(s["lu"].data_ptr(), n, 1e-14, s["piv"].data_ptr(), s["perm"].data_ptr(),
                                       C.byref(scale), C.byref(column)), "real LU")
    ok(lib.peec_gb300_lu_solve_device(s["lu"].data_ptr(), s["perm"].data_ptr(), n, s["b"].data_ptr(),
                                      s["x"].data_ptr(), 1), "real solve")
    return {"lu": s["lu"], "pivots": s["piv"], "x": s["x"]}


def run_dropin(s):
    lib, Z, B, X = s["lib"], s["Z"], s["B"], s["X"]
    h = HostFactor(lib)
    c = C.POINTER(abi.Complex)
    ok(lib.complex_lu_factorize(Z.ctypes.data_as(c), len(Z), C.byref(s["opt"]), C.byref(h.f)), "complex LU")
    ok(lib.complex_lu_solve_multiple(C.byref(h.f), B.ctypes.data_as(c), X.ctypes.data_as(c), len(B), 1), "solve")
    n, f = len(Z), h.f
    return {"lu": h.view(f.data, (n, n), abi.Complex, np.complex128),
            "pivots": h.view(f.pivots, (n,), C.c_size_t, np.int64),
            "row_scale": h.view(f.row_scale, (n,), C.c_double, np.float64),
            "column_scale": h.view(f.column_scale, (n,), C.c_double, np.float64), "x": X}


def fill_system(s):
    lib, ne, nv, n = s["lib"], s["ne"], s["nv"], s["ne"] + s["nv"]
    ok(lib.peec_gb300_harmonic_build_device(s["L"].data_ptr(), s["P"].data_ptr(), s["edges"].data_ptr(), None, ne, nv,
                                            s["frequency"], s["Z"].data_ptr()), "fill")
    for q, (k, e) in enumerate(zip(s["k"], s["e"])):
        ok(lib.peec_gb300_plane_wave_rhs_device(s["centers"].data_ptr(), s["vectors"].data_ptr(), ne, nv, k, e,
                                                2 * math.pi * s["frequency"] / C0,
                                                s["B"].data_ptr() + q * n * 16), "plane wave")
    return n


def run_plain(s):
    lib, n = s["lib"], fill_system(s)
    scale, column = C.c_double(), C.c_int()
    ok(lib.peec_gb300_complex_lu_factor_device(s["Z"].data_ptr(), n, 1e-14, s["piv"].data_ptr(), s["perm"].data_ptr(),
                                               s["rows"].data_ptr(), s["cols"].data_ptr(), C.byref(scale),
                                               C.byref(column)), "complex LU")
    ok(lib.peec_gb300_complex_lu_solve_device(s["Z"].data_ptr(), s["perm"].data_ptr(), s["rows"].data_ptr(),
                                              s["cols"].data_ptr(), n, s["B"].data_ptr(), s["X"].data_ptr(),
                                              s["case"]["nrhs"]), "solve")
    return {"x": s["X"]}


def run_mixed(s):
    lib, n = s["lib"], fill_system(s)
    eta, it = C.c_double(), C.c_int()
    ok(lib.peec_gb300_complex_solve_mixed_device(s["Z"].data_ptr(), n, s["B"].data_ptr(), s["X"].data_ptr(),
                                                 s["case"]["nrhs"], TOL, MAX_ITER, C.byref(eta), C.byref(it)), "mixed")
    return {"x": s["X"]}


def run_sweep(s):
    ok(s["lib"].peec_gb300_sweep_run(s["plan"].handle, dbl(s["frequencies"]), len(s["frequencies"]), TOL,
                                     s["X"].data_ptr(), dbl(s["eta"]), s["fallback"].ctypes.data_as(abi.c_int_p)),
       "sweep")
    return {"x": s["X"]}


def step(s, system):
    lib, c = s["lib"], s["case"]
    ok(lib.peec_gb300_copy_device(s["state"].data_ptr(), s["rest"].data_ptr(), s["state"].numel() * 8), "copy")
    ok(lib.peec_gb300_transient_lightning_batch(
        system.handle, c["nrun"], dbl(s["K"]), dbl(s["alpha"]), dbl(s["beta"]), dbl(s["delay"]), s["strike"], s["ret"],
        0, c["steps"], s["state"].data_ptr(), s["probe_nodes"].data_ptr(), s["probe_nodes"].numel(),
        s["probe_edges"].data_ptr(), s["probe_edges"].numel(), s["probes"].data_ptr()), "lightning")
    return {"state": s["state"], "probes": s["probes"]}


def run(s):
    job = s["case"]["job"]
    if job == "lightning":
        return step(s, s["system"])
    if job == "lightning_new":
        return step(s, new_system(s))
    return {"assemble": run_assemble, "retarded": run_retarded, "real_lu": run_real_lu, "dropin": run_dropin,
            "plain": run_plain, "mixed": run_mixed, "sweep": run_sweep}[job](s)


# ---------------------------------------------------------------------
# least work of a pass
# ---------------------------------------------------------------------
def work(case):
    job = case["job"]
    ne, nv = counts(case)
    n = ne + nv
    real_lu, complex_lu = 2 / 3 * n ** 3, 8 / 3 * n ** 3
    if job in ("assemble", "retarded"):
        # 1/R at 32 x 32 points for the patch pairs of the upper triangles
        # (two half cells an edge, four quarter cells a node; a third of the
        # edge pairs or, on a plate, a half are parallel), ten operations each
        edge_pairs = (2 * ne) ** 2 / 2 * (0.36 if case["shape"] == "box" else 0.5)
        cells = nv - 2 if case["shape"] == "box" else case["nx"] * case["ny"]
        node_pairs = (4 * cells) ** 2 / 2
        out = 8 * (ne ** 2 + nv ** 2)
        if job == "retarded":  # at least the coarsest rule, 8 x 8 points
            return {"bytes": 2 * out + 16 * n * n, "flops": 30 * 64 * (edge_pairs + node_pairs)}
        return {"bytes": out, "flops": 10 * 1024 * (edge_pairs + node_pairs)}
    if job == "real_lu":
        return {"bytes": 16 * n * n, "flops": real_lu}
    if job == "dropin":
        return {"bytes": 32 * n * n, "flops": complex_lu + 8 * n * n * case["nrhs"]}
    if job in ("plain", "mixed"):
        return {"bytes": 8 * (ne ** 2 + nv ** 2) + 16 * n * case["nrhs"],
                "flops": complex_lu + 8 * n * n * case["nrhs"]}
    if job == "sweep":
        return {"bytes": 8 * (ne ** 2 + nv ** 2) + 16 * n * case["nrhs"] * case["nfreq"],
                "flops": case["nfreq"] * (complex_lu + 8 * n * n * case["nrhs"])}
    # a step reads the system once (an n x n FP64 operator, larger than the caches)
    step_bytes, step_flops = 8 * n * n, 2 * n * n * case["nrun"]
    build = real_lu if job == "lightning_new" else 0
    return {"bytes": case["steps"] * step_bytes + (8 * (ne ** 2 + nv ** 2) if build else 0),
            "flops": case["steps"] * step_flops + build}


# ---------------------------------------------------------------------
# the same results in plain FP64 torch
# ---------------------------------------------------------------------
def harmonic_matrix(d, frequency):
    """Z = [j w L, A; -P A^T, j w I] and the plane waves' right-hand sides."""
    ne, n, w = d["ne"], d["ne"] + d["nv"], 2 * math.pi * frequency
    A = incidence(d)
    e = torch.from_numpy(d["edges"]).long().cuda()
    Z = torch.zeros((n, n), dtype=torch.complex128, device="cuda")
    Z[:ne, :ne] = 1j * w * d["L"]
    Z[:ne, ne:] = A.to(torch.complex128)
    Z[ne:, :ne] = -(d["P"][:, e[:, 1]] - d["P"][:, e[:, 0]]).to(torch.complex128)
    Z[ne:, ne:].diagonal().fill_(1j * w)
    k0 = w / C0
    c, v, k, p = (torch.from_numpy(d[x]).cuda() for x in ("centers", "vectors", "k_hat", "e_hat"))
    h = 0.5 * k0 * (k @ v.T)
    B = torch.zeros((len(k), n), dtype=torch.complex128, device="cuda")
    B[:, :ne] = -(p @ v.T) * torch.sinc(h / math.pi) * torch.exp(-1j * k0 * (k @ c.T))
    return Z, B


def host_system(d):
    Z, B = harmonic_matrix(d, d["frequency"])
    return Z.cpu().numpy(), B.cpu().numpy()


def solve64(Z, B):
    """Z x = b for the rows of B: LU with two steps of refinement."""
    lu, piv = torch.linalg.lu_factor(Z)
    x = torch.linalg.lu_solve(lu, piv, B.T)
    for _ in range(2):
        x = x + torch.linalg.lu_solve(lu, piv, B.T - Z @ x)
    return x.T.contiguous()


def exact(case, seed):
    job = case["job"]
    if job in ("assemble", "retarded"):
        return None  # adaptive analytic panel integrals
    d = inputs(case, seed)
    if job == "real_lu":
        return {"lu": None, "pivots": None, "x": solve64(d["M"], d["b"][None, :])[0]}
    if job == "dropin":
        Z, B = host_system(d)
        x = solve64(torch.from_numpy(Z).cuda(), torch.from_numpy(B).cuda())
        return {"lu": None, "pivots": None, "row_scale": None, "column_scale": None, "x": x.cpu().numpy()}
    if job in ("plain", "mixed"):
        return {"x": solve64(*harmonic_matrix(d, d["frequency"]))}
    if job == "sweep":
        return {"x": torch.stack([solve64(*harmonic_matrix(d, float(f))) for f in d["frequencies"]])}
    # trapezoidal steps of [I; V] from rest
    M, A, AS, F = transient_matrix(d)
    lu, piv = torch.linalg.lu_factor(M)
    ne = d["ne"]
    I = torch.zeros((ne, case["nrun"]), dtype=torch.float64, device="cuda")
    V = torch.zeros((d["nv"], case["nrun"]), dtype=torch.float64, device="cuda")
    pn, pe = (torch.from_numpy(d[k]).long().cuda() for k in ("probe_nodes", "probe_edges"))
    probes = []

    def source(t):
        J = torch.zeros_like(V)
        i = torch.from_numpy(d["K"] * (np.exp(-d["alpha"] * t) - np.exp(-d["beta"] * t))).cuda()
        at = torch.arange(case["nrun"], device="cuda")
        J[torch.from_numpy(d["strike"]).cuda(), at] += i
        J[torch.from_numpy(d["ret"]).cuda(), at] -= i
        return J

    for k in range(case["steps"]):
        top = d["L"] @ I / DT - 0.5 * (AS @ V)
        low = F[:, None] * V / DT + 0.5 * (A.T @ I) + 0.5 * source(k * DT) + 0.5 * source((k + 1) * DT)
        b = torch.cat([top, low])
        x = torch.linalg.lu_solve(lu, piv, b)
        x = x + torch.linalg.lu_solve(lu, piv, b - M @ x)
        I, V = x[:ne], x[ne:]
        probes.append(torch.cat([V[pn], I[pe]]).T)
    return {"state": torch.cat([I, V]).T.contiguous(), "probes": torch.stack(probes)}
