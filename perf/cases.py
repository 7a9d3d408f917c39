"""The work that a user of this framework has it do, as cases that can be timed.

A case advances a flow through the public API: the program keeps a resident
Case (or Batch) on its mesh and hands it the initial fields from pinned host
memory, runs SIMPLE iterations or PISO steps, and reads the fields back into
pinned host memory.  Two cases go another way: a whole `run_` call (mesh in
hand, results out), and one linear equation written with the operator DSL.

Fields a case starts from are made from the seed; the mesh is made from the
case alone and, like any mesh, is uploaded once and shared by the program's
cases on it.
"""
from __future__ import annotations

import functools
import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package directory's name holds a dot, so it is loaded by path."""
    name = "xcalibre_b200"
    if name not in sys.modules:
        pkg = os.path.join(ROOT, "xcalibre.jl_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


x = _package()
A = x._abi


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # whole run! calls of the lid-driven cavity at the size of the 2D example: a short steady run
        # where set-up, launches and latency are what the user waits for
        {"name": "run_cavity80_fp64", "kind": "run", "flow": "cavity", "nx": 80, "ny": 80, "nz": 1,
         "precision": "fp64", "steps": 40},
        # the smallest serving requests, alone: a coarse 2D slab (design sweeps, unit-sized runs)
        {"name": "cavity_37x29_fp64", "kind": "simple", "flow": "cavity", "nx": 37, "ny": 29, "nz": 1,
         "precision": "fp64", "steps": 10},
        # a few tens of thousands of cells, odd counts per axis: the usual workstation case
        {"name": "channel_47x25x23_fp64", "kind": "simple", "flow": "channel", "nx": 47, "ny": 25, "nz": 23,
         "precision": "fp64", "steps": 5},
        # a quarter of a million cells in mixed precision: between the block forms of the small
        # cases and the whole-GPU forms of the large ones
        {"name": "channel_64_mixed", "kind": "simple", "flow": "channel", "nx": 64, "ny": 64, "nz": 64,
         "precision": "mixed", "steps": 4},
        # the 2.1M-cell permuted channel, plain FP64 (the headline steady case)
        {"name": "channel_128_fp64", "kind": "simple", "flow": "channel", "nx": 128, "ny": 128, "nz": 128,
         "precision": "fp64", "steps": 2},
        # the same channel in mixed precision
        {"name": "channel_128_mixed", "kind": "simple", "flow": "channel", "nx": 128, "ny": 128, "nz": 128,
         "precision": "mixed", "steps": 2},
        # DILU-preconditioned pressure, as the reference's examples use where Jacobi converges slowly
        {"name": "channel_71x41x40_dilu", "kind": "simple", "flow": "channel_dilu", "nx": 71, "ny": 41, "nz": 40,
         "precision": "fp64", "steps": 3},
        # transient LES: the 96^3 periodic Smagorinsky box, PISO, each step one captured graph
        {"name": "les_96_mixed", "kind": "piso", "flow": "les", "nx": 96, "ny": 96, "nz": 96,
         "precision": "mixed", "steps": 4},
        # transient LES with the subgrid k equation on an odd-sized channel, FP64, host-driven steps
        {"name": "keq_channel_61x33x31", "kind": "piso", "flow": "keq", "nx": 61, "ny": 33, "nz": 31,
         "precision": "fp64", "steps": 5},
        # RANS (k, omega and kl transport) on the 2D flat plate
        {"name": "lke_plate_150x50", "kind": "simple", "flow": "lke", "nx": 150, "ny": 50, "nz": 1,
         "precision": "fp64", "steps": 5},
        # serving: resident cavity and channel requests advanced together, mixed precision
        {"name": "batch16_mixed", "kind": "batch", "flow": "batch", "count": 16, "n_max": 30000, "stream": 0,
         "precision": "mixed", "steps": 4},
        # one scalar equation from the operator DSL, solved tightly (potential / wall distance / user equations)
        {"name": "poisson_63x50x41", "kind": "equation", "flow": "poisson", "nx": 63, "ny": 50, "nz": 41,
         "precision": "fp64", "steps": 1},
    ]


def draw(rng: random.Random):
    flow = rng.choice(["cavity", "channel", "channel", "channel", "channel_dilu", "les", "keq", "lke", "batch",
                       "poisson", "run"])
    mixed = rng.random() < 0.5

    def size(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    def box(n, aspect):
        """About n cells, each axis its own count around n^(1/3)."""
        a = n ** (1.0 / 3.0)
        ny = max(4, int(round(a / aspect ** (1.0 / 3.0) * rng.uniform(0.9, 1.1))))
        nz = max(4, int(round(a / aspect ** (1.0 / 3.0) * rng.uniform(0.9, 1.1))))
        return max(4, int(n / (ny * nz))), ny, nz

    if flow == "batch":
        return {"kind": "batch", "flow": "batch", "count": rng.randint(2, 20), "n_max": int(size(3e3, 6e4)),
                "stream": rng.randint(1, 1000), "precision": "mixed" if mixed else "fp64", "steps": 3}
    if flow in ("cavity", "lke", "run"):
        n = size(1e3, 6e4 if flow != "run" else 2e4)
        ny = max(8, int(round(math.sqrt(n / rng.uniform(1.0, 4.0)))))
        nx, nz = max(8, int(n / ny)), 1
    elif flow == "les":
        # the seeded spectral field needs an n^3 box
        nx = ny = nz = int(round(size(4e3, 9e5) ** (1.0 / 3.0)))
    else:
        hi = {"channel": 2.09e6, "channel_dilu": 4e5, "keq": 3e5, "poisson": 3e5}[flow]
        nx, ny, nz = box(size(2e3, hi), rng.uniform(1.0, 3.0))
    kind = {"cavity": "simple", "lke": "simple", "channel": "simple", "channel_dilu": "simple", "les": "piso",
            "keq": "piso", "poisson": "equation", "run": "run"}[flow]
    n = nx * ny * nz
    steps = {"run": 30, "equation": 1}.get(kind, 2 if n > 5e5 else 4)
    if flow in ("lke", "poisson", "keq") or kind == "run":
        mixed = False
    return {"kind": kind, "flow": "cavity" if flow == "run" else flow, "nx": nx, "ny": ny, "nz": nz,
            "precision": "mixed" if mixed else "fp64", "steps": steps}


# ---------------------------------------------------------------------------
# meshes, uploaded once per program
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _context():
    return x.Context(0)


@functools.lru_cache(maxsize=4)
def _mesh(flow, nx, ny, nz):
    if flow == "cavity":
        pm = x.cavity_polymesh(ny, nx=nx, lx=nx / ny, seed=1)
    elif flow == "lke":
        pm = x.flatplate_polymesh(nx, ny, seed=1)
    elif flow == "les":
        pm = x.periodic_box_polymesh(nx, seed=1)
    else:
        pm = x.channel_polymesh(nx, ny, nz, seed=1)
    return x.build_mesh3(pm, device=0)


@functools.lru_cache(maxsize=4)
def _device_mesh(flow, nx, ny, nz):
    return x.DeviceMesh(_context(), _mesh(flow, nx, ny, nz))


def _mesh_key(case):
    flow = {"channel_dilu": "channel", "keq": "channel", "poisson": "channel"}.get(case["flow"], case["flow"])
    return flow, case["nx"], case["ny"], case["nz"]


# ---------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------
def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    b = t.numpy()
    b[...] = a
    return b


def _smooth_noise(mesh, rng, amplitude, modes=6, axes=(1, 1, 1)):
    """A sum of seeded sine waves over the mesh's box (along `axes`): what a developing flow's disturbance looks like."""
    c = mesh.cell_centre
    span = np.maximum(c.max(axis=0) - c.min(axis=0), 1e-12)
    t = (c - c.min(axis=0)) / span
    out = np.zeros(mesh.n_cells)
    for _ in range(modes):
        k = rng.integers(1, 5, size=3) * np.array(axes)
        out += rng.standard_normal() * np.sin(2.0 * np.pi * (t @ k) + rng.uniform(0, 2.0 * np.pi))
    return amplitude / math.sqrt(modes) * out


def _model(case, mesh):
    """(model, config, pref) of the case's flow."""
    c, flow, prec, steps = x.cases, case["flow"], case["precision"], case["steps"]
    if flow == "cavity":
        return (*c.cavity_case(mesh, iterations=steps, precision=prec), 0.0)
    if flow == "lke":
        return (*c.lke_flatplate_case(mesh, iterations=steps, precision=prec), None)
    if flow == "les":
        raise ValueError("the LES box takes its initial field: see _flow")
    if flow == "keq":
        return (*c.kequation_channel_case(mesh, steps=steps, precision=prec), None)
    model, config = c.channel_case(mesh, iterations=steps, precision=prec)
    if flow == "channel_dilu":
        p = config.solvers["p"]
        config.solvers["p"] = x.SolverSetup(solver=x.Cg(), preconditioner=x.DILU(), convergence=p.convergence,
                                            relax=p.relax, rtol=p.rtol)
    return model, config, None


def _flow(case, mesh, seed):
    """Model, configuration, reference pressure and the initial fields of one seed."""
    rng = np.random.default_rng(seed)
    n = mesh.n_cells
    if case["flow"] == "les":
        U = x.cases.fourier_field(mesh, seed=seed)
        # one time step for every seed: CFL about 0.5 at the field's largest speeds
        dt = 0.1 * (2.0 * np.pi / case["nx"])
        model, config = x.cases.periodic_les_case(mesh, steps=case["steps"], dt=dt, U0=U, precision=case["precision"])
        zero = np.zeros(mesh.n_faces)
        return model, config, 0.0, {A.FIELD_U: U, A.FIELD_P: np.zeros(n), A.FIELD_NUT: np.zeros(n),
                                    A.FIELD_NUTF: zero}
    model, config, pref = _model(case, mesh)
    U = np.zeros((3, n))
    y, z = mesh.cell_centre[:, 1], mesh.cell_centre[:, 2]
    if case["flow"] == "lke":
        U[0] = 5.4 * (1.0 + _smooth_noise(mesh, rng, 0.02))
        U[1] = _smooth_noise(mesh, rng, 0.02)
    elif case["flow"] == "cavity":
        U[0] = _smooth_noise(mesh, rng, 0.05)
        U[1] = _smooth_noise(mesh, rng, 0.05)
    else:
        # a channel at start-up: a weak through-flow that varies across the section, which the inlet then
        # drives; the pressure solve meets the smooth error of a flow that adjusts along the whole channel
        U[0] = 0.16 * y * (1.0 - y) * z * (1.0 - z) * _smooth_noise(mesh, rng, 1.0, axes=(0, 1, 1))
    fields = {A.FIELD_U: U, A.FIELD_P: np.zeros(n)}
    if case["flow"] in ("lke", "keq"):
        k = 0.0575 if case["flow"] == "lke" else 1e-3
        fields[A.FIELD_K] = k * np.exp(_smooth_noise(mesh, rng, 0.1))
        fields[A.FIELD_NUT] = np.zeros(n)
        fields[A.FIELD_NUTF] = np.zeros(mesh.n_faces)
    if case["flow"] == "lke":
        fields[A.FIELD_OMEGA] = 275.0 * np.exp(_smooth_noise(mesh, rng, 0.1))
        fields[A.FIELD_KL] = 0.0115 * np.exp(_smooth_noise(mesh, rng, 0.1))
        fields[A.FIELD_NUT] = fields[A.FIELD_K] / fields[A.FIELD_OMEGA]
    return model, config, pref, fields


class _Resident:
    """One resident case, its initial fields and the buffers its results are read into (pinned host memory)."""

    def __init__(self, dmesh, model, config, pref, fields, graph):
        self.dmesh = dmesh
        cfg, self.keep = x.build_config(model, config, pref=pref)
        self.case = x.Case(dmesh, cfg)
        self.case.set_graph_mode(graph)
        self.fields = {f: _pinned(np.ascontiguousarray(v)) for f, v in fields.items()}
        # the state a program keeps of the flow: the fields it set, and the face mass flux
        self.out = {f: _pinned(np.zeros_like(v)) for f, v in fields.items() if f != A.FIELD_NUTF}
        self.out[A.FIELD_MDOTF] = _pinned(np.zeros(dmesh.mesh.n_faces))

    def start(self):
        for f, v in self.fields.items():
            self.case.set_field(f, v)
        self.case.initial_calculations()

    def results(self):
        return {"field%d" % f: self.case.get_field(f, out=o) for f, o in self.out.items()}


def prepare(case, seed):
    if case["kind"] == "batch":
        ctx = _context()
        reqs = _requests(case["count"], case["n_max"], case["stream"])
        batch = x.Batch(ctx, max_cases=case["count"], budget_bytes=60 << 30)
        members = []
        for i, r in enumerate(reqs):
            model, config, pref = r.config(case["precision"], 1500, 1e-6)
            rng = np.random.default_rng([seed, i])
            U = np.zeros((3, r.mesh.n_cells))
            for d in range(2 if r.kind == "cavity" else 3):
                U[d] = _smooth_noise(r.mesh, rng, 0.05)
            m = _Resident(_request_mesh(case["count"], case["n_max"], case["stream"], i), model, config, pref,
                          {A.FIELD_U: U, A.FIELD_P: np.zeros(r.mesh.n_cells)}, False)
            if not batch.add(m.case):
                raise RuntimeError("the batch is full")
            members.append(m)
        return {"case": case, "batch": batch, "members": members}
    mesh = _mesh(*_mesh_key(case))
    if case["kind"] == "equation":
        return {"case": case, **_equation(case, mesh, seed)}
    model, config, pref, fields = _flow(case, mesh, seed)
    if case["kind"] == "run":
        model.momentum.U[:] = fields[A.FIELD_U]
        model.momentum.p[:] = fields[A.FIELD_P]
        return {"case": case, "model": model, "config": config, "pref": pref, "fields": fields}
    # the LES box replays each time step as one graph; the other cases run as a Case does by default
    r = _Resident(_device_mesh(*_mesh_key(case)), model, config, pref, fields, graph=case["flow"] == "les")
    return {"case": case, "resident": r}


@functools.lru_cache(maxsize=2)
def _requests(count, n_max, stream):
    serve = importlib.import_module(x.__name__ + ".serve")
    reqs = serve.make_requests(count, seed=stream, n_min=1e3, n_max=n_max)
    for r in reqs:
        r.build()
    return reqs


@functools.lru_cache(maxsize=64)
def _request_mesh(count, n_max, stream, i):
    return x.DeviceMesh(_context(), _requests(count, n_max, stream)[i].mesh)


def _equation(case, mesh, seed):
    """(-Laplacian{Linear}(k, T) == -Source(S)) -> ScalarEquation(T, BCs) with seeded k (per face) and S."""
    rng = np.random.default_rng(seed)
    T = np.zeros(mesh.n_cells)
    k = np.exp(0.3 * rng.standard_normal(mesh.n_faces))
    S = _smooth_noise(mesh, rng, 1.0)
    model, config, pref = _model({**case, "flow": "channel"}, mesh)
    cfg, keep = x.build_config(model, config)
    host = x.Case(_device_mesh(*_mesh_key(case)), cfg)
    bcs = [x.Dirichlet("inlet", 1.0), x.Dirichlet("outlet", 0.0), x.Zerogradient("walls")]
    eqn = (-x.Laplacian[x.Linear](k, T) == -x.Source(S)) >> x.ScalarEquation(T, bcs)
    E = x.dsl.Equation(host, eqn)
    setup = x.SolverSetup(solver=x.Cg(), preconditioner=x.Jacobi(), convergence=1e-9, relax=1.0, rtol=1e-10,
                          atol=0.0, itmax=5000)
    return {"equation": E, "setup": setup, "T": T, "host": host, "keep": keep}


def run(state):
    case = state["case"]
    if case["kind"] == "run":
        m = state["model"]
        m.momentum.U[:] = state["fields"][A.FIELD_U]
        m.momentum.p[:] = state["fields"][A.FIELD_P]
        hist = x.run_(m, state["config"], pref=state["pref"])
        return {"U": m.momentum.U, "p": m.momentum.p, **hist}
    if case["kind"] == "equation":
        E = state["equation"]
        E.discretise()
        E.apply_boundary_conditions(state["T"])
        T, res, its = E.solve(state["setup"], state["T"])
        return {"T": T}
    if case["kind"] == "batch":
        for m in state["members"]:
            m.start()
        for _ in range(case["steps"]):
            res, conv = state["batch"].simple_iterate()
        fields = [m.results() for m in state["members"]]
        return {"res": res, **{k: np.concatenate([f[k].ravel() for f in fields]) for k in fields[0]}}
    r = state["resident"]
    r.start()
    if case["kind"] == "piso":
        res, co = r.case.piso_step(case["steps"])
        return {"res": res, "co": co, **r.results()}
    res, conv = r.case.simple_iterate(case["steps"])
    return {"res": res, **r.results()}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Per step: the momentum and pressure systems assembled, and each solved
    with a number of Krylov iterations that grows with the cells across the
    box (CG to a tenth of its start: about 5 per cell of the longest axis in
    3D); an iteration reads its matrix (value and column) once and its
    vectors once."""
    s = 4 if case["precision"] == "mixed" else 8
    if case["kind"] == "batch":
        sizes = [(r.dims, 5) if r.kind == "cavity" else (r.dims, 7) for r in _make(case)]
    else:
        sizes = [((case["nx"], case["ny"], case["nz"]), 5 if case["nz"] == 1 else 7)]
    total = 0.0
    for dims, width in sizes:
        n = dims[0] * dims[1] * dims[2]
        its = 5.0 * max(dims) if case["kind"] != "piso" else 1.5 * max(dims)
        if case["kind"] == "equation":
            its = 8.0 * max(dims)
        cg = n * (width * (s + 4) + 8 * s)
        momentum = 0 if case["kind"] == "equation" else 3 * 4 * n * (2 * width * (s + 4) + 10 * s)
        assembly = n * 8 * 60
        total += case["steps"] * (its * cg + momentum + assembly)
    return {"bytes": float(total), "flops": float(total / 5.0)}


def _make(case):
    serve = importlib.import_module(x.__name__ + ".serve")
    return serve.make_requests(case["count"], seed=case["stream"], n_min=1e3, n_max=case["n_max"])


# ---------------------------------------------------------------------------
# in 64 bits, without the package's solvers
# ---------------------------------------------------------------------------
def exact(case, seed):
    """The DSL equation's solution by a plain torch CG to rounding; the
    nonlinear flow iterations have no value of their own to compare with."""
    if case["kind"] != "equation":
        return None
    mesh = _mesh(*_mesh_key(case))
    rng = np.random.default_rng(seed)
    k = np.exp(0.3 * rng.standard_normal(mesh.n_faces))
    S = _smooth_noise(mesh, rng, 1.0)
    dev = torch.device("cuda")
    nb = mesh.n_bfaces
    own = torch.from_numpy(np.asarray(mesh.face_owner, dtype=np.int64)).to(dev)
    nei = torch.from_numpy(np.asarray(mesh.face_neigh, dtype=np.int64)).to(dev)
    g = torch.from_numpy(k * mesh.face_area / mesh.face_delta).to(dev)
    o, m, gi = own[nb:], nei[nb:], g[nb:]
    n = mesh.n_cells
    diag = torch.zeros(n, dtype=torch.float64, device=dev)
    # the sign rule makes both sides negative: -div(k grad T) = -S, integrated over each cell
    diag.index_add_(0, o, gi)
    diag.index_add_(0, m, gi)
    b = torch.from_numpy(-S * mesh.cell_volume).to(dev)
    for name, value in (("inlet", 1.0), ("outlet", 0.0)):
        r = mesh.patch_range(name)
        diag.index_add_(0, own[r.start:r.stop], g[r.start:r.stop])
        b.index_add_(0, own[r.start:r.stop], g[r.start:r.stop] * value)

    def apply(v):
        y = diag * v
        y.index_add_(0, o, -gi * v[m])
        y.index_add_(0, m, -gi * v[o])
        return y

    T = torch.zeros_like(b)
    r = b.clone()
    z = r / diag
    p = z.clone()
    rz = torch.dot(r, z)
    stop = 1e-28 * rz
    for _ in range(4000):
        q = apply(p)
        a = rz / torch.dot(p, q)
        T += a * p
        r -= a * q
        z = r / diag
        new = torch.dot(r, z)
        if new < stop:
            break
        p = z + (new / rz) * p
        rz = new
    return {"T": T.cpu().numpy()}
