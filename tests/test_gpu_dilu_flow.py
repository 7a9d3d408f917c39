"""DILU sweeps and factor as a dataflow (every row waits for the values it
reads): equal to the oracle bit for bit at the sizes where the row and chunk
bookkeeping changes (a warp, a 256-row chunk and their neighbours), with rows
of more entries than a thread holds in registers, host-driven, in graph mode
and in a batch; FP32 inner solves equal to the per-level kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def merged_polymesh(x, nx, ny, nz, seed, first, count):
    """The channel's mesh with rows of `count` cells along x merged into one
    cell each (faces inside a merged cell dropped), so a cell has up to
    4 count + 2 neighbours; the cell at (first, 1, 1) takes the highest number
    and the one at (first, 2, 2) the lowest, so one row has all its entries
    below the diagonal and another all above."""
    pm = x.channel_polymesh(nx, ny, nz, seed=None)
    nc = nx * ny * nz
    rep = np.arange(nc)
    heads = []
    for j, k in ((1, 1), (2, 2)):
        ids = [first + i + nx * (j + ny * k) for i in range(count)]
        rep[ids] = ids[0]
        heads.append(ids[0])
    rng = np.random.default_rng(seed)
    order = [heads[1]] + [c for c in rng.permutation(np.unique(rep)) if c not in heads] + [heads[0]]
    new = np.empty(nc, dtype=np.int64)
    new[order] = np.arange(len(order))
    cell = new[rep]
    nI = pm.n_internal_faces
    off, nodes = np.asarray(pm.face_offsets), np.asarray(pm.face_nodes)
    o, n = cell[pm.owner], cell[pm.neighbour]
    faces, own, nei = [], [], []
    for f in range(pm.n_faces):
        q = nodes[off[f]:off[f + 1]]
        if f < nI:
            if o[f] == n[f]:
                continue
            a, b = int(o[f]), int(n[f])
            faces.append(q if a < b else q[::-1])
            own.append(min(a, b))
            nei.append(max(a, b))
        else:
            faces.append(q)
            own.append(int(o[f]))
    return type(pm)(points=pm.points, face_offsets=np.cumsum([0] + [len(q) for q in faces]).astype(np.int32),
                    face_nodes=np.concatenate(faces).astype(np.int32), owner=np.array(own, dtype=np.int32),
                    neighbour=np.array(nei, dtype=np.int32), patch_names=list(pm.patch_names),
                    patch_sizes=list(pm.patch_sizes))


MESHES = {
    "31": lambda x: x.channel_polymesh(31, 1, 1, seed=1),
    "32": lambda x: x.channel_polymesh(4, 4, 2, seed=2),
    "33": lambda x: x.channel_polymesh(11, 3, 1, seed=3),
    "255": lambda x: x.channel_polymesh(17, 5, 3, seed=4),
    "256": lambda x: x.channel_polymesh(16, 4, 4, seed=5),
    "257": lambda x: x.channel_polymesh(257, 1, 1, seed=None),  # 257 levels
    "4620": lambda x: x.channel_polymesh(22, 15, 14, seed=6),
    "merged": lambda x: merged_polymesh(x, 9, 6, 6, 7, 2, 3),
}


def _config(x, mesh, prec="fp64"):
    model, config = x.cases.channel_case(mesh, iterations=3, precision=prec)
    p = config.solvers["p"]
    config.solvers["p"] = x.SolverSetup(solver=x.Cg(), preconditioner=x.DILU(), convergence=p.convergence,
                                        relax=p.relax, rtol=0.05)
    return x.build_config(model, config)


def _start(x, c, mesh):
    rng = np.random.default_rng(3)
    c.set_field(x._abi.FIELD_U, 0.1 * rng.standard_normal((3, mesh.n_cells)))
    c.set_field(x._abi.FIELD_P, np.zeros(mesh.n_cells))


def _run(x, c, mesh, iters=3):
    _start(x, c, mesh)
    res, _ = c.simple_iterate(iters)
    return res, c.get_field(x._abi.FIELD_U), c.get_field(x._abi.FIELD_P)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("name", list(MESHES))
def test_dilu_flow_parity(x, orc, ctx, name, graph):
    mesh = x.build_mesh3(MESHES[name](x))
    if name == "merged":
        assert np.diff(mesh.cell_faces_offset).max() == 14
    cfg, keep = _config(x, mesh)
    dm = x.DeviceMesh(ctx, mesh)
    g = x.Case(dm, cfg)
    g.set_graph_mode(graph)
    o = orc.OracleCase(orc.OracleMesh.from_mesh3(mesh), cfg)
    for a, b in zip(_run(x, g, mesh), _run(x, o, mesh)):
        assert np.array_equal(a, b)
    g.close()
    dm.close()


@pytest.mark.parametrize("name", ["33", "4620", "merged"])
def test_dilu_flow_mixed_and_batch(x, ctx, name):
    """Mixed precision: the default sweeps equal the per-level kernels, alone
    and as a batch member beside a case of another size."""
    mesh, other = x.build_mesh3(MESHES[name](x)), x.build_mesh3(MESHES["257"](x))
    out = []
    for mode in (2, 0):
        cfg, keep = _config(x, mesh, "mixed")
        dm = x.DeviceMesh(ctx, mesh)
        c = x.Case(dm, cfg)
        c.set_inner_cg(1)
        c.set_dilu_mode(mode)
        out.append(_run(x, c, mesh))
        c.close()
        dm.close()
    batch = x.api.Batch(ctx, 2, 1 << 33)
    members = []
    for m in (other, mesh):
        cfg, keep = _config(x, m, "mixed")
        dm = x.DeviceMesh(ctx, m)
        c = x.Case(dm, cfg)
        _start(x, c, m)
        assert batch.add(c)
        members.append((c, dm, keep))
    res = np.array([batch.simple_iterate()[0][1] for _ in range(3)])
    c = members[1][0]
    out.append((res, c.get_field(x._abi.FIELD_U), c.get_field(x._abi.FIELD_P)))
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a, b)
    batch.close()
    for c, dm, _ in members:
        c.close()
        dm.close()


@pytest.mark.parametrize("modes", [(0, 2), (0, 1), (3, 1), (0, 3, 2)])
def test_dilu_form_changed_between_steps(x, ctx, modes):
    """A DILU-CG whose solves run captured chunks of iterations takes another
    form between host-driven steps: the same results as without the change."""
    mesh = x.build_mesh3(MESHES["4620"](x))
    out = []
    for ms in ((0,) * len(modes), modes):
        cfg, keep = _config(x, mesh)
        cfg.p_solver.rtol = 1e-12
        dm = x.DeviceMesh(ctx, mesh)
        c = x.Case(dm, cfg)
        _start(x, c, mesh)
        its = []
        for m in ms:
            c.set_dilu_mode(m)
            # U, then p: the step calls are host-driven whatever the iteration
            c.initial_calculations()
            c.solve_equation(x._abi.EQN_U)
            c.pressure_predictor()
            c.flux_divergence()
            c.solve_equation(x._abi.EQN_P)
            its.append(int(c.solve_report()["iterations"][3]))
        assert min(its) > 60, its  # chunks of 4, 8, 16 and captured ones of 32
        out.append((its, c.get_field(x._abi.FIELD_U), c.get_field(x._abi.FIELD_P)))
        c.close()
        dm.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("before", [False, True])
def test_dilu_mode_back_to_default(x, ctx, before):
    """Mode 0 after another mode, set before or after the first step, is a new
    case's choice: the same forms and as many launches per step."""
    mesh = x.build_mesh3(MESHES["4620"](x))
    out = []
    for modes in ((), (1, 0), (2, 0), (3, 0)):
        cfg, keep = _config(x, mesh, "mixed")
        dm = x.DeviceMesh(ctx, mesh)
        c = x.Case(dm, cfg)
        _start(x, c, mesh)
        if before:
            for m in modes:
                c.set_dilu_mode(m)
        c.simple_iterate(1)
        if not before:
            for m in modes:
                c.set_dilu_mode(m)
            _start(x, c, mesh)
        t = c.tuning()
        l0 = x.launch_count()
        c.simple_iterate(1)
        out.append((t, x.launch_count() - l0))
        c.close()
        dm.close()
    assert out[0][0]["U"]["dilu_grid"] and out[0][0]["p"]["dilu_grid"]
    for o in out[1:]:
        assert o[0] == out[0][0]
        assert o[1] == out[0][1]


_SIZE_CLASS = """
import sys
sys.path.insert(0, sys.argv[1])
prec, sizes = sys.argv[2], [tuple(map(int, a.split("x"))) for a in sys.argv[3:]]
import numpy as np
import __graft_entry__ as ge
x = ge.load_package()
ctx = x.Context(0)
n = []
for dims in sizes:
    mesh = x.build_mesh3(x.channel_polymesh(*dims))
    model, config = x.cases.channel_case(mesh, iterations=2, precision=prec)
    u = config.solvers["U"]
    config.solvers["U"] = x.SolverSetup(solver=x.Cg(), preconditioner=x.Jacobi(), convergence=u.convergence,
                                        relax=u.relax, rtol=u.rtol)
    config.solvers["p"].preconditioner = x.DILU()
    cfg, keep = x.build_config(model, config)
    c = x.Case(x.DeviceMesh(ctx, mesh), cfg)
    l0 = x.launch_count()
    c.tuning()
    n.append(x.launch_count() - l0)
    l0 = x.launch_count()
    c.tuning()
    assert x.launch_count() == l0
    c.close()
print("trials", *n)
"""


def _trials(prec, *sizes):
    """Kernels each case's tuning launched, the cases made in turn in a process
    of its own (choices are kept per process); only p's DILU is tuned."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _SIZE_CLASS, root, prec, *sizes], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return [int(v) for v in r.stdout.split("trials")[1].split()]


def test_dilu_form_timed_above_the_untimed_sizes():
    """524,288 rows take the dataflow untimed, 720,000 (of the same power of
    two) have their forms timed although a case of the first size came before."""
    n = _trials("fp64", "128x64x64", "100x90x80")
    assert n[0] == 0 and n[1] >= 9, n  # three forms, each at least three times


@pytest.mark.parametrize("prec,dims,one_block", [("mixed", (7, 73, 1), False), ("mixed", (8, 8, 8), True),
                                                 ("mixed", (819, 5, 1), True), ("mixed", (16, 16, 16), False),
                                                 ("fp64", (8, 8, 8), False)])
def test_dilu_form_of_small_systems(x, ctx, prec, dims, one_block):
    """A DILU-CG in mixed precision runs one-block sweeps at 512 to 4,095 rows
    and the dataflow at 511 and 4,096, with the results of the level kernels; a
    BiCGSTAB (fused) and FP64 take the dataflow."""
    mesh = x.build_mesh3(x.channel_polymesh(*dims, seed=2))
    out = []
    for mode in (0, 2):
        cfg, keep = _config(x, mesh, prec)
        dm = x.DeviceMesh(ctx, mesh)
        c = x.Case(dm, cfg)
        c.set_inner_cg(1)
        c.set_dilu_mode(mode)
        if mode == 0:
            t = c.tuning()
            assert t["p"]["dilu_one_block"] == one_block and not t["U"]["dilu_one_block"]
        out.append(_run(x, c, mesh))
        c.close()
        dm.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
