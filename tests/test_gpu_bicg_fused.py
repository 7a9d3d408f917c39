"""BiCGSTAB of the three momentum components side by side (and of one scalar):
equal to the oracle bit for bit with each preconditioner, over one and many
iterations, at tile edges, with long rows, host-driven and in graph mode; on a
mesh whose walls couple the components (they are then solved in turn); in
mixed precision equal to the separate kernels (which profiling selects)."""
import numpy as np
import pytest

from test_gpu_dilu_flow import merged_polymesh

pytestmark = pytest.mark.gpu

MESHES = {
    "105": lambda x: x.channel_polymesh(7, 5, 3, seed=2),
    "2048": lambda x: x.channel_polymesh(32, 16, 4, seed=3),
    "2049": lambda x: x.channel_polymesh(683, 3, 1, seed=4),
    "merged": lambda x: merged_polymesh(x, 30, 9, 8, 3, 4, 5),
    "tilted": lambda x: tilted(x, 12, 9, 7),
}


def tilted(x, *n):
    """The channel turned by 30 degrees about z: wall normals with two components."""
    pm = x.channel_polymesh(*n, seed=5)
    c, s = np.cos(np.pi / 6), np.sin(np.pi / 6)
    pts = np.asarray(pm.points)
    pm.points = np.stack([c * pts[:, 0] - s * pts[:, 1], s * pts[:, 0] + c * pts[:, 1], pts[:, 2]], axis=1)
    return pm


def _config(x, mesh, pre, rtol, prec="fp64"):
    model, config = x.cases.channel_case(mesh, iterations=3, precision=prec)
    u = config.solvers["U"]
    config.solvers["U"] = x.SolverSetup(solver=x.Bicgstab(), preconditioner=pre() if pre else None,
                                        convergence=u.convergence, relax=u.relax, rtol=rtol)
    return x.build_config(model, config)


def _run(x, c, mesh):
    rng = np.random.default_rng(5)
    c.set_field(x._abi.FIELD_U, 0.1 * rng.standard_normal((3, mesh.n_cells)))
    c.set_field(x._abi.FIELD_P, 0.01 * rng.standard_normal(mesh.n_cells))
    res, _ = c.simple_iterate(3)
    return res, c.get_field(x._abi.FIELD_U), c.get_field(x._abi.FIELD_P)


@pytest.mark.parametrize("rtol", [0.1, 1e-9])
@pytest.mark.parametrize("pre", ["DILU", "Jacobi", None])
@pytest.mark.parametrize("name", list(MESHES))
def test_fused_parity(x, orc, ctx, name, pre, rtol):
    mesh = x.build_mesh3(MESHES[name](x))
    cfg, keep = _config(x, mesh, getattr(x, pre) if pre else None, rtol)
    ref = _run(x, orc.OracleCase(orc.OracleMesh.from_mesh3(mesh), cfg), mesh)
    for graph in (False, True):
        dm = x.DeviceMesh(ctx, mesh)
        c = x.Case(dm, cfg)
        c.set_graph_mode(graph)
        for a, b in zip(_run(x, c, mesh), ref):
            assert np.array_equal(a, b)
        c.close()
        dm.close()


@pytest.mark.parametrize("rtol", [0.1, 1e-7])
@pytest.mark.parametrize("pre", ["DILU", "Jacobi"])
@pytest.mark.parametrize("name", list(MESHES))
def test_fused_mixed(x, ctx, name, pre, rtol):
    mesh = x.build_mesh3(MESHES[name](x))
    cfg, keep = _config(x, mesh, getattr(x, pre), rtol, "mixed")
    outs = []
    for separate, graph in ((True, False), (False, False), (False, True)):
        dm = x.DeviceMesh(ctx, mesh)
        c = x.Case(dm, cfg)
        c.set_inner_cg(1)
        c.set_profiling(separate)
        c.set_graph_mode(graph)
        outs.append(_run(x, c, mesh) + (c.solve_report()["iterations"],))
        c.close()
        dm.close()
    for out in outs[1:]:
        for a, b in zip(outs[0], out):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_captured_step_is_the_same_under_profiling(x, ctx, prec):
    """A step captured in graph mode while profiling is on is the one captured
    with it off: as many launches, then and once profiling is off again."""
    mesh = x.build_mesh3(MESHES["2049"](x))
    counts = []
    for profiled in (False, True):
        cfg, keep = _config(x, mesh, x.DILU, 0.1, prec)
        dm = x.DeviceMesh(ctx, mesh)
        c = x.Case(dm, cfg)
        c.set_graph_mode(True)
        c.set_profiling(profiled)
        n = []
        for k in range(2):
            l0 = x.launch_count()
            out = _run(x, c, mesh)
            n.append(x.launch_count() - l0)
            c.set_profiling(False)
        counts.append(n)
        c.close()
        dm.close()
    assert counts[0][1] == counts[1][1], counts
