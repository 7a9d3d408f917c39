"""The pressure CG with its matrix in shared memory (one tile of 2048 rows per
block; a cluster up to 16 tiles, the grid beyond): equal to the oracle bit for
bit around the sizes where the number of tiles or the last tile's rows change,
host-driven and in graph mode, and to the block forms in FP32."""
import numpy as np
import pytest

from test_gpu_dilu_flow import merged_polymesh

pytestmark = pytest.mark.gpu

# cells per axis: below a tile, one tile exactly and one row more, 2 and 3
# tiles, 16 tiles exactly and one more (cluster -> grid), 33 tiles with 33
# rows in the last
SIZES = [(7, 5, 3), (32, 16, 4), (683, 3, 1), (64, 8, 8), (61, 17, 4), (64, 32, 16), (3641, 3, 3), (69, 49, 20)]


def _case(x, ctx, mesh, prec="fp64", form=None, graph=False):
    model, config = x.cases.channel_case(mesh, iterations=2, precision=prec)
    cfg, keep = x.build_config(model, config)
    dm = x.DeviceMesh(ctx, mesh)
    c = x.Case(dm, cfg)
    c.set_inner_cg(1)
    if form is not None:
        c.set_persistent(form)
    c.set_graph_mode(graph)
    return c, (dm, cfg, keep)


def _run(x, c, mesh):
    rng = np.random.default_rng(5)
    c.set_field(x._abi.FIELD_U, 0.1 * rng.standard_normal((3, mesh.n_cells)))
    c.set_field(x._abi.FIELD_P, 0.01 * rng.standard_normal(mesh.n_cells))
    res, _ = c.simple_iterate(2)
    return res, c.get_field(x._abi.FIELD_U), c.get_field(x._abi.FIELD_P)


@pytest.mark.parametrize("n", SIZES + ["merged"])
def test_resident_parity(x, orc, ctx, n):
    pm = merged_polymesh(x, 30, 18, 12, 3, 4, 5) if n == "merged" else x.channel_polymesh(*n, seed=2)
    mesh = x.build_mesh3(pm)
    outs = []
    for graph in (False, True):
        c, keep = _case(x, ctx, mesh, graph=graph)
        outs.append(_run(x, c, mesh))
        c.close()
    o = orc.OracleCase(orc.OracleMesh.from_mesh3(mesh), keep[1])
    ref = _run(x, o, mesh)
    for out in outs:
        for a, b in zip(out, ref):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("n", SIZES)
def test_resident_fp32(x, ctx, n):
    mesh = x.build_mesh3(x.channel_polymesh(*n, seed=2))
    outs = []
    for form in (256, 1):
        c, keep = _case(x, ctx, mesh, "mixed", form)
        outs.append(_run(x, c, mesh))
        c.close()
    for a, b in zip(*outs):
        assert np.array_equal(a, b)


def test_resident_batch_mixed_sizes(x, ctx):
    """Members of 1, 2, 3 and 17 tiles: with the last one the clusters do not
    cover the batch, and one cooperative launch runs it; each equals itself
    alone."""
    meshes = [x.build_mesh3(x.channel_polymesh(*n, seed=2)) for n in (SIZES[0], SIZES[2], SIZES[4], SIZES[6])]
    for prec in ("fp64", "mixed"):
        for pick in (meshes[:3], meshes):
            alone = []
            for m in pick:
                c, keep = _case(x, ctx, m, prec)
                alone.append(_run(x, c, m))
                c.close()
            batch = x.api.Batch(ctx, 4, 1 << 34)
            members = []
            for m in pick:
                c, keep = _case(x, ctx, m, prec)
                rng = np.random.default_rng(5)
                c.set_field(x._abi.FIELD_U, 0.1 * rng.standard_normal((3, m.n_cells)))
                c.set_field(x._abi.FIELD_P, 0.01 * rng.standard_normal(m.n_cells))
                assert batch.add(c)
                members.append((c, keep))
            res = [batch.simple_iterate()[0] for _ in range(2)]
            for i, (c, keep) in enumerate(members):
                assert np.array_equal(np.array([r[i] for r in res]), alone[i][0])
                assert np.array_equal(c.get_field(x._abi.FIELD_P), alone[i][2])
            batch.close()
            for c, keep in members:
                c.close()


@pytest.mark.parametrize("n", [(7, 5, 3), (69, 49, 20)])
def test_resident_tables_only_where_read(x, ctx, n):
    """A system none of whose solves can be a resident CG holds no tables for
    it: a Jacobi-BiCGSTAB U against a Jacobi-CG U."""
    mesh = x.build_mesh3(x.channel_polymesh(*n, seed=2))
    size = {}
    for u in ("Bicgstab", "Cg"):
        model, config = x.cases.channel_case(mesh, iterations=2)
        s = config.solvers["U"]
        config.solvers["U"] = x.SolverSetup(solver=getattr(x, u)(), preconditioner=x.Jacobi(),
                                            convergence=s.convergence, relax=s.relax, rtol=s.rtol)
        cfg, keep = x.build_config(model, config)
        dm = x.DeviceMesh(ctx, mesh)
        c = x.Case(dm, cfg)
        size[u] = c.footprint()[0]
        c.close()
        dm.close()
    # two bytes per row at least
    assert size["Cg"] - size["Bicgstab"] >= 2 * mesh.n_cells, size
