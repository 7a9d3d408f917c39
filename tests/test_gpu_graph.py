"""Graph mode: a SIMPLE iteration / PISO step replayed as one CUDA graph with
device-driven Krylov loops (conditional WHILE nodes) gives the same results,
bit for bit, as host-polled steps and as the default, which replays small FP64
cases from their third step on -- FP64 and mixed precision, steady and
transient (periodic LES)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(x, ctx, mesh, model, config, graph, steps, pref=None, piso=False):
    cfg, keep = x.build_config(model, config, pref=pref)
    dm = x.DeviceMesh(ctx, mesh)
    c = x.Case(dm, cfg)
    c.set_field(x._abi.FIELD_U, model.momentum.U)
    c.set_field(x._abi.FIELD_P, model.momentum.p)
    c.set_graph_mode(True if graph else None)  # None: host-polled, whatever the size
    if piso:
        res, co = c.piso_step(steps)
    else:
        res, conv = c.simple_iterate(steps)
        co = None
    return res, co, c.get_field(x._abi.FIELD_U), c.get_field(x._abi.FIELD_P), (c, dm, keep)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_graph_simple_identical(x, ctx, prec):
    mesh = x.build_mesh3(x.channel_polymesh(16, 8, 8, seed=11))
    out = []
    for graph in (False, True):
        model, config = x.cases.channel_case(mesh, iterations=6, precision=prec)
        out.append(_run(x, ctx, mesh, model, config, graph, 6))
    (r0, _, U0, p0, _), (r1, _, U1, p1, _) = out
    assert np.array_equal(r0, r1), (r0, r1)
    assert np.array_equal(U0, U1) and np.array_equal(p0, p1)


def test_graph_cavity_dilu_identical(x, ctx):
    mesh = x.build_mesh3(x.cavity_polymesh(20))
    out = []
    for graph in (False, True):
        model, config = x.cases.cavity_case(mesh, iterations=10)
        out.append(_run(x, ctx, mesh, model, config, graph, 10, pref=0.0))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][2], out[1][2]) and np.array_equal(out[0][3], out[1][3])


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_graph_piso_periodic_identical(x, ctx, prec):
    mesh = x.build_mesh3(x.periodic_box_polymesh(10, seed=4))
    U0 = x.cases.fourier_field(mesh, seed=4)
    out = []
    for graph in (False, True):
        model, config = x.cases.periodic_les_case(mesh, steps=4, U0=U0, precision=prec)
        out.append(_run(x, ctx, mesh, model, config, graph, 4, pref=0.0, piso=True))
    (r0, c0, U0_, p0, _), (r1, c1, U1, p1, _) = out
    assert np.array_equal(r0, r1), (r0, r1)
    assert np.array_equal(c0, c1)
    assert np.array_equal(U0_, U1) and np.array_equal(p0, p1)


def test_graph_launch_count_reported(x, ctx):
    """Launch counting follows the kernels the WHILE bodies actually ran."""
    mesh = x.build_mesh3(x.channel_polymesh(12, 6, 6, seed=1))
    model, config = x.cases.channel_case(mesh, iterations=3)
    cfg, keep = x.build_config(model, config)
    dm = x.DeviceMesh(ctx, mesh)
    c = x.Case(dm, cfg)
    c.set_field(x._abi.FIELD_U, model.momentum.U)
    c.set_field(x._abi.FIELD_P, model.momentum.p)
    c.simple_iterate(1)
    c.set_graph_mode(True)
    l0 = x.launch_count()
    c.simple_iterate(2)
    n = x.launch_count() - l0
    assert n > 50, n


def test_autotuner_choices(x, ctx):
    """The autotuner picks a valid launch shape per equation; parity with the
    oracle under those shapes is covered by the SIMPLE parity tests (they run
    through simple_iterate, which tunes first)."""
    mesh = x.build_mesh3(x.channel_polymesh(24, 12, 12, seed=5))
    model, config = x.cases.channel_case(mesh, iterations=2)
    cfg, keep = x.build_config(model, config)
    dm = x.DeviceMesh(ctx, mesh)
    c = x.Case(dm, cfg)
    t = c.tuning()
    assert t["U"]["spmv_rows_per_thread"] in (0, 1, 2, 4)
    assert t["U"]["spmv_block"] in (128, 256, 512)
    assert isinstance(t["U"]["dilu_one_block"], bool)
    c.set_field(x._abi.FIELD_U, model.momentum.U)
    c.set_field(x._abi.FIELD_P, model.momentum.p)
    r1, _ = c.simple_iterate(2)
    # a second case of the same size class reuses the cached choices
    c2 = x.Case(x.DeviceMesh(ctx, mesh), cfg)
    assert c2.tuning() == t


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_persistent_cg_identical(x, ctx, prec):
    """The pressure CG as one launch (q on chip) gives the two-kernel loop's
    results bit for bit, in each form: the automatic choice, the cluster form
    (14 tiles: one 16-block cluster, hardware barriers), the 1024-, 512-
    and 256-thread cooperative forms forced, and the one-block-per-SM forms
    (here one tile per block)."""
    mesh = x.build_mesh3(x.channel_polymesh(48, 24, 24, seed=6))
    out = []
    modes = (False, True, 2, 1024, 512, 256, 4, 5)
    for persist in modes:
        model, config = x.cases.channel_case(mesh, iterations=4, precision=prec)
        cfg, keep = x.build_config(model, config)
        dm = x.DeviceMesh(ctx, mesh)
        c = x.Case(dm, cfg)
        c.set_persistent(persist)
        c.set_inner_cg(1)  # mixed: the canonical FP32 kernels in every form
        c.set_field(x._abi.FIELD_U, model.momentum.U)
        c.set_field(x._abi.FIELD_P, model.momentum.p)
        c.set_profiling(True)
        res, _ = c.simple_iterate(4)
        ms, its = c.profile(5)
        out.append((res, c.get_field(x._abi.FIELD_U), c.get_field(x._abi.FIELD_P), its))
    assert out[0][3] == 0                        # the persistent kernel ran only when enabled
    for m, o in zip(modes[1:], out[1:]):
        assert o[3] > 0, m
        assert np.array_equal(out[0][0], o[0]), m
        assert np.array_equal(out[0][1], o[1]) and np.array_equal(out[0][2], o[2]), m


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_persistent_multi_tile_identical(x, ctx, prec):
    """One block per SM owning several tiles (160 tiles over at most 148
    blocks: some blocks run two) gives the two-kernel loop's results bit for
    bit, with 1024 and with 512 threads per block."""
    mesh = x.build_mesh3(x.channel_polymesh(80, 64, 64, seed=9))
    assert mesh.n_cells > 148 * 2048
    out = []
    for persist in (False, 4, 5):
        model, config = x.cases.channel_case(mesh, iterations=2, precision=prec)
        cfg, keep = x.build_config(model, config)
        dm = x.DeviceMesh(ctx, mesh)
        c = x.Case(dm, cfg)
        c.set_persistent(persist)
        c.set_inner_cg(1)
        c.set_field(x._abi.FIELD_U, model.momentum.U)
        c.set_field(x._abi.FIELD_P, model.momentum.p)
        c.set_profiling(True)
        res, _ = c.simple_iterate(2)
        ms, its = c.profile(5)
        out.append((res, c.get_field(x._abi.FIELD_U), c.get_field(x._abi.FIELD_P), its))
        c.close()
        dm.close()
    assert out[0][3] == 0
    for o in out[1:]:
        assert o[3] > 0
        assert np.array_equal(out[0][0], o[0])
        assert np.array_equal(out[0][1], o[1]) and np.array_equal(out[0][2], o[2])


_FIRST_RUN = """
import sys
sys.path.insert(0, sys.argv[1])
import __graft_entry__ as ge
x = ge.load_package()
ctx = x.Context(0)
mesh = x.build_mesh3(x.channel_polymesh(16, 8, 8, seed=1))
n = []
for k in range(2):
    model, config = x.cases.channel_case(mesh, iterations=2, precision=sys.argv[2])
    cfg, keep = x.build_config(model, config)
    dm = x.DeviceMesh(ctx, mesh)
    c = x.Case(dm, cfg)
    c.set_field(x._abi.FIELD_U, model.momentum.U)
    c.set_field(x._abi.FIELD_P, model.momentum.p)
    l0 = x.launch_count()
    c.simple_iterate(2)
    n.append(x.launch_count() - l0)
    if k == 0:
        c.tuning()
    c.close()
    dm.close()
print("launches", *n)
"""


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_no_trials_for_fused_solves(prec):
    """The first case of a process launches no trials of kernels its solves do
    not run: as many launches as a second one, whose choices are cached."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _FIRST_RUN, root, prec], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    n = [int(v) for v in r.stdout.split("launches")[1].split()]
    assert n[0] == n[1], n


def _replay_modes(x, ctx, mesh, build, step, names):
    """Seven FP64 steps, the fields set anew before the fifth, never replayed,
    replayed from the third on (the default) and always: results, launches of
    the last step and reports per mode."""
    out = []
    for mode in (None, False, True):
        model, config, pref, fields = build()
        cfg, keep = x.build_config(model, config, pref=pref)
        dm = x.DeviceMesh(ctx, mesh)
        c = x.Case(dm, cfg)
        c.set_graph_mode(mode)
        res = []
        for k in range(7):
            if k in (0, 4):
                for f, v in fields(k).items():
                    c.set_field(getattr(x._abi, f), v)
            l0 = x.launch_count()
            res.append(step(c))
            launches = x.launch_count() - l0
        out.append((np.array(res), [c.get_field(getattr(x._abi, f)) for f in names], c.solve_report(), launches))
        c.close()
        dm.close()
    for o in out[1:]:
        assert np.array_equal(o[0], out[0][0])
        for a, b in zip(o[1], out[0][1]):
            assert np.array_equal(a, b)
        for key in ("iterations", "status"):
            assert np.array_equal(o[2][key], out[0][2][key]), key
        assert o[2]["itmax_hits"] == out[0][2]["itmax_hits"]
    # the default's last step is the captured one, the first mode's is not
    assert out[1][3] == out[2][3] != out[0][3], [o[3] for o in out]


@pytest.mark.parametrize("pre", ["Jacobi", "DILU"])
def test_replayed_steps_equal_host_driven(x, ctx, pre):
    mesh = x.build_mesh3(x.channel_polymesh(16, 8, 8, seed=11))

    def build():
        model, config = x.cases.channel_case(mesh, iterations=7)
        config.solvers["p"].preconditioner = getattr(x, pre)()
        config.solvers["p"].itmax = 25  # some solves stop there
        rng = np.random.default_rng(3)
        U = [0.1 * rng.standard_normal((3, mesh.n_cells)) for _ in range(2)]
        return model, config, None, lambda k: {"FIELD_U": U[k // 4], "FIELD_P": np.zeros(mesh.n_cells)}

    _replay_modes(x, ctx, mesh, build, lambda c: c.simple_iterate(1)[0][0], ("FIELD_U", "FIELD_P", "FIELD_MDOTF"))


def test_replayed_piso_steps_equal_host_driven(x, ctx):
    mesh = x.build_mesh3(x.periodic_box_polymesh(10, seed=4))
    U = [x.cases.fourier_field(mesh, seed=s) for s in (4, 5)]

    def build():
        model, config = x.cases.periodic_les_case(mesh, steps=7, U0=U[0])
        return model, config, 0.0, lambda k: {"FIELD_U": U[k // 4], "FIELD_P": np.zeros(mesh.n_cells)}

    _replay_modes(x, ctx, mesh, build, lambda c: np.append(c.piso_step(1)[0][0], c.max_courant()),
                  ("FIELD_U", "FIELD_P", "FIELD_NUT"))


def test_replayed_komega_steps_equal_host_driven(x, ctx):
    from test_gpu_komega import komega_channel_case
    mesh = x.build_mesh3(x.channel_polymesh(14, 8, 8, seed=2))
    n = mesh.n_cells

    def build():
        model, config = komega_channel_case(x, mesh, 7, "DILU")
        U = np.zeros((3, n))
        U[0] = 1.0
        return model, config, None, lambda k: {"FIELD_U": U * (1.0 + 0.1 * k), "FIELD_P": np.zeros(n),
                                               "FIELD_K": np.full(n, 0.01), "FIELD_OMEGA": np.full(n, 10.0),
                                               "FIELD_NUT": np.full(n, 1e-3)}

    _replay_modes(x, ctx, mesh, build, lambda c: c.simple_iterate(1)[0][0],
                  ("FIELD_U", "FIELD_P", "FIELD_K", "FIELD_OMEGA", "FIELD_NUT"))
