"""Waits that run out: a kernel whose rows or blocks wait for one another's
values ends by its poll limit when a value is never written, with its error
flag set, and the context keeps running work; a case reports it once."""
import ctypes as C
from importlib import import_module

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = {"dilu_factor": 0, "dilu_lower": 1, "dilu_upper": 2, "fused": 3, "resident_cg": 4}


@pytest.mark.parametrize("kind", list(KINDS))
def test_wait_gives_up(x, ctx, kind):
    L = import_module(x.__name__ + "._lib").lib()
    gave, flag, after = C.c_int32(-1), C.c_int32(-1), C.c_int32(-1)
    code = L.xcal_check_wait(ctx.h, KINDS[kind], 1 << 15, C.byref(gave), C.byref(flag), C.byref(after))
    assert code == 0, L.xcal_last_error(ctx.h)
    assert (gave.value, flag.value, after.value) == (1, 1, 1)
    assert L.xcal_check_wait(ctx.h, KINDS[kind], 0, None, None, None) == x._abi.XCAL_ERR_INVALID
    assert L.xcal_check_wait(ctx.h, len(KINDS), 1, None, None, None) == x._abi.XCAL_ERR_INVALID


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("solver", ["Bicgstab", "Cg"])
def test_given_up_wait_is_reported_once(x, ctx, solver, prec):
    """The host-driven step after a wait that ran out ends as XCAL_ERR_TIMEOUT,
    the next one runs (DILU momentum solves, and a DILU-CG pressure solve)."""
    L = import_module(x.__name__ + "._lib").lib()
    mesh = x.build_mesh3(x.channel_polymesh(12, 6, 6, seed=1))
    model, config = x.cases.channel_case(mesh, iterations=3, precision=prec)
    if solver == "Cg":
        for name, pre in (("U", x.Jacobi), ("p", x.DILU)):
            config.solvers[name].preconditioner = pre()
    cfg, keep = x.build_config(model, config)
    dm = x.DeviceMesh(ctx, mesh)
    c = x.Case(dm, cfg)
    c.set_field(x._abi.FIELD_U, model.momentum.U)
    c.set_field(x._abi.FIELD_P, model.momentum.p)
    c.simple_iterate(1)
    assert L.xcal_case_check_wait(c.h, 1 << 10) == 0
    assert L.xcal_simple_iterate(c.h, 1, None, None, None) == x._abi.XCAL_ERR_TIMEOUT
    for _ in range(3):
        res, _ = c.simple_iterate(1)
        assert np.all(np.isfinite(res))
    assert L.xcal_case_check_wait(c.h, 0) == x._abi.XCAL_ERR_INVALID
    c.close()
    dm.close()
