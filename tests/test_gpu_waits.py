"""Waits that run out: a kernel whose rows or blocks wait for one another's
values ends by its poll limit when a value is never written, with its error
flag set, and the context keeps running work."""
import ctypes as C
from importlib import import_module

import pytest

pytestmark = pytest.mark.gpu

KINDS = {"dilu_factor": 0}


@pytest.mark.parametrize("kind", list(KINDS))
def test_wait_gives_up(x, ctx, kind):
    L = import_module(x.__name__ + "._lib").lib()
    gave, flag, after = C.c_int32(-1), C.c_int32(-1), C.c_int32(-1)
    code = L.xcal_check_wait(ctx.h, KINDS[kind], 1 << 15, C.byref(gave), C.byref(flag), C.byref(after))
    assert code == 0, L.xcal_last_error(ctx.h)
    assert (gave.value, flag.value, after.value) == (1, 1, 1)
    assert L.xcal_check_wait(ctx.h, KINDS[kind], 0, None, None, None) == x._abi.XCAL_ERR_INVALID
