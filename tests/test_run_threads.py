"""The host threads of a plan's build: every item once, and an exception in one of them reaches the caller."""
import ctypes

import pytest


@pytest.mark.parametrize("n", [0, 1, 2, 33, 1000])
def test_run_threads(lib_built, n):
    from grgl_gb300 import _lib

    total = ctypes.c_longlong(-1)
    run = _lib.lib().grgx_debug_run_threads
    run.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.POINTER(ctypes.c_longlong)]
    assert run(n, -1, ctypes.byref(total)) == _lib.OK and total.value == n * (n - 1) // 2
    for fails in {0, n // 2, n - 1} if n else ():
        assert run(n, fails, ctypes.byref(total)) == _lib.ERR_OOM
    assert run(n, -1, ctypes.byref(total)) == _lib.OK
