"""Calls of entry points with plain numbers (``host_call.c``) and its stand-in through ctypes: every argument arrives, whatever
registers and places of the stack the two kinds of arguments take."""
import ctypes
from ctypes import c_float, c_int, c_longlong, c_void_p

import numpy as np
import pytest

from zlm_b200.csrc.build import _through_ctypes, host_call

CALLS = [pytest.param(host_call(), id="host_call"), pytest.param(_through_ctypes, id="ctypes")]

# kinds of an entry point's arguments: i int, p pointer, l long long, f float
SIGNATURES = ["", "i", "f", "pipif", "f" * 8, "i" * 6 + "f" + "p" * 4, "ppifpilfppi" * 3, "i" * 8 + "p" + "f" + "i" * 30 + "l" + "fffffff"]


@pytest.mark.parametrize("call", CALLS)
@pytest.mark.parametrize("signature", SIGNATURES)
def test_arguments_arrive(call, signature):
    types = {"i": c_int, "p": c_void_p, "l": c_longlong, "f": c_float}
    got = []
    entry = ctypes.CFUNCTYPE(c_int, *(types[s] for s in signature))(lambda *a: (got.extend(a), -7)[1])
    given, want = [], []
    for n, s in enumerate(signature):
        if s == "f":
            given.append(c_float(n + 0.3))
            want.append(c_float(n + 0.3).value)
        elif s == "p":
            given.append([None, 0x7FFF_1234_5678 + n, c_void_p(0x7FFF_0000_0000 + n)][n % 3])
            want.append([None, 0x7FFF_1234_5678 + n, 0x7FFF_0000_0000 + n][n % 3])
        elif s == "l":
            given.append(-(1 << 40) - n)
            want.append(-(1 << 40) - n)
        else:
            given.append([n - 5, np.int64(n), c_int(-n), n % 2 == 0][n % 4])
            want.append([n - 5, n, -n, int(n % 2 == 0)][n % 4])
    assert call(ctypes.cast(entry, c_void_p).value, *given) == -7
    assert got == want


@pytest.mark.parametrize("call", CALLS)
@pytest.mark.parametrize("wrong", [1.5, "1", [1]])
def test_what_is_no_argument_is_refused(call, wrong):
    entry = ctypes.CFUNCTYPE(c_int, c_int)(lambda a: 0)
    with pytest.raises(TypeError):
        call(ctypes.cast(entry, c_void_p).value, wrong)


def test_the_native_caller_is_the_one_that_runs():
    """Where it can be built: on Linux on one of the two processors, with a compiler and Python's headers."""
    import os
    import platform
    import shutil
    import sys
    import sysconfig
    if not (sys.platform.startswith("linux") and platform.machine() in ("x86_64", "aarch64") and (shutil.which("gcc") or shutil.which("cc"))
            and os.path.isfile(os.path.join(sysconfig.get_paths()["include"], "Python.h"))):
        pytest.skip("host_call.c cannot be built here")
    assert host_call(verbose=False) is not _through_ctypes


def test_as_many_arguments_as_there_are_places():
    call = host_call(verbose=False)
    if call is _through_ctypes:
        pytest.skip("the stand-in has no limit")
    got = []
    entry = ctypes.CFUNCTYPE(c_int, *[c_longlong] * 64, *[c_float] * 8)(lambda *a: (got.extend(a), 3)[1])
    at = ctypes.cast(entry, c_void_p).value
    ints, floats = [n * n - (1 << 40) for n in range(64)], [c_float(n + 0.3) for n in range(8)]
    assert call(at, *ints, *floats) == 3
    assert got == ints + [f.value for f in floats]
    for more in (ints + [0] + floats, ints + floats + [c_float(0.0)]):
        with pytest.raises(TypeError):
            call(at, *more)
    assert len(got) == 72                                     # (nothing was called with too many)
