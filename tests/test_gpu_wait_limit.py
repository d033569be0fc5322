"""The bounded waits of the kernels: one that nothing ends gives up by itself and
says so, and the calls that wait for their work report it as an error."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import so3_b200 as so3
from so3_b200 import build, synth
from tests.helpers import params

pytestmark = pytest.mark.gpu

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "wait_limit.cu")


def test_wait_gives_up(tmp_path):
    lib = str(tmp_path / "wait_limit.so")
    subprocess.run([build.NVCC] + build.ARCH + build.FLAGS + ["-shared", SRC, "-o", lib], check=True, timeout=300)
    flag, ok, ns = ctypes.c_int(), (ctypes.c_int * 2)(), ctypes.c_ulonglong()
    assert ctypes.CDLL(lib).run_wait(ctypes.byref(flag), ok, ctypes.byref(ns)) == 0
    assert (flag.value, ok[0], ok[1]) == (4, 1, 0)
    assert 1.9e9 < ns.value < 10e9  # the limit is 2 s of polling


@pytest.mark.parametrize("call", ["inverse", "forward", "adjoint_inverse", "adjoint_forward"])
def test_dropin_calls_report_a_wait_that_gave_up(lib, call):
    p = params(12, 3)
    x = synth.gen_flmn(p, 2)
    if call in ("forward", "adjoint_inverse"):
        x = so3.inverse(x, p)
    good = getattr(so3, call)(x, p)
    word = lib.so3g_dropin_fault_word
    word.restype, word.argtypes = ctypes.POINTER(ctypes.c_int), [ctypes.c_int]
    word(0)[0] = 4  # as the contraction kernel sets it
    with pytest.raises(so3.SO3Error, match="status 2"):
        getattr(so3, call)(x, p)
    assert np.array_equal(getattr(so3, call)(x, p), good)  # reported once


def test_a_failed_call_leaves_no_report_to_the_next(lib):
    p, bad = params(12, 3), params(12, 3, sampling=1)
    f = so3.inverse(synth.gen_flmn(p, 2), p)
    good = so3.adjoint_inverse(f, p)
    word = lib.so3g_dropin_fault_word
    word.restype, word.argtypes = ctypes.POINTER(ctypes.c_int), [ctypes.c_int]
    word(0)[0] = 4
    with pytest.raises(so3.SO3Error, match="status 3"):  # adjoints are MW only
        so3.adjoint_inverse(np.zeros(so3.f_size(bad), np.complex128), bad)
    assert np.array_equal(so3.adjoint_inverse(f, p), good)
