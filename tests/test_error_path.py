"""A call that fails after it has queued work: the C ABI waits for the handle's streams before it
returns, so that the next call may write the pinned staging buffers.  The headers are built for
the host over a fake of the CUDA runtime (tests/native/error_path_host.cpp)."""
import ctypes as C
import importlib
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
fmm = importlib.import_module("exafmm-dev_b200")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("err") / "liberr.so"
    # (the fake's own functions, also where another library brings a CUDA runtime)
    subprocess.check_call(["/usr/bin/g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-w",
                           "-Wl,-Bsymbolic", "-I", "/usr/local/cuda/include",
                           "-I", os.path.join(ROOT, "exafmm-dev_b200", "csrc"),
                           os.path.join(ROOT, "tests", "native", "error_path_host.cpp"),
                           "-o", str(out)])
    return C.CDLL(str(out))


@pytest.mark.parametrize("sides", [0, 1])
@pytest.mark.parametrize("how,code", [(0, "FMM_OK"), (1, "FMM_ERR_NOT_SUPPORTED"),
                                      (2, "FMM_ERR_INVALID"), (3, "FMM_ERR_NO_MEMORY"),
                                      (4, "FMM_ERR_NOT_SUPPORTED")])
def test_failed_call_waits(how, code, sides, lib):
    n = (C.c_int * 3)()
    assert lib.failed_call(how, sides, n) == getattr(fmm, code)
    assert list(n) == ([0, 0, 0] if how == 0 else [1, sides, sides])
