"""The Green operator's C entries when something inside them fails: a status and a message, no exception
across the C boundary, no scratch left behind (the runtime is a fake, no GPU)."""
import ctypes
import os
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "creep_modeling_b200" / "csrc"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"
    if cxx is None or not (cuda / "cuda_runtime.h").exists():
        pytest.skip("no C++ compiler or CUDA headers")
    out = tmp_path_factory.mktemp("green") / "libgreencheck.so"
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", f"-I{CSRC}", f"-isystem{cuda}", "-o",
                    str(out), str(HERE / "host_green_check.cpp")], check=True)
    L = ctypes.CDLL(str(out))
    L.green_call.argtypes = [ctypes.c_int] * 5 + [ctypes.c_char_p, ctypes.POINTER(ctypes.c_int)]
    L.green_message.restype = ctypes.c_char_p
    return L


def _call(lib, noalloc, shape, launch, fail=""):
    left = ctypes.c_int(-1)
    rc = lib.green_call(noalloc, *shape, launch, fail.encode(), ctypes.byref(left))
    return rc, lib.green_message().decode(), left.value


@pytest.mark.parametrize("noalloc, shape", [(0, (256, 4, 4)), (1, (256, 4, 4)), (0, (256, 256, 256))])
def test_failures_inside_the_entries(lib, noalloc, shape):
    assert _call(lib, noalloc, shape, 0) == (0, "", 0)
    rc, msg, left = _call(lib, noalloc, shape, 1)  # a length whose pencils fit no block: not supported
    assert rc == -2 and "256" in msg and left == 0, (rc, msg, left)
    rc, msg, left = _call(lib, noalloc, shape, 2)  # a launch that failed
    assert rc == -6 and msg and left == 0, (rc, msg, left)
    for call in ("cudaMemcpyAsync", "cudaStreamSynchronize"):
        rc, msg, left = _call(lib, noalloc, shape, 0, call)
        assert rc == -6 and msg and left == 0, (call, rc, msg, left)
