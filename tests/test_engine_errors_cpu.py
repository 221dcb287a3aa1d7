"""A CUDA call that fails while the engine captures its iterations: the stream leaves capture mode, nothing is left
behind, and the next launch works (the runtime is a fake, no GPU)."""
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
    out = tmp_path_factory.mktemp("engine") / "libenginecheck.so"
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", f"-I{CSRC}", f"-isystem{cuda}", "-o",
                    str(out), str(HERE / "host_engine_check.cpp")], check=True)
    L = ctypes.CDLL(str(out))
    L.engine_case.argtypes = [ctypes.c_char_p, ctypes.c_int]
    return L


@pytest.mark.parametrize("call", ["throw", "cudaEventRecord", "cudaStreamWaitEvent", "cudaGetLastError", "cudaGraphInstantiate",
                                  "cudaStreamCreateWithPriority", "cudaEventCreateWithFlags", "cudaStreamGetPriority",
                                  "cudaStreamBeginCapture"])
def test_the_engine_survives_a_failed_call(lib, call):
    found = {n: lib.engine_case(call.encode(), n) for n in range(6)}
    assert found[0] == 0 and set(found.values()) <= {0, -1}, found
