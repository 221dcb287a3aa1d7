"""Device memory that evp_green_apply leaves with the library: nothing from a call with a large spectrum, a bounded
amount from smaller ones, and nothing after evp_release_memory."""
import ctypes

import numpy as np
import pytest

from creep_modeling_b200 import _lib
from tests import green_cases

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _call(shape, c0, s0):
    import torch

    dp = ctypes.POINTER(ctypes.c_double)
    tau = torch.zeros(9, int(np.prod(shape)), dtype=torch.float64, device="cuda")
    tau[2, 0] = 1.0
    out = torch.empty_like(tau)
    _lib.check(_lib.load().evp_green_apply(ctypes.c_void_p(tau.data_ptr()), ctypes.c_void_p(out.data_ptr()), *shape,
                                           c0.ctypes.data_as(dp), s0.ctypes.data_as(dp), None))
    del tau, out
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_scratch_is_bounded_and_given_back(oracle_lib):
    c0, s0 = (np.ascontiguousarray(a.reshape(-1)) for a in green_cases.medium(oracle_lib))
    lib = _lib.load()
    _call((8, 8, 8), c0, s0)  # module loading
    assert lib.evp_release_memory() == 0
    free = _call((8, 8, 8), c0, s0)
    large = _call((200, 160, 128), c0, s0)  # a spectrum of 298 MB
    assert large >= free - 2 * MB
    kept = _call((120, 90, 80), c0, s0)  # 63 MB
    assert kept >= free - 256 * MB
    assert lib.evp_release_memory() == 0
    import torch

    assert torch.cuda.mem_get_info()[0] >= free - 2 * MB
