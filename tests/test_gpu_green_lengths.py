"""Axis lengths whose nine pencils do not fit one block are refused with a status by both Green-operator entries,
whichever pass finds out, and the next call works."""
import ctypes

import numpy as np
import pytest

from creep_modeling_b200 import _lib
from tests import green_cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(256, 4, 4), (4, 4, 256), (250, 2, 2), (2, 4, 250)])
def test_long_axes_are_refused(oracle_lib, shape):
    import torch

    L, dp = _lib.load(), ctypes.POINTER(ctypes.c_double)
    c0, s0 = (np.ascontiguousarray(a.reshape(-1)) for a in green_cases.medium(oracle_lib))
    for entry in (L.evp_green_apply, L.evp_green_apply_noalloc):
        for n, status in ((shape, -2), ((8, 8, 8), 0)):
            tau = torch.ones(9, int(np.prod(n)), dtype=torch.float64, device="cuda")
            out = torch.empty_like(tau)
            rc = entry(ctypes.c_void_p(tau.data_ptr()), ctypes.c_void_p(out.data_ptr()), *n, c0.ctypes.data_as(dp),
                       s0.ctypes.data_as(dp), None)
            assert rc == status, (n, rc, L.evp_last_error())
            if status:
                assert b"do not fit" in L.evp_last_error()
            torch.cuda.synchronize()
