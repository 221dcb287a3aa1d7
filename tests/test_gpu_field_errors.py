"""Reading a field leaves no error message behind, and a refused read writes neither the buffer nor *written."""
import ctypes

import numpy as np
import pytest

from creep_modeling_b200 import Solve, _lib, decks

pytestmark = pytest.mark.gpu


def test_field_reads_and_their_errors(tmp_path):
    case = decks.case_c1(nsteps=1)
    case.n, case.ngrains = 8, 4
    lib = _lib.load()
    with Solve(decks.write_case(case, tmp_path), mix=1, modal=0) as s:
        assert lib.evp_set_deadline(None, 0.0) == -7  # leaves the message of another call
        before = lib.evp_last_error()
        assert b"null handle" in before
        assert s.field("sg").size == 9 * 8 ** 3 and s.field("macro").size == 279
        assert lib.evp_last_error() == before
        buf, n = np.full(4, 7.0), ctypes.c_longlong(-5)
        rc = lib.evp_get_field(s._h, b"sg", buf.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), 4, ctypes.byref(n))
        assert rc == -7 and b"too small" in lib.evp_last_error()
        assert n.value == -5 and np.all(buf == 7.0)
        with pytest.raises(_lib.EvpError, match="unknown field"):
            s.field("no such field")
