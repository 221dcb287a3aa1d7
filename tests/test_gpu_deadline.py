"""A served solve whose work is far beyond its wall-clock budget at any speed ends with -8."""
import pytest

from creep_modeling_b200 import decks
from creep_modeling_b200.serve import Server

pytestmark = pytest.mark.gpu


def test_overrun_ends_with_its_own_status(tmp_path):
    case = decks.case_c1(nsteps=30000)  # at 32^3 an increment takes two milliseconds: a minute of work
    case.n = 32
    fft = decks.write_case(case, tmp_path)
    with Server(0, 8) as srv:
        st = srv.wait(srv.submit(fft, tmp_path / "out", mix=1, modal=0, csv_only=True, deadline_s=0.5), timeout=600)
    assert st["status"] == -8 and "deadline" in st["error"], st
    assert 0 < st["macrosteps"] < 30000
    assert 0.5 <= st["run_s"] < 30.0
