"""Tiles in a cache file that another generation of the FFT kernels wrote are not taken over: the passes are
timed again and the file gets lines of this generation."""
import pytest

from creep_modeling_b200 import decks
from creep_modeling_b200.solver import Solve, tune_cache

pytestmark = pytest.mark.gpu


def test_lines_without_this_generation_are_timed_again(tmp_path):
    case = decks.case_c1(nsteps=1)
    case.n, case.ngrains = (12, 18, 20), 8  # a grid no other test uses, so this process has not tuned it
    fft = decks.write_case(case, tmp_path / "deck")
    cache = tmp_path / "tiles.save"
    old = [f"evp-tile {p} 1 0 12 18 20 1" for p in range(3)]
    cache.write_text("\n".join(old) + "\n")
    tune_cache(cache)
    try:
        Solve(fft, mix=1, modal=0).close()
        lines = cache.read_text().splitlines()
        assert lines[:3] == old and {int(l.split()[1]) for l in lines[3:]} == {0, 1, 2}
        tune_cache(cache)  # read back: now known
        Solve(fft, mix=1, modal=0).close()
        assert cache.read_text().splitlines() == lines
    finally:
        tune_cache(None)
