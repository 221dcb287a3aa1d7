"""A single-crystal stiffness file whose 6x6 matrix is not symmetric (the reader takes all 36 numbers as
they stand, IO_functions.f90:640-720): every operator formed from it is then asymmetric and each step has
to use all of its entries, against the oracle."""
import dataclasses
from pathlib import Path

import numpy as np
import pytest

from creep_modeling_b200 import Solve, decks, solve_files
from tests import parity

pytestmark = pytest.mark.gpu

CUEL = ("0 \t\t\t\t\tISO\n"
        "250000.0 158000.0 146000.0 0.0 0.0 0.0\n"
        "150000.0 250000.0 153000.0 0.0 0.0 0.0\n"
        "144000.0 150000.0 250000.0 0.0 0.0 9000.0\n"
        "0.0 0.0 0.0 120000.0 5000.0 0.0\n"
        "0.0 0.0 0.0 0.0 120000.0 0.0\n"
        "0.0 0.0 0.0 0.0 0.0 120000.0\n")


@pytest.mark.parametrize("n, slip, modal, gas, nrs", [
    ((10, 8, 6), "fcc", 0, False, 10.0),
    ((10, 8, 6), "fcc", 1, False, 10.0),
    ((10, 8, 6), "fcc", 0, True, 12.6),
    ((6, 10, 2), "bcc24", 0, False, 10.0),
    ((40, 24, 24), "fcc", 0, False, 20.0),  # 23,040 voxels: a second batch for some warps
])
def test_asymmetric_stiffness_matches_oracle(tmp_path, n, slip, modal, gas, nrs):
    base = decks.case_c1(nsteps=3) if gas else decks.case_c2(nsteps=3)
    case = dataclasses.replace(base, n=n, ngrains=9)
    case.material = dataclasses.replace(case.material, slip=slip, nrs=nrs)
    if gas:
        case.phase2_frac, case.phase2_gas, case.complgas = 0.1, True, 1.0
    fft = decks.write_case(case, tmp_path)
    (tmp_path / "cuel.sx").write_text(CUEL)
    g, o, rg, ro, dg, do = parity.run_both(fft, 3, mix=1, modal=modal)
    parity.assert_rows_match(rg, ro, dg, do)
    for f in ("sg", "edotp", "sg66", "c066mod", "velgrad"):
        assert parity.field_rel_err(g, o, f) <= parity.RTOL, f
    g.close()
    o.close()


def test_in_a_batch_as_alone(tmp_path):
    """Beside symmetric members, whose launches it does not share."""
    ffts, alone, outs = [], [], []
    for i, n in enumerate((8, 16, 12)):
        case = decks.case_c1(nsteps=2)
        case.n, case.ngrains = n, 8
        ffts.append(decks.write_case(case, tmp_path / f"d{i}"))
        if i < 2:
            (tmp_path / f"d{i}" / "cuel.sx").write_text(CUEL)
        alone.append(tmp_path / f"alone{i}")
        outs.append(str(tmp_path / f"batch{i}") + "/")
        with Solve(ffts[i], out_dir=str(alone[i]) + "/", mix=1, modal=0, csv_only=True) as s:
            s.run()
    assert all(r.status == 0 for r in solve_files(ffts, outs, modal=0, csv_only=True))
    for a, b in zip(alone, outs):
        x, y = (np.delete(np.loadtxt(Path(d) / "results.csv", delimiter=",", skiprows=1, ndmin=2), 4, axis=1) for d in (a, b))
        np.testing.assert_array_equal(x, y)
