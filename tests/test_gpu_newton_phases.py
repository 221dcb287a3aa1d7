"""The local solve where its column is only partly used, and where its Newton steps are halved, against the oracle:
phases with different numbers of systems side by side (or with none), modes with different exponents, and a rate
that jumps by five orders of magnitude, so that the first corrections overshoot by far."""
import dataclasses
import re
from pathlib import Path

import pytest

from creep_modeling_b200 import decks
from tests import parity

pytestmark = pytest.mark.gpu

NO_SYSTEMS = ("NO SLIP\nCUBIC\n1. 1. 1.\n1\n0\n{111}<110>\n1 12 10.0 1e-3 0.0 0\n100. 100. 40. 500. 20. 0\n1.0 1.4\n"
              + "\n".join("%d %d %d %d %d %d" % r for r in decks.FCC_SLIP) + "\n")


def _check(fft, nmacro, modal=0):
    g, o, rg, ro, dg, do = parity.run_both(fft, nmacro, mix=1, modal=modal)
    parity.assert_rows_match(rg, ro, dg, do)
    for f in ("sg", "edotp", "gamdot", "trialtau", "velgrad"):
        assert parity.field_rel_err(g, o, f) <= parity.RTOL, f
    g.close()
    o.close()


@pytest.mark.parametrize("slip, nrs, second, modal", [
    ("fcc", 10.0, decks.Material(slip="bcc24", nrs=12.0, tau0f=140.0, tau0b=130.0), 0),
    ("fcc", 10.0, decks.Material(slip="bcc24", nrs=12.0, tau0f=140.0, tau0b=130.0), 1),
    ("bcc24", 12.6, decks.Material(nrs=10.0, tau0f=140.0), 0),
    ("fcc", 10.0, None, 0),
])
def test_phases_of_different_systems(tmp_path, slip, nrs, second, modal):
    case = dataclasses.replace(decks.case_c2(nsteps=2), n=(12, 10, 8), ngrains=9, phase2_frac=0.2)
    case.material = dataclasses.replace(case.material, slip=slip, nrs=nrs)
    fft = decks.write_case(case, tmp_path)
    if second is None:
        (tmp_path / "cupl2_2.sx").write_text(NO_SYSTEMS)
    else:
        decks.write_cupl2(tmp_path / "cupl2_2.sx", second)
    _check(fft, 2, modal)


@pytest.mark.parametrize("exponents", [("10.0", "20.0"), ("10.0", "12.6")])
def test_modes_of_different_exponents(tmp_path, exponents):
    case = dataclasses.replace(decks.case_c2(nsteps=2), n=(12, 10, 8), ngrains=9)
    case.material = dataclasses.replace(case.material, slip="bcc24")
    fft = decks.write_case(case, tmp_path)
    slip = Path(tmp_path / "cupl2.sx")
    for mode, nrs in enumerate(exponents, start=1):
        slip.write_text(re.sub(rf"(?m)^{mode}   12   \S+", f"{mode}   12   {nrs}", slip.read_text()))
    _check(fft, 2)


@pytest.mark.parametrize("nrs", [20.0, 12.6])
def test_halved_steps(tmp_path, nrs):
    case = dataclasses.replace(decks.case_c2(), n=(6, 4, 4), ngrains=5)
    case.material = dataclasses.replace(case.material, nrs=nrs, tau0f=1.0, tau0b=1.0, tau1=0.5, thet0=5.0, thet1=0.2)
    case.processes = [decks.Loading(kind="tension", udot33=1e-6, tdot=1.0, nsteps=1),
                      decks.Loading(kind="tension", udot33=1e-1, tdot=0.5, nsteps=2)]
    _check(decks.write_case(case, tmp_path), 3)
