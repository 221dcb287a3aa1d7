"""Every field of a solve on a grid of a few voxels, where one voxel's record is larger than the whole half
spectrum, against the oracle."""
import dataclasses

import numpy as np
import pytest

from creep_modeling_b200 import decks
from tests import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, slip", [((1, 1, 1), "fcc"), ((2, 1, 1), "fcc"), ((2, 2, 1), "bcc24"), ((4, 1, 1), "bcc24")])
def test_fields_of_tiny_grids_match_oracle(tmp_path, n, slip):
    case = dataclasses.replace(decks.case_c2(nsteps=1), n=n, ngrains=1)
    case.material = dataclasses.replace(case.material, slip=slip, nrs=10.0)
    g, o, *_ = parity.run_both(decks.write_case(case, tmp_path), 1)
    for f in ("sg", "sch", "crss", "c066mod", "sg66", "defgrad"):
        assert g.field(f).size == o.field(f).size, f
        assert parity.field_rel_err(g, o, f) <= parity.RTOL, f
    g.close()
    o.close()
