"""The one-voxel-per-thread local solve at the sizes and phases where its batches of 32 can go
wrong, against the oracle, and its reciprocal against the correctly rounded one."""
import dataclasses
import shutil
import subprocess
from pathlib import Path

import pytest

from creep_modeling_b200 import decks
from tests import parity

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("n, slip, modal, gas, nrs", [
    ((6, 10, 2), "fcc", 0, False, 10.0),     # 120 voxels: a last batch of 24 lanes
    ((2, 4, 2), "fcc", 1, False, 10.0),      # fewer voxels than one warp
    ((22, 6, 1), "bcc24", 0, False, 12.6),   # 24 systems, non-integer exponent, four lanes left over
    ((10, 8, 6), "fcc", 0, True, 10.0),      # gas and solid voxels in one warp
    ((10, 8, 6), "fcc", 1, True, 10.0),      # and with the augmented Lagrangian's operator
    ((26, 16, 10), "bcc24", 1, False, 10.0),
    ((40, 32, 32), "fcc", 0, False, 20.0),   # 40,960 voxels: the full block size, a second batch for some warps
])
def test_newton_batches_match_oracle(tmp_path, n, slip, modal, gas, nrs):
    base = decks.case_c1(nsteps=2) if gas else decks.case_c2(nsteps=2)
    case = dataclasses.replace(base, n=n, ngrains=9)
    case.material = dataclasses.replace(case.material, slip=slip, nrs=nrs, tau0f=110.0, tau0b=95.0)
    if gas:
        case.phase2_frac, case.phase2_gas, case.complgas = 0.1, True, 1.0
    fft = decks.write_case(case, tmp_path)
    g, o, rg, ro, dg, do = parity.run_both(fft, 2, mix=1, modal=modal)
    parity.assert_rows_match(rg, ro, dg, do)
    for f in ("sg", "edotp", "gamdot", "trialtau", "velgrad"):
        assert parity.field_rel_err(g, o, f) <= parity.RTOL, f
    g.close()
    o.close()


def test_reciprocal_is_within_one_ulp(tmp_path):
    """Two Newton steps from 20 bits leave the rounding of the last one: below one unit in the last place (2^-52)."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no CUDA compiler")
    exe = tmp_path / "rcp_check"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2",
                    f"-I{ROOT / 'creep_modeling_b200' / 'csrc'}", "-o", str(exe), str(ROOT / "tests" / "rcp_check.cu")], check=True)
    assert float(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout) < 2.0 ** -52
