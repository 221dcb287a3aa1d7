"""The Green operator's transforms at the lengths where a stage's radix or place in the plan differs:
one stage, two, three, every odd radix first or last, and a plan of no stages (n3 = 1)."""
import numpy as np
import pytest

from tests import green_cases
from tests.test_gpu_green import _apply

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2, 2), (4, 8, 2), (26, 22, 14), (6, 10, 50), (16, 64, 8), (30, 18, 1), (12, 128, 16), (36, 98, 4)])
def test_every_radix_matches_oracle(oracle_lib, shape):
    c0, s0 = green_cases.medium(oracle_lib)
    tau = np.random.default_rng(5).standard_normal((9, int(np.prod(shape))))
    got = _apply(tau, shape, c0, s0)
    ref = oracle_lib.green_apply(tau, shape, c0, s0)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
