"""The list kernels on every side of the warps-per-panel rule (one, two or four
warps by the tree's panels and a warp's splits: panels of 1, 4 and 9 points at
levels 3 to 6) and at every panel size whose loops are unrolled by rows (36 to
121 points), with the checks, inputs and tolerances of the list kernels' own
tests."""
import pytest

from test_gpu_list32 import test_mixed_list_sums as mixed_list_sums
from test_gpu_list64 import test_list_sums as list_sums

pytestmark = pytest.mark.gpu

CASES = [(3, 0, 0.7), (5, 0, 0.7), (4, 1, 0.7), (5, 1, 0.7), (6, 1, 0.8), (3, 2, 0.7), (5, 2, 0.7), (2, 5, 0.7), (2, 6, 0.7),
         (2, 7, 0.7), (2, 8, 0.7), (2, 9, 0.7), (2, 10, 0.7)]


@pytest.mark.parametrize("levels,degree,theta", CASES)
def test_float64(sb, levels, degree, theta):
    list_sums(sb, levels, degree, theta, 1e-4)


@pytest.mark.parametrize("levels,degree,theta", [c for c in CASES if c[1] <= 4])
def test_mixed(sb, levels, degree, theta):
    mixed_list_sums(sb, levels, degree, theta)
