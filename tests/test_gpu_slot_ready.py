"""Slots of three hops and more whose middle hops have many edges and whose last hop adds few: the columns of a middle hop are translated
next to the CSC of the last one, and cross PCIe with the arrays that are there before the last list is merged."""
import pytest

from test_gpu_slot_copies import M, check, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fanouts", [[20, 20, 1], [20, 10, 1, 1], [4, 40, 1]])
@pytest.mark.parametrize("policy", ["recent", "uniform"])
def test_columns_of_the_middle_hops(fanouts, policy):
    data, b = make(2)
    for n in (3, 500, 4000):
        for _ in range(3):
            check(data, b, M // 2, M // 2 + n, fanouts, policy)
