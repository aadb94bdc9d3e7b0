"""The peel on both sides of the line where the scan and the update of a (block,
group) pair run together: the grouped update equals the ungrouped one, with few
pairs from the first iteration on, with many at first and few at last, and with
more blocks of 32 columns than warps."""
import pytest

from tests.test_gpu_peel_units import test_grouped_update_equals_ungrouped as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,NT,nt,P,scale", [(2, 300, 61, 6, False), (24, 4000, 61, 6, False),
                                             (96, 45000, 61, 6, False), (33, 90000, 41, 4, True)])
def test_few_and_many_pairs(K, NT, nt, P, scale):
    check(K, NT, nt, P, scale)
