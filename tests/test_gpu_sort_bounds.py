"""A sort pass whose digit counts are of other keys (what a grid barrier that gave up can
leave to the pair-key sort) stores nothing past its result."""
import pytest

from mechanic_b200.physics import InvalidArgument, selftest_sort_bounds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2048, 5000, 65_537, 100_001])
def test_pass_with_other_counts_stays_inside(cuda_lib, n):
    assert selftest_sort_bounds(n) == 0


def test_argument_range(cuda_lib):
    for n in (0, (1 << 20) + 1):
        with pytest.raises(InvalidArgument):
            selftest_sort_bounds(n)
