"""The temporal search in planes of up to 4 candidate positions (a lane pair per block) and of a few
more (the rows kernel): lists equal the CPU oracle's."""
import pytest

from test_match_temporal_gpu import test_temporal_lists_equal_oracle as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["noise", "levels"])
@pytest.mark.parametrize("P", [2, 6])
@pytest.mark.parametrize("w,h", [(8, 8), (9, 9), (11, 8), (8, 11), (12, 8), (8, 12), (10, 9), (10, 10)])
def test_small_planes(w, h, P, kind):
    check(w, h, 8, 9, 2, 2, P, kind, 0)
