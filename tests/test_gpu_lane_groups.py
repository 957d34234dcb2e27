"""Patterns of 9 to 16 samples go in lane groups, two or three beams a warp: the same bytes as with one lane
per beam, around the largest pattern that does."""
import pytest

from tests import test_gpu_packing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vertices", [9, 10, 14, 15])
@pytest.mark.parametrize("beams", [1, 33, 4865, 20011])
def test_lane_groups_write_the_same(rgl, vertices, beams):
    test_gpu_packing.test_every_packing_writes_the_same(rgl, 1, vertices, beams)
