"""The samples that the occupancy raycast's search passes without a lookup (occ_box_steps, compiled here for
the host) lie in the octant they are passed for: next to the world's origin, in a map far from it, and for
a camera far behind its map."""
import pytest

from tests import host_build


@pytest.mark.parametrize("res,offset,back,rotated,some", [
    ("0.02", "0", "4", "0", True), ("0.4", "30", "60", "1", True), ("0.02", "3e3", "5", "1", True),
    ("0.02", "1e5", "5", "0", False), ("0.02", "1e6", "5", "0", False), ("0.02", "1e6", "5", "1", False),
    ("0.02", "0", "2e5", "0", False), ("0.02", "0", "2e4", "1", False), ("0.4", "1e7", "60", "0", False)])
def test_passed_samples_lie_in_the_octant(tmp_path, res, offset, back, rotated, some):
    rays, passed, outside = (int(v) for v in host_build.run("occ_march", tmp_path, res, offset, back, rotated).split())
    assert rays == 20000
    assert outside == 0
    assert not some or passed > 5 * rays
