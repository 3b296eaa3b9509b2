"""The ray batches' voxel update (ri_update_voxel, compiled here for the host) equals the division by the
voxel's weight, bit for bit, for integer weights and for those of a block that became coarser."""
from tests import host_build


def test_update_is_the_division(tmp_path):
    n, wrong = (int(v) for v in host_build.run("ray_voxel", tmp_path).split())
    assert n > 10000
    assert wrong == 0
