"""A warp's propagation of four octree nodes (occ_propagate_set, compiled here for the host) with its lanes as
far apart as they may drift: the nodes' data, the pruning and the next propagation set equal the serial
result's."""
from tests import host_build


def test_lanes_may_drift(tmp_path):
    nodes, pruned, differ = (int(v) for v in host_build.run("occ_propagate", tmp_path).split())
    assert nodes == 160 and pruned >= 20
    assert differ == 0
