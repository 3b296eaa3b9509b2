"""Ray batches whose blocks become coarser and are updated again: a scanner backs off a wall, one timestamp
a batch. A block that went to a coarser scale holds weights that are no integers (ceil(sum) / count).
Against the oracle's serial integration after each batch, bit for bit."""
import numpy as np
import pytest

from supereight2_gb300.synthetic import wall_rays
from tests.test_gpu_ray_integrator import _batch, _compare, _maps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,res,distances", [(25.6, 0.05, (5.0, 9.0, 9.5, 16.0, 16.5)),
                                               (51.2, 0.1, (10.0, 17.0, 18.0, 32.0, 33.0))])
def test_scanner_backs_off_a_wall(oracle, gpu, dim, res, distances):
    leica = dict(width=360, height=180, near_plane=0.2, far_plane=40.0) # 1 degree
    om, gm = _maps(oracle, gpu, dim, res)
    scales, grew, fractional = {}, 0, 0
    first = np.array([0, 512, 576, 584])
    for k, distance in enumerate(distances):
        pose = np.eye(4, dtype=np.float32)
        pose[0, 3] = 0.4 * dim - distance
        o, g = _batch(oracle, gpu, om, gm, leica, pose, wall_rays(distance, -6.0, 0.5, 24), k)
        assert o == g
        _compare(om, gm)
        coords, sc, _, mean, _, _ = om.blocks()
        now = {tuple(c): int(s) for c, s in zip(coords, sc[:, 0])}
        coarser = [i for i, c in enumerate(coords) if 0 <= scales.get(tuple(c), 9) < sc[i, 0]]
        grew += len(coarser)
        for i in coarser:
            w = mean[i, first[sc[i, 0]]:first[sc[i, 0]] + (8 >> sc[i, 0]) ** 3, 1]
            fractional += int((w != np.floor(w)).sum())
        scales = now
    assert grew > 100 and fractional > 100
