"""Ray batches at the edges of the ray kernel's chunks (16 rays to a CTA, 152 CTAs in flight): one ray,
a chunk less one, a chunk, one more, several, and more rays than are in flight at once, from one place
(every hand-over in the scanner's block) and from poses far apart (none). Against the oracle's serial
integration, bit for bit, over two batches so that blocks are found as well as allocated."""
import numpy as np
import pytest

from tests.test_gpu_ray_integrator import _batch, _compare, _maps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spread", [(1, 0.0), (15, 0.0), (16, 0.0), (17, 0.0), (50, 4.0), (2600, 0.0), (2600, 4.0)])
def test_ray_chunks(oracle, gpu, n, spread):
    leica = dict(width=360, height=180, near_plane=0.2, far_plane=12.0, elevation_resolution_deg=0.5,
                 azimuth_resolution_deg=0.5)
    om, gm = _maps(oracle, gpu, 25.6, 0.1)
    rng = np.random.default_rng(n)
    for k in range(2):
        d = rng.normal(size=(n, 3))
        rays = (d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0.1, 14.0, (n, 1))).astype(np.float32)
        poses = np.tile(np.eye(4, dtype=np.float32), (n, 1, 1))
        poses[:, :3, 3] = (0.31, -0.17, 0.05) + spread * rng.uniform(-1, 1, (n, 3))
        o, g = _batch(oracle, gpu, om, gm, leica, poses, rays, k)
        assert o == g
        _compare(om, gm)
