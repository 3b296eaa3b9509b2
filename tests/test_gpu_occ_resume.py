"""The occupancy raycast's rays along the edge of what has been seen (set aside by the first launch, taken
up by the second), against the oracle: a depth image with large holes seen again from the side, so that
rays run along the holes' edges; the smallest images, the largest map,
no scale output. Bars as in the occupancy raycast's other tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,dim,res,angle,scale", [
    (53, 39, 5.12, 0.02, 0.5, True), (53, 39, 5.12, 0.04, -0.7, False), (33, 26, 81.92, 0.01, 0.4, True),
    (2, 1, 5.12, 0.02, 0.5, True)])
def test_rays_along_the_edge(oracle, gpu, width, height, dim, res, angle, scale):
    import torch
    spec = dict(width=64, height=48, fx=50.0, fy=50.0, cx=31.5, cy=23.5, near_plane=0.1, far_plane=6.0)
    y, x = np.mgrid[0:48, 0:64]
    depth = (1.6 + 0.3 * np.cos(0.2 * x) * np.cos(0.15 * y)).astype(np.float32)
    depth[(x // 9 + y // 7) % 2 == 0] = 0.0
    T = np.eye(4, dtype=np.float32)
    om = oracle.OracleOccMap(dim, res)
    gm = gpu.Map(dim, res, res_type="multi", field="occupancy", max_blocks=1 << 16)
    integ = gpu.MapIntegrator(gm)
    for k in range(3):
        T[0, 3] = 0.003 * k
        om.integrate_depth(depth, oracle.pinhole(**spec), T, k)
        integ.integrateDepth(k, torch.from_numpy(depth).cuda(), gpu.PinholeCamera(**spec), T)
    gm.check()
    view = dict(spec, width=width, height=height, cx=(width - 1) / 2, cy=(height - 1) / 2)
    c, s = np.cos(angle), np.sin(angle)
    V = np.array([[c, 0, s, -0.8 * s], [0, 1, 0, 0.1], [-s, 0, c, 0.3], [0, 0, 0, 1]], np.float32)
    op, on, osc = om.raycast(oracle.pinhole(**view), V)
    pts = torch.full((height, width, 3), 7.0, device="cuda")
    nrm = torch.full_like(pts, 7.0)
    sc = torch.full((height, width), 7, dtype=torch.int8, device="cuda") if scale else None
    gpu.raycast_volume(gm, gpu.PinholeCamera(**view), V, pts, nrm, sc)
    gp, gn = pts.cpu().numpy(), nrm.cpu().numpy()
    same = (op == gp).all(-1) & (on == gn).all(-1)
    if scale:
        same &= osc == sc.cpu().numpy()
    assert same.mean() >= 0.999
