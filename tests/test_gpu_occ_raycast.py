"""The occupancy raycast at the edges of its launch and of the octree, against the oracle: images that
are not multiples of the 8 x 4 warp tile, the smallest octree (two levels) and a deep one, a camera
outside the map, rays that end in unknown space. The GPU follows the oracle's float operations, so the
images are compared bit for bit where both hit, with the parity tests' share of pixels (99.9 %) for
the rest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,dim,res,back", [
    (1, 1, 10.24, 0.04, 0.0), (31, 9, 10.24, 0.04, 0.0), (65, 33, 10.24, 0.02, 0.0), (48, 36, 40.96, 0.01, 0.0),
    (40, 30, 0.64, 0.04, 0.0), (40, 30, 10.24, 0.04, 5.0)])
def test_occ_raycast_edges(oracle, gpu, width, height, dim, res, back):
    import torch
    f = 50.0
    spec = dict(width=64, height=48, fx=f, fy=f, cx=31.5, cy=23.5, near_plane=0.1, far_plane=8.0)
    y, x = np.mgrid[0:48, 0:64]
    depth = (0.4 * dim * (0.8 + 0.2 * np.cos(0.2 * x) * np.cos(0.15 * y))).clip(0.15, 3.0).astype(np.float32)
    depth[(x + 3 * y) % 17 == 0] = 0.0
    depth[20:28, 30:36] = 0.0
    T = np.eye(4, dtype=np.float32)
    om = oracle.OracleOccMap(dim, res)
    gm = gpu.Map(dim, res, res_type="multi", field="occupancy", max_blocks=1 << 15)
    integ = gpu.MapIntegrator(gm)
    for k in range(3):
        T[0, 3] = 0.003 * k
        om.integrate_depth(depth, oracle.pinhole(**spec), T, k)
        integ.integrateDepth(k, torch.from_numpy(depth).cuda(), gpu.PinholeCamera(**spec), T)
    gm.check()
    view = dict(spec, width=width, height=height, cx=(width - 1) / 2 + 0.3, cy=(height - 1) / 2 - 0.2)
    V = T.copy()
    V[2, 3] = -back - (0.4 * dim if back else 0.0)
    view["far_plane"] = 8.0 + back + dim
    op, on, osc = om.raycast(oracle.pinhole(**view), V)
    pts = torch.full((height, width, 3), 7.0, device="cuda")
    nrm = torch.full_like(pts, 7.0)
    sc = torch.full((height, width), 7, dtype=torch.int8, device="cuda")
    gpu.raycast_volume(gm, gpu.PinholeCamera(**view), V, pts, nrm, sc)
    gp, gn, gs = pts.cpu().numpy(), nrm.cpu().numpy(), sc.cpu().numpy()
    same = (op == gp).all(-1) & (on == gn).all(-1) & (osc == gs)
    assert same.mean() >= 0.999
