"""Occupancy raycasts whose views are known to hold hits, normals and rays that are put aside after two
points in a row without an interpolation (the oracle counts them): a wall with holes seen from the front, from
outside the map (back) and from the side (angle), image sizes that are no multiples of a warp's tile, a deep
octree and a small one, maps at the world's origin and 200 km from it. Against the oracle, over the pixels that
either side hits and over the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPEC = dict(width=64, height=48, fx=50.0, fy=50.0, cx=31.5, cy=23.5, near_plane=0.1, far_plane=8.0)


def _scene(oracle, dim, res, origin, front):
    """Three frames of a wavy wall with holes, and the oracle's map of them."""
    y, x = np.mgrid[0:48, 0:64]
    if front:
        depth = (0.4 * dim * (0.8 + 0.2 * np.cos(0.2 * x) * np.cos(0.15 * y))).clip(0.15, 3.0).astype(np.float32)
        depth[(x + 3 * y) % 17 == 0] = 0.0
        depth[20:28, 30:36] = 0.0
    else:
        depth = (1.6 + 0.3 * np.cos(0.2 * x) * np.cos(0.15 * y)).astype(np.float32)
        depth[(x // 9 + y // 7) % 2 == 0] = 0.0
    T_MW = np.eye(4, dtype=np.float32)
    T_MW[:3, 3] = dim / 2 - np.float32(origin)
    om = oracle.OracleOccMap(dim, res, T_MW=T_MW)
    poses = []
    for k in range(3):
        T = np.eye(4, dtype=np.float32)
        T[:3, 3] = origin
        T[0, 3] += np.float32(0.003 * k)
        om.integrate_depth(depth, oracle.pinhole(**SPEC), T, k)
        poses.append(T)
    return depth, T_MW, om, poses


def _view(width, height, dim, origin, angle, back):
    view = dict(SPEC, width=width, height=height, cx=(width - 1) / 2, cy=(height - 1) / 2)
    V = np.eye(4, dtype=np.float32)
    if angle:
        c, s = np.cos(angle), np.sin(angle)
        V = np.array([[c, 0, s, -0.8 * s], [0, 1, 0, 0.1], [-s, 0, c, 0.3], [0, 0, 0, 1]], np.float32)
    elif back:
        V[2, 3] = -back - 0.4 * dim
        view.update(fx=200.0, fy=200.0, far_plane=8.0 + back + dim)
    V[:3, 3] += np.float32(origin)
    return view, V


@pytest.mark.parametrize("width,height,dim,res,angle,back,origin", [
    (65, 33, 10.24, 0.02, 0.0, 0.0, 0.0), (31, 9, 10.24, 0.04, 0.0, 0.0, 0.0),
    (48, 36, 40.96, 0.04, 0.0, 0.0, 0.0), (40, 30, 0.64, 0.04, 0.0, 0.0, 0.0),
    (320, 240, 10.24, 0.04, 0.0, 5.0, 0.0), (53, 39, 5.12, 0.02, 0.5, 0.0, 0.0),
    (53, 39, 5.12, 0.04, -0.7, 0.0, 0.0), (33, 26, 81.92, 0.01, 0.4, 0.0, 0.0)])
def test_views_with_hits(oracle, gpu, width, height, dim, res, angle, back, origin):
    import torch
    depth, T_MW, om, poses = _scene(oracle, dim, res, origin, not angle)
    gm = gpu.Map(dim, res, res_type="multi", field="occupancy", T_MW=T_MW, max_blocks=1 << 16)
    integ = gpu.MapIntegrator(gm)
    for k, T in enumerate(poses):
        integ.integrateDepth(k, torch.from_numpy(depth).cuda(), gpu.PinholeCamera(**SPEC), T)
    gm.check()
    view, V = _view(width, height, dim, origin, angle, back)
    misses = np.zeros((height, width), np.int32)
    op, on, osc = om.raycast(oracle.pinhole(**view), V, misses)
    pts = torch.full((height, width, 3), 7.0, device="cuda")
    nrm = torch.full_like(pts, 7.0)
    sc = torch.full((height, width), 7, dtype=torch.int8, device="cuda")
    gpu.raycast_volume(gm, gpu.PinholeCamera(**view), V, pts, nrm, sc)
    gp, gn, gs = pts.cpu().numpy(), nrm.cpu().numpy(), sc.cpu().numpy()
    hit = (op != 0).any(-1) | (gp != 0).any(-1)
    assert (op != 0).any(-1).sum() >= 100 and (on != 0).any(-1).sum() >= 30
    assert (misses > 2).sum() >= 20
    same = (op == gp).all(-1) & (on == gn).all(-1) & (osc == gs)
    assert same[hit].mean() >= 0.999 and same[~hit].mean() >= 0.999
