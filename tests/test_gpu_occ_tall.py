"""Occupancy raycasts of tall images: more rows than one launch dimension of 4-row tiles counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("height", [262140, 262141, 300001])
def test_tall_image(oracle, gpu, height):
    import torch
    spec = dict(width=64, height=48, fx=50.0, fy=50.0, cx=31.5, cy=23.5, near_plane=0.1, far_plane=8.0)
    depth = np.full((48, 64), 1.5, np.float32)
    depth[10:20, 20:30] = 0.0
    om = oracle.OracleOccMap(5.12, 0.04)
    gm = gpu.Map(5.12, 0.04, res_type="multi", field="occupancy", max_blocks=1 << 14)
    T = np.eye(4, dtype=np.float32)
    integ = gpu.MapIntegrator(gm)
    for k in range(3):
        om.integrate_depth(depth, oracle.pinhole(**spec), T, k)
        integ.integrateDepth(k, torch.from_numpy(depth).cuda(), gpu.PinholeCamera(**spec), T)
    gm.check()
    view = dict(spec, width=2, height=height, fy=float(height), cx=0.5, cy=(height - 1) / 2)
    op, on, osc = om.raycast(oracle.pinhole(**view), T)
    pts = torch.full((height, 2, 3), 7.0, device="cuda")
    nrm = torch.full_like(pts, 7.0)
    sc = torch.full((height, 2), 7, dtype=torch.int8, device="cuda")
    gpu.raycast_volume(gm, gpu.PinholeCamera(**view), T, pts, nrm, sc)
    gp, gn, gs = pts.cpu().numpy(), nrm.cpu().numpy(), sc.cpu().numpy()
    assert (op != 0).any(-1).mean() > 0.3
    same = (op == gp).all(-1) & (on == gn).all(-1) & (osc == gs)
    assert same.mean() >= 0.999
