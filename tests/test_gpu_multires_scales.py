"""Multi-resolution raycasts and field queries with the surface at each integration scale, against the
oracle: the gradient takes its samples by block table at scales 0 and 1 and one by one from scale 2 on.
Points lie around the surface, on block boundaries and outside the map; the image is no multiple of the
warp tile. Bars as in the multi-resolution parity tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f,scales,storage,grads", [(200.0, {0}, "f32", True), (45.0, {1}, "f32", True),
                                                    (22.0, {2}, "f32", True), (8.0, {3}, "f32", False),
                                                    (40.0, {0, 1}, "f16", True)])
def test_scales(oracle, gpu, f, scales, storage, grads):
    import torch
    w, h, dim, res = 61, 45, 5.12, 0.02
    spec = dict(width=w, height=h, fx=f, fy=f, cx=(w - 1) / 2, cy=(h - 1) / 2, near_plane=0.1, far_plane=6.0)
    y, x = np.mgrid[0:h, 0:w]
    depth = (1.6 + 0.1 * np.cos(0.2 * x) * np.cos(0.15 * y)).astype(np.float32)
    depth[(x + 3 * y) % 17 == 0] = 0.0
    T = np.eye(4, dtype=np.float32)
    om = oracle.OracleMap(dim, res, multires=True)
    gm = gpu.Map(dim, res, max_blocks=1 << 15, res_type="multi", storage=storage)
    integ = gpu.MapIntegrator(gm)
    for k in range(3):
        T[0, 3] = 0.003 * k
        om.integrate_depth(depth, oracle.pinhole(**spec), T, k)
        integ.integrateDepth(k, torch.from_numpy(depth).cuda(), gpu.PinholeCamera(**spec), T)
    gm.check()

    view = dict(spec, width=37, height=19, cx=18.2, cy=9.1)
    op, on, osc = om.raycast(oracle.pinhole(**view), T)
    pts = torch.full((19, 37, 3), 7.0, device="cuda")
    nrm, sc = torch.full_like(pts, 7.0), torch.full((19, 37), 7, dtype=torch.int8, device="cuda")
    gpu.raycast_volume(gm, gpu.PinholeCamera(**view), T, pts, nrm, sc)
    gp, gn, gs = pts.cpu().numpy(), nrm.cpu().numpy(), sc.cpu().numpy()
    ohit, ghit = (op != 0).any(-1), (gp != 0).any(-1)
    both = ohit & ghit
    assert both.sum() > 100 and scales <= set(osc[both].tolist())
    if storage == "f16":  # the stored values are rounded: the image has to be whole
        assert (ohit == ghit).mean() >= 0.98
        return
    assert (ohit == ghit).mean() >= 0.999
    assert (np.abs(gp - op)[both].max(-1) <= 1e-4).mean() >= 0.999
    assert (gs[both] == osc[both]).mean() >= 0.999
    has = (on != 0).any(-1)
    assert (has == (gn != 0).any(-1))[both].mean() >= 0.999
    assert (has & both).any() == grads
    if grads:
        assert (np.sum(gn * on, -1)[has & both] > 1 - 1e-6).mean() >= 0.999

    rng = np.random.default_rng(3)
    hits = op[ohit]
    q = (hits[rng.choice(len(hits), 600)] + rng.normal(0, 0.04, (600, 3))).astype(np.float32)
    q[:200] = np.round(q[:200] / (8 * res)) * (8 * res)  # block corners
    q[200:300, 2] = np.round(q[200:300, 2] / (8 * res)) * (8 * res)
    q[300:310] = rng.uniform(-dim, dim, (10, 3))
    gv, gvalid = gm.getFieldInterp(torch.from_numpy(q).cuda())
    gg, ggvalid = gm.getFieldGrad(torch.from_numpy(q).cuda())
    gv, gvalid, gg, ggvalid = (a.cpu().numpy() for a in (gv, gvalid, gg, ggvalid))
    n = 0
    for i, p in enumerate(q):
        v, g = om.field_interp(p), om.field_grad(p)
        assert (v is not None) == bool(gvalid[i]) and (g is not None) == bool(ggvalid[i])
        if v is not None:
            assert abs(v - gv[i]) <= 1e-5
        if g is not None:
            assert np.allclose(g, gg[i], rtol=1e-4, atol=1e-3)
            n += 1
    assert (n > 50) == grads
