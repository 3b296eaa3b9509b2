"""Multi-resolution maps stored in 16-bit words: raycast and field queries against the oracle's FP32 map, with the
surface at each scale. A stored value is rounded to 18 bits of significand, three updates are off by 3 x 2^-19
of the truncation (16 cm) at most: under 1e-6 m along a ray, 1e-5 in a value, and 1e-5 / 0.02 m in a gradient
of 6.25 per metre; the bars leave a factor of ten and, where a rounding may decide, 2 % of the pixels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f,scale", [(200.0, 0), (45.0, 1), (22.0, 2)])
def test_f16_scales(oracle, gpu, f, scale):
    import torch
    w, h, dim, res = 61, 45, 5.12, 0.02
    spec = dict(width=w, height=h, fx=f, fy=f, cx=(w - 1) / 2, cy=(h - 1) / 2, near_plane=0.1, far_plane=6.0)
    y, x = np.mgrid[0:h, 0:w]
    depth = (1.6 + 0.1 * np.cos(0.2 * x) * np.cos(0.15 * y)).astype(np.float32)
    depth[(x + 3 * y) % 17 == 0] = 0.0
    T = np.eye(4, dtype=np.float32)
    om = oracle.OracleMap(dim, res, multires=True)
    gm = gpu.Map(dim, res, max_blocks=1 << 15, res_type="multi", storage="f16")
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
    has = both & (on != 0).any(-1) & (gn != 0).any(-1)
    assert both.sum() > 100 and has.sum() > 50 and scale in osc[both]
    assert (ohit == ghit).mean() >= 0.98
    assert (np.abs(gp - op)[both].max(-1) <= 1e-5).mean() >= 0.98
    assert (gs == osc)[both].mean() >= 0.98
    assert ((on != 0).any(-1) == (gn != 0).any(-1))[both].mean() >= 0.98
    assert (np.sum(gn * on, -1)[has] > 1 - 1e-4).mean() >= 0.98

    rng = np.random.default_rng(3)
    hits = op[ohit]
    q = (hits[rng.choice(len(hits), 600)] + rng.normal(0, 0.04, (600, 3))).astype(np.float32)
    q[:200] = np.round(q[:200] / (8 * res)) * (8 * res)  # block corners
    gv, gvalid = gm.getFieldInterp(torch.from_numpy(q).cuda())
    gg, ggvalid = gm.getFieldGrad(torch.from_numpy(q).cuda())
    gv, gvalid, gg, ggvalid = (a.cpu().numpy() for a in (gv, gvalid, gg, ggvalid))
    values = gradients = 0
    for i, p in enumerate(q):
        v, g = om.field_interp(p), om.field_grad(p)
        assert (v is not None) == gvalid[i] and (g is not None) == ggvalid[i]
        if v is not None:
            assert abs(v - gv[i]) <= 1e-4
            values += 1
        if g is not None:
            assert np.abs(g - gg[i]).max() <= 5e-3
            gradients += 1
    assert values > 50 and gradients > 50
