"""Tracking with more than 220,000 inliers (clean frames, cameras larger than 640x480): the elimination of the
6x6 system stays in FP64's range. Poses against the oracle's on the same reference images, within the parity
bar or twice the oracle's own spread over start poses one float step away."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _angle(A, B):
    R = A[:3, :3].astype(np.float64).T @ B[:3, :3].astype(np.float64)
    s = 0.5 * np.linalg.norm([R[2, 1] - R[1, 2], R[0, 2] - R[2, 0], R[1, 0] - R[0, 1]])
    return float(np.arctan2(s, (np.trace(R) - 1) / 2))


def _distance(A, B):
    return float(np.linalg.norm(A[:3, 3].astype(np.float64) - B[:3, 3]))


@pytest.mark.parametrize("width,height,seed", [(640, 480, 5), (1280, 960, 6)])
def test_clean_frames(oracle, gpu, width, height, seed):
    import torch
    from supereight2_gb300 import synthetic as syn
    f = 525.0 * width / 640
    spec = syn.PinholeSpec(width, height, f, f, (width - 1) / 2, (height - 1) / 2, 0.4, 6.0)
    scene = syn.make_scene(seed)
    T0, T1 = [T.astype(np.float32) for T in syn.random_walk_trajectory(2, seed=seed + 1, sigma_m=0.005, sigma_deg=0.3)]
    d0, d1 = [syn.render_depth(scene, spec, T, 0, noise=False).astype(np.float32) for T in (T0, T1)]
    cam = gpu.PinholeCamera.from_spec(spec)
    m = gpu.Map(10.24, 0.01, max_blocks=1 << 18)
    gpu.MapIntegrator(m).integrateDepth(0, torch.from_numpy(d0).cuda(), cam, T0)
    pts = torch.zeros((height, width, 3), device="cuda")
    nrm = torch.zeros_like(pts)
    gpu.raycast_volume(m, cam, T0, pts, nrm)

    osn = oracle.pinhole(width, height, f, f, (width - 1) / 2, (height - 1) / 2, 0.4, 6.0)
    op, on = pts.cpu().numpy(), nrm.cpu().numpy()
    accepted, T_o, stats = oracle.track(osn, oracle.tracker_config(), d1, T0, op, on)
    assert accepted and stats.reduction[28] > 220000 and _distance(T_o, T1) < 0.01
    spread_t = spread_r = 0.0
    for a in range(3):
        start = T0.copy()
        start[a, 3] = np.nextafter(start[a, 3], np.float32(np.inf))
        _, T_q, _ = oracle.track(osn, oracle.tracker_config(), d1, start, op, on)
        spread_t, spread_r = max(spread_t, _distance(T_o, T_q)), max(spread_r, _angle(T_o, T_q))
    for persistent in (True, False):
        tracker = gpu.Tracker(m, cam)
        tracker.set_persistent(persistent)
        T = T0.copy()
        assert tracker.track(torch.from_numpy(d1).cuda(), T, pts, nrm)
        assert tracker.last_reduction()[0][28] > 220000
        assert _distance(T, T_o) <= max(1e-5, 2 * spread_t) and _angle(T, T_o) <= max(1e-5, 2 * spread_r)
