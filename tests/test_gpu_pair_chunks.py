"""The FP32 pair sums of S do not depend on how many pairs the other blocks have:
an EUCM camera with fixed params on more poses than the one-CTA solver takes,
two groups of poses that share no point, the second with few or with many
points.  The first group's blocks of S and rows of the rhs keep their bits."""
import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu

EUCM = np.array([300.0, 300.0, 320.0, 240.0, 0.5, 1.0])


def _scene(pkg, first, second):
    """`first` points seen by 25 of the poses 1 .. 45, then `second` points seen by the poses 46 .. 61."""
    rng = np.random.default_rng(7)
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=62, n_pt=first + 4200, seed=pkg.synth.BASE_SEED + 33)
    sees = np.stack([rng.permutation(45)[:25] + 1 for _ in range(first)])
    cam = np.concatenate([sees.ravel(), np.tile(np.arange(46, 62), second)]).astype(np.int32)
    pt = np.concatenate([np.repeat(np.arange(first), 25), np.repeat(np.arange(first, first + second), 16)])
    q, v = -prob.poses_true[cam, 1:4], prob.points_true[pt] - prob.poses_true[cam, 4:]
    u = 2.0 * np.cross(q, v)
    prob.obs_uv = pkg.synth.eucm_project(EUCM, v + prob.poses_true[cam, :1] * u + np.cross(q, u))
    prob.obs_cam, prob.obs_pt = cam, pt.astype(np.int32)
    n = first + second
    prob.points, prob.points_true = prob.points[:n], prob.points_true[:n]
    prob.point_const = None
    prob.intrinsics, prob.camera_model, prob.eucm_alpha_beta = EUCM[:4].copy(), 1, EUCM[4:].copy()
    return prob


def test_fp32_partition(pkg):
    out = []
    for second in (20, 4200):
        prob = _scene(pkg, 400, second)
        with pkg.native.Problem(prob, device=0) as p:
            assert not p.layout().float_float_lin
            p.init(fixed_iter_params(pkg, 1, prob.initial_lm_damping))
            p.step()
            S, rhs, _ = p.last_system()
            out.append((S[:270, :270], rhs[:270]))
    assert np.isfinite(out[0][0]).all() and np.abs(out[0][0]).max() > 0
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
