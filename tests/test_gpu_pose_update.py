"""The trial poses exp(delta) T of sixteen lanes a pose (pose_update16) against
the same in numpy's f64, at the edges of its CTAs (16 poses).  Rounding: no value
passes through more than 64 operations of relative error 2^-53 on terms bounded
by 1 + |t|; constant poses are copied."""
import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu


def _hat(w):
    return np.array([[0.0, -w[2], w[1]], [w[2], 0.0, -w[0]], [-w[1], w[0], 0.0]])


def _update(xi, T):
    w, nu = xi[:3], xi[3:]
    th = np.linalg.norm(w)
    W = _hat(w)
    if th < 1e-4:  # series: the next terms are below 2^-53
        e = np.concatenate([[1 - th**2 / 8], w * (0.5 - th**2 / 48)])
        V = np.eye(3) + W * (0.5 - th**2 / 24) + W @ W * (1 / 6)
    else:
        e = np.concatenate([[np.cos(th / 2)], w * np.sin(th / 2) / th])
        V = np.eye(3) + W * (2 * np.sin(th / 2) ** 2 / th**2) + W @ W * ((th - np.sin(th)) / th**3)
    a, b, v = e[0], T[0], e[1:]
    q = np.concatenate([[a * b - v @ T[1:4]], T[1:4] * a + v * b + np.cross(v, T[1:4])])
    u = 2 * np.cross(v, T[4:])
    t = T[4:] + a * u + np.cross(v, u) + V @ nu
    return np.concatenate([q if q[0] >= 0 else -q, t])


@pytest.mark.parametrize("cams", [2, 15, 16, 17, 33, 47])
def test_trial_poses(pkg, cams):
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=cams, n_pt=200, seed=pkg.synth.BASE_SEED + cams)
    with pkg.native.Problem(prob, device=0) as p:
        p.init(fixed_iter_params(pkg, 1, prob.initial_lm_damping))
        before, _ = p.variables()
        p.step()
        delta = p.last_system()[2]
        after, _ = p.variables()
    free = [j for j in range(cams) if not prob.pose_const[j]]
    assert not np.array_equal(before, after)  # the step was accepted
    for j in range(cams):
        if j not in free:
            assert np.array_equal(before[j], after[j])
            continue
        k = free.index(j)
        xi = delta[6 * k:6 * k + 6]
        # th below 1e-3: a = (1 - cos th) / th^2 carries 2^-53 / th^2 of |w| |nu|
        th = max(np.linalg.norm(xi[:3]), 1e-3)
        bound = 64 * 2.0**-53 * (1 + np.abs(before[j, 4:]).max() + np.linalg.norm(xi[3:]) / th)
        assert np.abs(after[j] - _update(xi, before[j])).max() < bound
