"""Trial poses (pose_update16) over the steps of a converging run, so that the
series for small rotations are taken (|w| below 1e-6, theta^2 below 1e-6) as well
as the closed forms: against numpy's f64 as in test_gpu_pose_update.  The tables
that the update leaves for the trial cost are those of k_pose_tables, bit for bit:
the accepted step's cost is that of a run that starts at its variables."""
import numpy as np
import pytest

from conftest import fixed_iter_params
from test_gpu_pose_update import _update

pytestmark = pytest.mark.gpu


def _scene(pkg, const):
    """A circle without pixel error, started near the truth."""
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=9, n_pt=200, seed=pkg.synth.BASE_SEED + 14)
    q, v = -prob.poses_true[prob.obs_cam, 1:4], prob.points_true[prob.obs_pt] - prob.poses_true[prob.obs_cam, 4:]
    u = 2.0 * np.cross(q, v)
    c = v + prob.poses_true[prob.obs_cam, :1] * u + np.cross(q, u)
    prob.obs_uv = c[:, :2] / c[:, 2:] * prob.intrinsics[:2] + prob.intrinsics[2:4]
    prob.pose_const = np.zeros(9, np.uint8)
    prob.pose_const[list(const)] = 1
    for j in const:
        prob.poses[j] = prob.poses_true[j]
    return prob


@pytest.mark.parametrize("const", [(0,), (0, 4)])
def test_converging_steps(pkg, const):
    prob = _scene(pkg, const)
    free = [j for j in range(9) if not prob.pose_const[j]]
    angles = []
    with pkg.native.Problem(prob, device=0) as p:
        p.init(fixed_iter_params(pkg, 12, prob.initial_lm_damping))
        for _ in range(12):
            before, _ = p.variables()
            p.step()
            delta = p.last_system()[2]
            after, _ = p.variables()
            if np.array_equal(before, after):
                continue  # rejected
            for k, j in enumerate(free):
                xi = delta[6 * k:6 * k + 6]
                angles.append(np.linalg.norm(xi[:3]))
                # below 1e-3 rad V = I + W / 2: W^2 / 6 is left out, and a = (1 - cos th) / th^2 carries 2^-53 / th^2 above
                th = max(angles[-1], 1e-3)
                bound = 64 * 2.0**-53 * (1 + np.abs(before[j, 4:]).max() + np.linalg.norm(xi[3:]) / th)
                if angles[-1] <= 1e-3:
                    bound += angles[-1] ** 2 / 6 * np.linalg.norm(xi[3:])
                assert np.abs(after[j] - _update(xi, before[j])).max() < bound
            for j in set(range(9)) - set(free):
                assert np.array_equal(before[j], after[j])
            merit = p.cost()
            with pkg.native.Problem(prob, device=0) as q:
                q.set_variables(*p.variables())
                q.init(fixed_iter_params(pkg, 1, prob.initial_lm_damping))
                assert q.cost() == merit
    angles = np.array(angles)
    assert (angles > 1e-3).any() and ((angles < 1e-3) & (angles > 1e-6)).any() and (angles < 1e-6).any(), np.sort(angles)
