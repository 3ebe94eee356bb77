"""The one-CTA float-float solver of small reduced systems (k_small_dense) at
the edges of its panels, tiles and thread counts: one pose block, a few, the
largest with 256 threads (19 blocks), the smallest with 512, the widest tiles
and the largest system it takes (39 blocks, 234 rows).

Every pose is free and two priors hold the gauge, so the step's pose part is
the solver's x itself (no gauge projection).  LDL^T is backward stable:
|S x - b| <= c n eps (|S| |x| + |b|) in norms; with float-float eps = 2^-46
(products and sums each within a few 2^-48), n <= 234 and c = 4 that is
1.4e-11."""
import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu

BOUND = 4 * 234 * 2.0 ** -46


@pytest.mark.parametrize("cams", [2, 3, 6, 11, 19, 20, 27, 28, 39])
def test_backward_error(pkg, cams):
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=cams, n_pt=150 + cams, seed=pkg.synth.BASE_SEED + cams)
    prob.pose_const = np.zeros(cams, np.uint8)
    with pkg.native.Problem(prob, device=0) as p:
        p.set_pose_priors([0, 1], prob.poses_true[:2], np.array([1e4 * np.eye(6)] * 2))
        lay = p.layout()
        assert lay.solver == pkg.native.SOLVER_DENSE_SMALL and lay.n_free_poses == cams
        p.init(fixed_iter_params(pkg, 1, prob.initial_lm_damping))
        p.step()
        S, b, delta = p.last_system()
    S = np.tril(S) + np.tril(S, -1).T
    x = delta[:6 * cams]
    err = np.linalg.norm(S @ x - b) / (np.linalg.norm(S, 2) * np.linalg.norm(x) + np.linalg.norm(b))
    assert np.all(np.isfinite(x)) and err < BOUND, err
