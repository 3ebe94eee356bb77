"""Priors on constant poses beside priors on free ones, in every order of their
indices: a constant pose's prior adds its cost and nothing else, so S, the rhs,
the step and the covariance keep the bits that they have without it."""
import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("const", [(0,), (2,), (5,), (0, 3), (0, 1, 2, 4)])
def test_constant_pose_priors(pkg, oracle, const):
    rng = np.random.default_rng(sum(const))
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=6, n_pt=80, seed=pkg.synth.BASE_SEED + 31)
    prob.pose_const = np.zeros(6, np.uint8)
    prob.pose_const[list(const)] = 1
    sel = np.array([5, 0, 2, 1, 2, 0, 4, 3], np.int32)
    means = np.array([oracle.se3_mul(oracle.se3_exp(0.05 * rng.standard_normal(6)), prob.poses[j]) for j in sel])
    Ws = np.array([(lambda a: 50.0 * (a @ a.T + 6 * np.eye(6)))(rng.standard_normal((6, 6))) for _ in sel])
    free = prob.pose_const[sel] == 0
    nu = prob.initial_lm_damping
    out = []
    for keep in (free, np.ones(len(sel), bool)):
        with pkg.native.Problem(prob, device=0) as p:
            p.set_pose_priors(sel[keep], means[keep], Ws[keep])
            p.covariance_prepare()
            cov = np.stack(p.covariance_blocks([((1, j), (1, j)) for j in range(6) if not prob.pose_const[j]]))
            p.init(fixed_iter_params(pkg, 1, nu))
            cost = p.cost()
            p.step()
            out.append((cost, cov) + tuple(np.asarray(a) for a in p.last_system()))
    extra = 0.0
    for j, E, W in zip(sel[~free], means[~free], Ws[~free]):
        g = oracle.se3_log(oracle.se3_mul(prob.poses[j], oracle.se3_inverse(E)))
        extra += g @ W @ g
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(a, b)
    # the costs are float-float sums (48 bits)
    assert abs(out[1][0] - out[0][0] - extra) <= 2.0**-40 * out[1][0]
