"""Residuals and Jacobians of pose-graph edges and pose priors where the SE(3) log
changes its form: the zero residual, just below and above |q_v| = 1e-6 (series of
the rotation log) and theta^2 = 1e-6 (series of V^-1), and near a half turn.

The H blocks are queried in f64 (J_m^T J_n of an edge stands alone in its block, a
prior's J^T W J is the difference of two), the residuals through the cost of
scenes without pixel error.  The Jacobian in f64 is J_l^-1(xi) Ad_A with the
Bernoulli series of J_l^-1.  Below theta^2 = 1e-6 the log takes 1/12 for the
coefficient of V^-1, 1e-6 / 720 off, and no derivative for it, theta / 360 off: at
most 1e-8 / 360 theta |t| in D, 3e-11 |t| ; above it cancellation leaves 2^-53 /
theta |t|, 1e-13 |t|.  H = D^T W D sums 36 products of twice that: 1e-8 of
|W| (1 + |t|)^2.  The cost is a float-float sum (2^-40), its residuals within
1e-14 (1 + |t|) / theta of the log's."""
import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu

PRECISION = 1
ANGLES = [0.0, 1e-9, 1.9e-6, 2.1e-6, 9.9e-4, 1.01e-3, 0.3, np.pi - 1e-2, np.pi - 1e-5]


def _hat(w):
    return np.array([[0.0, -w[2], w[1]], [w[2], 0.0, -w[0]], [-w[1], w[0], 0.0]])


def _jl_inv(xi):
    ad = np.zeros((6, 6))
    ad[:3, :3] = ad[3:, 3:] = _hat(xi[:3])
    ad[3:, :3] = _hat(xi[3:])
    out, term = np.eye(6) - 0.5 * ad, np.eye(6)
    sq = ad @ ad
    for n in range(1, 40):  # B_2n / (2n)! = (-1)^(n + 1) 2 zeta(2n) / (2 pi)^2n
        term = term @ sq / (2 * np.pi) ** 2
        zeta = np.pi**2 / 6 if n == 1 else sum(k ** (-2.0 * n) for k in range(1, 2000)) + 2000.0 ** (1 - 2 * n) / (2 * n - 1)
        out = out + (-1) ** (n + 1) * 2 * zeta * term
    return out


def _adjoint(T):
    w, x, y, z = T[:4]
    R = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                  [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                  [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]])
    A = np.zeros((6, 6))
    A[:3, :3] = A[3:, 3:] = R
    A[3:, :3] = _hat(T[4:]) @ R
    return A


def _scene(pkg):
    """A circle without pixel error, the focal length 1: its part of H is of the edges' size."""
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=6, n_pt=60, seed=pkg.synth.BASE_SEED + 12)
    prob.poses, prob.points = prob.poses_true.copy(), prob.points_true.copy()
    prob.intrinsics = np.array([1.0, 1.0, 0.0, 0.0])
    q, v = -prob.poses[prob.obs_cam, 1:4], prob.points[prob.obs_pt] - prob.poses[prob.obs_cam, 4:]
    u = 2.0 * np.cross(q, v)
    c = v + prob.poses[prob.obs_cam, :1] * u + np.cross(q, u)
    prob.obs_uv = c[:, :2] / c[:, 2:]
    return prob


def _residual(rng, theta):
    w = rng.standard_normal(3)
    return np.concatenate([theta * w / np.linalg.norm(w), rng.standard_normal(3)])


def _cost(pkg, p):
    p.init(fixed_iter_params(pkg, 1, 1e-3))
    return p.cost()


def test_series(oracle):
    """J_l^-1 of the series against central differences of the oracle's log."""
    rng = np.random.default_rng(1)
    xi = _residual(rng, 2.5)
    T, h = oracle.se3_exp(xi), 1e-4
    D = np.stack([(oracle.se3_log(oracle.se3_mul(oracle.se3_exp(h * e), T))
                   - oracle.se3_log(oracle.se3_mul(oracle.se3_exp(-h * e), T))) / (2 * h) for e in np.eye(6)], axis=1)
    assert np.abs(D - _jl_inv(xi)).max() < 1e-7


@pytest.mark.parametrize("theta", ANGLES)
def test_edge(pkg, oracle, theta):
    rng = np.random.default_rng(int(1e3 * theta))
    prob = _scene(pkg)
    T, pairs = prob.poses, [(1, 2), (4, 3), (5, 1)]
    xis = [_residual(rng, theta) for _ in pairs]
    prob.edge_pose = np.array(pairs, np.int32)
    prob.edge_mn = np.array([oracle.se3_mul(oracle.se3_exp(-xi), oracle.se3_mul(oracle.se3_inverse(T[m]), T[n]))
                             for (m, n), xi in zip(pairs, xis)])
    with pkg.native.Problem(prob, device=0) as p:
        cost = _cost(pkg, p)
        p.covariance_prepare()
        H = p.covariance_blocks([((1, m), (1, n)) for m, n in pairs], PRECISION)
    ref, t = 0.0, 1.0
    for (m, n), mn, h in zip(pairs, prob.edge_mn, H):
        A = oracle.se3_inverse(T[m])
        xi = oracle.se3_log(oracle.se3_mul(A, oracle.se3_mul(T[n], oracle.se3_inverse(mn))))
        D = _jl_inv(xi) @ _adjoint(A)
        s = (1 + np.abs(T[:, 4:]).max() + np.linalg.norm(xi[3:])) ** 2
        assert np.abs(h + D.T @ D).max() < 1e-8 * s
        ref, t = ref + xi @ xi, max(t, s)
    assert abs(cost - ref) < 2.0**-40 * ref + 1e-13 * t


@pytest.mark.parametrize("theta", ANGLES)
def test_prior(pkg, oracle, theta):
    rng = np.random.default_rng(int(1e3 * theta) + 7)
    prob = _scene(pkg)
    T, sel = prob.poses, [1, 3, 5]
    xis = [_residual(rng, theta) for _ in sel]
    means = np.array([oracle.se3_mul(oracle.se3_exp(-xi), T[j]) for j, xi in zip(sel, xis)])
    Ws = np.array([(lambda a: a @ a.T + np.eye(6))(rng.standard_normal((6, 6))) for _ in sel])
    query = [((1, j), (1, j)) for j in sel]
    with pkg.native.Problem(prob, device=0) as p:
        p.covariance_prepare()
        base = p.covariance_blocks(query, PRECISION)
        p.set_pose_priors(np.array(sel, np.int32), means, Ws)
        cost = _cost(pkg, p)
        p.covariance_prepare()
        H = p.covariance_blocks(query, PRECISION)
    ref, t = 0.0, 1.0
    for j, E, W, h, b in zip(sel, means, Ws, H, base):
        xi = oracle.se3_log(oracle.se3_mul(T[j], oracle.se3_inverse(E)))
        D = _jl_inv(xi)
        s = np.abs(W).max() * (1 + np.abs(T[:, 4:]).max() + np.linalg.norm(xi[3:])) ** 2
        assert np.abs(h - b - D.T @ W @ D).max() < 1e-8 * s
        ref, t = ref + xi @ W @ xi, max(t, s)
    assert abs(cost - ref) < 2.0**-40 * ref + 1e-13 * t
