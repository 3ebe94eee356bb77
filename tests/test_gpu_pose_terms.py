"""Pose-graph edges and pose priors, eight lanes a term (k_pose_terms), at the
edges of its CTAs (8 terms), with several edges in a term and past its largest
grid (2048 terms): cost and blocks of S against numpy.

Reference: the logs of the oracle, D by central differences (h = 1e-4: h^2 of
third derivatives of O(1), 1e-8; 1e-16 / h from rounding).  S is float-float, so
a difference of two S carries 2^-40 of the largest entry."""
import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu

H = 1e-4


def _deriv(oracle, A, B):
    f = lambda x: oracle.se3_log(oracle.se3_mul(oracle.se3_mul(A, oracle.se3_exp(x)), B))  # noqa: E731
    return f(np.zeros(6)), np.stack([(f(H * e) - f(-H * e)) / (2 * H) for e in np.eye(6)], axis=1)


def _system(pkg, prob, priors=None):
    with pkg.native.Problem(prob, device=0) as p:
        if priors:
            p.set_pose_priors(*priors)
        p.init(fixed_iter_params(pkg, 1, prob.initial_lm_damping))
        c = p.cost()
        p.step()
        return c, p.last_system()[0]


@pytest.mark.parametrize("n_edge,n_dup,n_prior", [(1, 0, 1), (7, 2, 8), (8, 0, 9), (9, 3, 0), (2052, 5, 2051)])
def test_blocks_and_cost(pkg, oracle, n_edge, n_dup, n_prior):
    rng = np.random.default_rng(n_edge + n_prior)
    n_cam = 6 if n_edge < 20 else 47
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=n_cam, n_pt=60, seed=pkg.synth.BASE_SEED + 5)
    T, free = prob.poses, np.nonzero(prob.pose_const == 0)[0]
    row = {int(j): 6 * k for k, j in enumerate(free)}
    rel = lambda m, n: oracle.se3_mul(oracle.se3_exp(0.3 * rng.standard_normal(6)),  # noqa: E731
                                      oracle.se3_mul(oracle.se3_inverse(T[m]), T[n]))
    pairs = [(m, n) for m in range(n_cam) for n in range(n_cam) if m != n][:n_edge + 1]
    pairs += pairs[1:1 + n_dup]
    mns = [rel(m, n) for m, n in pairs]
    base, full = prob.copy(), prob.copy()
    for p, k in ((base, 1), (full, len(pairs))):
        p.edge_pose, p.edge_mn = np.array(pairs[:k], np.int32), np.array(mns[:k])
    sel = rng.choice(free, n_prior)
    means = np.array([oracle.se3_mul(oracle.se3_exp(0.3 * rng.standard_normal(6)), T[j]) for j in sel]).reshape(-1, 7)
    Ws = np.array([(lambda a: a @ a.T + np.eye(6))(rng.standard_normal((6, 6))) for _ in sel]).reshape(-1, 6, 6)
    nu = prob.initial_lm_damping
    c0, S0 = _system(pkg, base)
    c1, S1 = _system(pkg, full, (sel.astype(np.int32), means, Ws) if n_prior else None)
    ref, cost, seen = np.zeros_like(S0), 0.0, {pairs[0]}
    for (m, n), mn in list(zip(pairs, mns))[1:]:
        g, D = _deriv(oracle, oracle.se3_inverse(T[m]), oracle.se3_mul(T[n], oracle.se3_inverse(mn)))
        cost += g @ g
        damp = 0.0 if (m, n) in seen else nu
        seen.add((m, n))
        for j in (m, n):
            if j in row:
                ref[row[j]:row[j] + 6, row[j]:row[j] + 6] += D.T @ D + damp * np.eye(6)
        if m in row and n in row:
            a, b = max(row[m], row[n]), min(row[m], row[n])
            ref[a:a + 6, b:b + 6] -= D.T @ D
    for j in set(sel.tolist()) & set(row):
        ref[row[j]:row[j] + 6, row[j]:row[j] + 6] += nu * np.eye(6)
    eye = np.array([1.0, 0, 0, 0, 0, 0, 0])
    for j, E, W in zip(sel, means, Ws):
        g, D = _deriv(oracle, eye, oracle.se3_mul(T[j], oracle.se3_inverse(E)))
        cost += g @ W @ g
        if j in row:
            ref[row[j]:row[j] + 6, row[j]:row[j] + 6] += D.T @ W @ D
    assert abs(c1 - c0 - cost) <= 1e-12 * (c1 + cost)
    tol = 1e-7 * (1 + np.abs(ref).max()) + 2.0**-40 * np.abs(S1).max()
    assert np.abs(np.tril(S1 - S0 - ref)).max() < tol
