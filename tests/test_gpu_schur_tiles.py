"""The tiled Schur pass (k_schur_dense) at the edges of its tiles (8 pose
blocks), rounds (16 points) and round groups (8 rounds a pass of a CTA): S of
one LM step against the same sum formed in f64 from the per-term Jacobians.

The pass works on FP32 Z (24 bits) with FP32 products over rounds of 16
points.  An entry of sum Z Z^T is bounded by its diagonal entries
(Cauchy-Schwarz); each of the 48 FP32 products of a round and the Z it reads
carry at most a few 2^-24 of them, so the entries are within
64 x 2^-24 = 4e-6 of sqrt(U_ii U_jj)."""
import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu


def _reference_s(p, prob, nu):
    """S in f64 from the float-float Jacobians at the initial variables."""
    order = np.lexsort((prob.obs_cam, prob.obs_pt))
    oc, op = prob.obs_cam[order], prob.obs_pt[order]
    jp, jm = p.jacobians(oc, op, precision=1)
    n, m = prob.n_cam - 1, prob.n_pt
    V = np.zeros((m, 3, 3))
    np.add.at(V, op, np.einsum("kri,krj->kij", jm, jm))
    V[:, range(3), range(3)] += nu * np.bincount(op, minlength=m)[:, None]
    W = np.zeros((m, 6 * n, 3))
    U = np.zeros((6 * n, 6 * n))
    for k in np.nonzero(oc > 0)[0]:
        r = slice(6 * (oc[k] - 1), 6 * oc[k])
        W[op[k], r] += jp[k].T @ jm[k]
        U[r, r] += jp[k].T @ jp[k]
    d = np.sqrt(np.diag(U))
    U[range(6 * n), range(6 * n)] += nu * np.repeat(np.bincount(oc, minlength=n + 1)[1:], 6)
    return U - np.einsum("mik,mkl,mjl->ij", W, np.linalg.inv(V), W), d


@pytest.mark.parametrize("cams,points", [(2, 15), (9, 16), (10, 17), (17, 127), (18, 129), (26, 300), (40, 257)])
def test_reduced_system(pkg, cams, points):
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=cams, n_pt=points, seed=pkg.synth.BASE_SEED + points)
    with pkg.native.Problem(prob, device=0) as p:
        ref, d = _reference_s(p, prob, prob.initial_lm_damping)
        p.init(fixed_iter_params(pkg, 1, prob.initial_lm_damping))
        p.step()
        S, _, _ = p.last_system()
    err = np.abs(np.tril(S - ref)) / np.outer(d, d)
    assert err.max() < 64 * 2.0 ** -24, err.max()
