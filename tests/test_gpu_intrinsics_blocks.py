"""The free intrinsics' rows of S and of the rhs (k_intr_terms, k_intr_points,
k_intr_cams) at the edges of their splits (warps of 32 and CTAs of 64 terms, 8
points a CTA and 608 CTAs, 64-term quarters of a pose's 256-term tiles): one LM
step's system against the same sums formed in f64.

The sums are float-float; the Z of a term that they read is FP32 (24 bits).  By
Cauchy-Schwarz each product is within its two diagonal entries, and the three
products of an entry and their two operands carry at most a few 2^-24 of that:
64 x 2^-24 of sqrt(H_ii H_jj), as for the other rows of S.  The rhs is the
float-float sum of FP32-split residuals: 64 x 2^-24 of sqrt(H_ii) |r|."""
import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu


def _reference(p, prob, nu):
    order = np.lexsort((prob.obs_cam, prob.obs_pt))
    oc, op = prob.obs_cam[order], prob.obs_pt[order]
    jp, jm = p.jacobians(oc, op, precision=1)
    # world_from_camera: camera coordinates with the conjugate of (w x y z)
    q, v = -prob.poses[oc, 1:4], prob.points[op] - prob.poses[oc, 4:]
    u = 2.0 * np.cross(q, v)
    c = v + prob.poses[oc, :1] * u + np.cross(q, u)
    xy = c[:, :2] / c[:, 2:]
    uv = prob.obs_uv[order]
    r = uv - (xy * prob.intrinsics[:2] + prob.intrinsics[2:4])
    jk = np.zeros((len(oc), 2, 6))
    jk[:, 0, 0], jk[:, 1, 1], jk[:, 0, 2], jk[:, 1, 3] = -xy[:, 0], -xy[:, 1], -1.0, -1.0
    n, m = prob.n_cam - 1, prob.n_pt
    V = np.zeros((m, 3, 3))
    np.add.at(V, op, np.einsum("kri,krj->kij", jm, jm))
    V[:, range(3), range(3)] += nu * np.bincount(op, minlength=m)[:, None]
    bm = np.zeros((m, 3))
    np.add.at(bm, op, np.einsum("kri,kr->ki", jm, r))
    W = np.zeros((m, 6, 3))
    np.add.at(W, op, np.einsum("kri,krj->kij", jk, jm))
    Vi = np.linalg.inv(V)
    hkk = np.einsum("kri,krj->ij", jk, jk)
    S = np.zeros((6, 6 * (n + 1)))
    S[:, :6] = hkk - np.einsum("mik,mkl,mjl->ij", W, Vi, W)
    d = np.zeros(6 * (n + 1))
    d[:6] = np.sqrt(np.diag(hkk))
    for j in range(n):
        k = np.nonzero(oc == j + 1)[0]
        X = np.einsum("kri,krj->kij", jp[k], jm[k])
        cols = slice(6 + 6 * j, 12 + 6 * j)
        S[:, cols] = np.einsum("kri,krj->ij", jk[k], jp[k]) - np.einsum("kia,kab,kjb->ij", W[op[k]], Vi[op[k]], X)
        d[cols] = np.sqrt(np.einsum("kri,kri->i", jp[k], jp[k]))
    rhs = -np.einsum("kri,kr->i", jk, r) + np.einsum("mik,mkl,ml->i", W, Vi, bm)
    return S, rhs, d, np.linalg.norm(r)


@pytest.mark.parametrize("cams,points", [(2, 31), (3, 32), (2, 33), (5, 63), (4, 65), (9, 257), (3, 511), (6, 5000)])
def test_intrinsics_rows(pkg, cams, points):
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=cams, n_pt=points, seed=pkg.synth.BASE_SEED + points)
    prob.intrinsics = prob.intrinsics * np.array([1.02, 0.985, 1.0, 1.0]) + np.array([0.0, 0.0, 3.0, -2.0])
    prob.intrinsics_free = True
    prob.huber_delta = 0.0
    nu = prob.initial_lm_damping
    with pkg.native.Problem(prob, device=0) as p:
        ref, rref, d, rn = _reference(p, prob, nu)
        p.init(fixed_iter_params(pkg, 1, nu))
        p.step()
        S, rhs, _ = p.last_system()
    off = np.abs(S[6:, :6].T - ref[:, 6:])[:4] / np.outer(d[:4], d[6:])
    # the block's damping is nu per term on its diagonal: compared off the diagonal
    dia = np.abs((S[:6, :6] - ref[:, :6]) * (1 - np.eye(6)))[:4, :4] / np.outer(d[:4], d[:4])
    bound = 64 * 2.0 ** -24
    assert off.max() < bound, off.max()
    assert dia.max() < bound, dia.max()
    assert (np.abs(rhs[:4] - rref[:4]) / (d[:4] * rn)).max() < bound
