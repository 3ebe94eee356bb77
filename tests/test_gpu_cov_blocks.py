"""Covariance of the solution at the edges of the blocked factor and inverse
(factor panels and inverse blocks of 48 rows, doubling levels of the inverse,
eight lanes a row in a point query): n just below, at and above one, two and
four blocks, a ragged last block, every kind of block against the oracle.

Both sides work in f64 on the same S up to its rounding: a block's error is that
rounding, 2^-53 of the sums of S, times S's condition (below 1e8 for these dense
spheres with two constant poses): 1e-7 of the largest entry."""
import numpy as np
import pytest

from test_gpu_covariance import _check, _observed_points, _queries, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("free", [1, 7, 8, 9, 15, 16, 17, 31, 33])
def test_blocks(pkg, oracle, free):
    prob = pkg.synth.generate(pkg.synth.SPHERE, n_cam=free + 2, n_pt=40 * (free + 2), seed=pkg.synth.BASE_SEED + free)
    prob.pose_const[:] = 0
    prob.pose_const[:2] = 1
    gp, at = _solve(pkg, prob)
    with gp:
        info = gp.covariance_prepare()
        assert info.n == info.rank == 6 * free
        poses = list(range(2, free + 2))
        _check(gp, oracle, at, _queries(prob, poses, _observed_points(prob, 3)))
        got = gp.covariance_blocks([((1, j), (1, j)) for j in poses])
    for b in got:  # a covariance: symmetric, positive
        assert np.abs(b - b.T).max() <= 1e-12 * np.abs(b).max() and np.linalg.eigvalsh(b).min() > 0
