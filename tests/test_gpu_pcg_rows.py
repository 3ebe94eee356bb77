"""The row-per-warp PCG kernel (k_pcg_rows) and the general one (k_pcg_solve)
at the edges of their rule (16-row groups, 512 rows, rows of 195 blocks): the
relative residual after eight iterations against the same recurrences in numpy.

Eight iterations on systems of condition below 1e4 amplify the rounding of the
vectors (2^-53) and of the float-float products (2^-44) to well below 1e-8 of
the residual."""
import numpy as np
import pytest

from pcg_systems import random_system

pytestmark = pytest.mark.gpu


def _cg(nf, rows, cols, blocks, b, iters):
    """Chronopoulos-Gear with the block-Jacobi preconditioner; |r| / |b|."""
    A = np.zeros((6 * nf, 6 * nf))
    for j, k, B in zip(rows, cols, blocks.reshape(-1, 6, 6)):
        A[6 * j:6 * j + 6, 6 * k:6 * k + 6] = B
        A[6 * k:6 * k + 6, 6 * j:6 * j + 6] = B.T
    D = np.stack([np.linalg.inv(A[6 * j:6 * j + 6, 6 * j:6 * j + 6]) for j in range(nf)])
    P = lambda v: np.einsum("jab,jb->ja", D, v.reshape(nf, 6)).ravel()  # noqa: E731
    r, p, s, u = b.copy(), np.zeros_like(b), np.zeros_like(b), P(b)
    for it in range(iters):
        w = A @ u
        g, d = r @ u, w @ u
        beta = 0.0 if it == 0 else g / gamma
        alpha = g / d if it == 0 else g / (d - beta * g / alpha)
        gamma = g
        p, s = u + beta * p, w + beta * s
        r = r - alpha * s
        u = P(r)
    return np.linalg.norm(r) / np.linalg.norm(b)


@pytest.mark.parametrize("nf,band", [(3, 2), (15, 2), (16, 15), (17, 5), (65, 64), (120, 119), (194, 193), (210, 209),
                                     (511, 3), (512, 40), (513, 3)])
def test_residual_after_eight_iterations(pkg, nf, band):
    rows, cols, blocks, b, x = random_system(nf, seed=nf, band=band)
    with pkg.native.PcgTrainSet(device=0) as ts:
        ts.add(nf, rows, cols, blocks, b, x)
        it, rr, _ = ts.evaluate(0, 1, max_iterations=8, tolerance=1e-30)
    assert it == 8
    ref = _cg(nf, rows, cols, blocks, b, 8)
    assert abs(rr - ref) <= 1e-8 * ref, (rr, ref)
