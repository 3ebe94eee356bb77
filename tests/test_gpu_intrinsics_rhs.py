"""The reduced rhs has rows for the camera params after those of the poses: with
10 or 16 free poses these rows lie beyond 6 nf doubles rounded up to 256 bytes,
and at 15 they end with them.  Its values against the f64 sums, with a second
problem of the same kind whose buffers follow."""
import numpy as np
import pytest

from conftest import fixed_iter_params
from test_gpu_intrinsics_blocks import _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cams", [11, 16, 17])
def test_rhs_rows(pkg, cams):
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=cams, n_pt=300, seed=pkg.synth.BASE_SEED + cams)
    prob.intrinsics = prob.intrinsics * np.array([1.02, 0.985, 1.0, 1.0]) + np.array([0.0, 0.0, 3.0, -2.0])
    prob.intrinsics_free = True
    prob.huber_delta = 0.0
    nu = prob.initial_lm_damping
    with pkg.native.Problem(prob, device=0) as p, pkg.native.Problem(prob, device=0) as q:
        _, rref, d, rn = _reference(p, prob, nu)
        got = []
        for x in (p, q):
            x.init(fixed_iter_params(pkg, 1, nu))
            x.step()
            got.append(x.last_system()[1])
    assert np.array_equal(got[0], got[1])
    # float-float sums of FP32-split residuals: 64 x 2^-24 of sqrt(H_ii) |r|
    assert (np.abs(got[0][:4] - rref[:4]) / (d[:4] * rn)).max() < 64 * 2.0 ** -24
