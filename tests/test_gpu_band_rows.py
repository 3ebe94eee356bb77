"""The forward sweep's rows of a CTA (one, or two neighbours from 153 rows of all
segments on) and its ring of solved columns: odd and even row counts, a band
wider and narrower than a panel, bands shorter than the ring.  The LM step against
an f64 solve of the exported reduced system, outside the scale gauge: the
float-float solver's error is 2^-44 times the condition of the scaled S (below
1e7 for these loops)."""
import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cams,per_cam", [(60, 30), (61, 60), (90, 40), (141, 30), (173, 45), (260, 30)])
def test_step_matches_f64(pkg, cams, per_cam):
    prob = pkg.synth.generate(pkg.synth.LOOP, n_cam=cams, n_pt=per_cam * cams, seed=pkg.synth.BASE_SEED + cams)
    with pkg.native.Problem(prob, device=0) as p:
        assert p.layout().solver == pkg.native.SOLVER_BAND
        p.init(fixed_iter_params(pkg, 2, prob.initial_lm_damping))
        poses, _ = p.variables()
        p.step()
        S, rhs, delta = p.last_system()
    n = len(rhs)
    d = 1.0 / np.sqrt(np.diag(S))
    x = d * np.linalg.solve(S * np.outer(d, d), rhs * d)
    v = np.zeros(n)
    c = poses[np.nonzero(prob.pose_const)[0][0], 4:]
    for k, j in enumerate(np.nonzero(prob.pose_const == 0)[0]):
        v[6 * k + 3:6 * k + 6] = poses[j, 4:] - c
    v /= np.linalg.norm(v)
    off = lambda y: y - v * (v @ y)  # noqa: E731
    assert np.linalg.norm(off(delta[:n]) - off(x)) < 2.0**-44 * 1e7 * np.linalg.norm(off(x))
