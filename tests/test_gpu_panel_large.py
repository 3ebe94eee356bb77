"""The panel solver past 48 KB of its solve's right-hand side (12,288 rows; the
limit is 4,096 free poses): the steps lower the cost, as just below."""
import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cams", [2049, 2060])
def test_solve(pkg, cams):
    prob = pkg.synth.generate(pkg.synth.SPHERE, n_cam=cams, n_pt=30000, seed=pkg.synth.BASE_SEED + 3)
    with pkg.native.Problem(prob, device=0) as p:
        assert p.layout().solver == pkg.native.SOLVER_DENSE_PANELS
        recs, _ = p.optimize(fixed_iter_params(pkg, 3, prob.initial_lm_damping))
    merits = [r.merit for r in recs]
    assert np.isfinite(merits).all() and merits[-1] < 0.9 * merits[0], merits
