"""Set-up and read-back through the page-locked staging blocks (4 MB each, 16 in
the process): more problems at once than blocks, arrays that fill a block, that
pass its end and that are larger than it.  Copies carry every bit, and the cost
does not depend on how the arrays came to the device."""
import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu


def _scene(pkg, cams, points, k):
    return pkg.synth.generate(pkg.synth.CIRCLE, n_cam=cams, n_pt=points, seed=pkg.synth.BASE_SEED + k)


@pytest.mark.parametrize("count,cams,points", [(24, 6, 150), (3, 20, 4000), (2, 30, 9000), (1, 40, 40000)])
def test_copies(pkg, count, cams, points):
    scenes = [_scene(pkg, cams, points + 7 * k, k) for k in range(count)]
    many = pkg.native.create_problems(scenes, threads=16)
    try:
        costs = []
        for p, s in zip(many, scenes):
            poses, pts = p.variables()
            assert np.array_equal(pts, s.points)
            assert np.array_equal(poses, np.where(s.poses[:, :1] < 0, np.c_[-s.poses[:, :4], s.poses[:, 4:]], s.poses))
            p.init(fixed_iter_params(pkg, 1, s.initial_lm_damping))
            costs.append(p.cost())
    finally:
        for p in many:
            p.close()
    for s, c in zip(scenes, costs):
        with pkg.native.Problem(s, device=0) as p:
            p.init(fixed_iter_params(pkg, 1, s.initial_lm_damping))
            assert p.cost() == c
