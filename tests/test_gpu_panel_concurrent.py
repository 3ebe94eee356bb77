"""The panel solver of large dense systems (k_ldlt_panel) beside other work on the
GPU, whose CTAs delay some of a panel's: the records and variables are those of
the same problem alone, bit for bit."""
import threading

import numpy as np
import pytest

from conftest import fixed_iter_params

pytestmark = pytest.mark.gpu


def test_beside_other_problems(pkg):
    prob = pkg.synth.generate(pkg.synth.SPHERE, n_cam=420, n_pt=20000, seed=pkg.synth.BASE_SEED + 9)
    loop = pkg.synth.generate(pkg.synth.LOOP, n_cam=300, n_pt=60000, seed=pkg.synth.BASE_SEED)
    params = fixed_iter_params(pkg, 3, prob.initial_lm_damping)
    with pkg.native.Problem(prob, device=0) as p:
        assert p.layout().solver == pkg.native.SOLVER_DENSE_PANELS
        alone, _ = p.optimize(params)
        ref = p.variables()
    got, stop = [None, None], threading.Event()

    def panels(k):
        with pkg.native.Problem(prob, device=0) as p:
            recs, _ = p.optimize(params)
            got[k] = [r.merit for r in recs], p.variables()

    def load():
        with pkg.native.Problem(loop, device=0) as p:
            while not stop.is_set():
                p.set_variables(loop.poses, loop.points)
                p.optimize(fixed_iter_params(pkg, 3, loop.initial_lm_damping))

    busy = threading.Thread(target=load)
    work = [threading.Thread(target=panels, args=(k,)) for k in range(2)]
    busy.start()
    for t in work:
        t.start()
    for t in work:
        t.join()
    stop.set()
    busy.join()
    for merits, variables in got:
        assert merits == [r.merit for r in alone]
        for a, b in zip(variables, ref):
            assert np.array_equal(a, b)
