"""The tiled Schur pass of one problem by its ways: rounds split over CTAs in one
pass and in two (k_schur_dense_split: 36 MB of sums a pass, here 15 tiles and
438 rounds), not split with eight groups a CTA (over 64 MB in all:
k_schur_dense<8>) and with two (more than 304 tiles: k_schur_dense<2>).  The
batched launches add the rounds in the same order, so a batch gives the same
bits (k_schur_dense_w<8>, and <2> past 304 tiles in a group; more windows than
SMs, which go to the solver by size); S of the larger ones against the f64 sum,
within test_gpu_schur_tiles' 64 x 2^-24 of sqrt(U_ii U_jj)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, fixed_iter_params
from test_gpu_schur_tiles import _reference_s

pytestmark = pytest.mark.gpu


def _scenes(pkg, shapes):
    return [pkg.synth.generate(pkg.synth.WINDOW, n, m, seed=1000 + i) for i, (n, m) in enumerate(shapes)]


def _same_as_single(pkg, scenes, iters):
    params = fixed_iter_params(pkg, iters, scenes[0].initial_lm_damping)
    batch = pkg.native.create_problems(scenes)
    try:
        results = pkg.native.batch_optimize(batch, params)
        for p, s, (recs, *_) in zip(batch, scenes, results):
            with pkg.native.Problem(s, device=0) as q:
                one, _ = q.optimize(params)
                assert [r.merit for r in one] == [r.merit for r in recs]
                for a, b in zip(p.variables(), q.variables()):
                    assert np.array_equal(a, b)
    finally:
        for p in batch:
            p.close()


def test_passes(pkg):
    _same_as_single(pkg, _scenes(pkg, [(40, 4000), (40, 7000), (40, 4167), (34, 5001), (40, 8001), (9, 33), (8, 16)]), 3)


def test_more_windows_than_sms(pkg):
    """Up to four groups a batch: 700 windows are past 304 tiles and 152 windows in each."""
    rng = np.random.default_rng(5)
    shapes = [(int(rng.integers(5, 41)), int(rng.integers(60, 300))) for _ in range(700)]
    _same_as_single(pkg, _scenes(pkg, shapes), 2)


@pytest.mark.parametrize("cams,points", [(40, 8001), (201, 160)])
def test_reduced_system(pkg, cams, points):
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=cams, n_pt=points, seed=pkg.synth.BASE_SEED + points)
    with pkg.native.Problem(prob, device=0) as p:
        ref, d = _reference_s(p, prob, prob.initial_lm_damping)
        p.init(fixed_iter_params(pkg, 1, prob.initial_lm_damping))
        p.step()
        S, _, _ = p.last_system()
    err = np.abs(np.tril(S - ref)) / np.outer(d, d)
    assert err.max() < 64 * 2.0 ** -24, err.max()


_GROWTH = """
import sys
sys.path[:0] = [%r, %r]
import torch
import __graft_entry__ as g
from conftest import fixed_iter_params
pkg = g.load_package()
prob = pkg.synth.generate(pkg.synth.WINDOW, 40, 7000, seed=3)
keep = [pkg.native.Problem(prob, device=0) for _ in range(8)]
before = torch.cuda.mem_get_info()[0]
for p in keep:
    p.init(fixed_iter_params(pkg, 1, prob.initial_lm_damping))
print(before - torch.cuda.mem_get_info()[0])
"""


def test_memory(pkg):
    """Eight kept maps whose rounds' sums are 60 MB each: 36 MB of them and the sums between
    passes, the pool's growth in steps of 32 MB, the records and the graphs."""
    out = subprocess.run([sys.executable, "-c", _GROWTH % (ROOT, os.path.join(ROOT, "tests"))], capture_output=True,
                         text=True, check=True)
    assert int(out.stdout) < 368 << 20, out.stdout
