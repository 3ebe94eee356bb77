"""Free camera params with more terms than the per-term buffers hold (2^18): the
system against the f64 sums, just above one chunk and with several, and the
device memory that the free params add.

Bounds as in test_gpu_intrinsics_blocks: 64 x 2^-24 of sqrt(H_ii H_jj), and of
sqrt(H_ii) |r| for the rhs."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, fixed_iter_params
from test_gpu_intrinsics_blocks import _reference

pytestmark = pytest.mark.gpu


def _scene(pkg, cams, points):
    prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=cams, n_pt=points, seed=pkg.synth.BASE_SEED + points)
    prob.intrinsics = prob.intrinsics * np.array([1.02, 0.985, 1.0, 1.0]) + np.array([0.0, 0.0, 3.0, -2.0])
    prob.intrinsics_free = True
    prob.huber_delta = 0.0
    return prob


@pytest.mark.parametrize("cams,points", [(12, 22000), (12, 21800), (9, 80000)])
def test_chunks(pkg, cams, points):
    prob = _scene(pkg, cams, points)
    nu = prob.initial_lm_damping
    with pkg.native.Problem(prob, device=0) as p:
        ref, rref, d, rn = _reference(p, prob, nu)
        p.init(fixed_iter_params(pkg, 1, nu))
        p.step()
        S, rhs, _ = p.last_system()
    off = np.abs(S[6:, :6].T - ref[:, 6:])[:4] / np.outer(d[:4], d[6:])
    dia = np.abs((S[:6, :6] - ref[:, :6]) * (1 - np.eye(6)))[:4, :4] / np.outer(d[:4], d[:4])
    bound = 64 * 2.0 ** -24
    assert off.max() < bound, off.max()
    assert dia.max() < bound, dia.max()
    assert (np.abs(rhs[:4] - rref[:4]) / (d[:4] * rn)).max() < bound


_GROWTH = """
import sys
sys.path[:0] = [%r, %r]
import torch
import __graft_entry__ as g
pkg = g.load_package()
prob = pkg.synth.generate(pkg.synth.CIRCLE, n_cam=9, n_pt=160000, seed=3)
keep, used = [], []
for free in (False, True, False):
    prob.intrinsics_free = free
    before = torch.cuda.mem_get_info()[0]
    keep.append(pkg.native.Problem(prob, device=0))
    used.append(before - torch.cuda.mem_get_info()[0])
print(used[1] - used[2], prob.n_obs)
"""


def test_memory(pkg):
    """1.4M terms: bounded buffers, where 432 bytes a term would be 600 MB."""
    out = subprocess.run([sys.executable, "-c", _GROWTH % (ROOT, os.path.join(ROOT, "tests"))], capture_output=True,
                         text=True, check=True)
    extra, n_obs = map(int, out.stdout.split())
    assert n_obs > 1200000
    # the chunk buffer 38 MB, 144 bytes a point 23 MB, pool granularity; beside the larger S and pair lists
    assert extra < 200 << 20, extra
