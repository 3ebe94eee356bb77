"""Creating and closing many problems at once leaves no page-locked host memory
behind in the process (it is mapped shared: RssShmem), and the copies of small
and large arrays carry every bit, whatever way they go."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shared_kb():
    with open("/proc/self/status") as f:
        for line in f:
            if line.startswith("RssShmem"):
                return int(line.split()[1])
    pytest.skip("no RssShmem on this kernel")


def test_nothing_page_locked_stays(pkg):
    scenes = [pkg.synth.generate(pkg.synth.WINDOW, 20, 1000, seed=k) for k in range(48)]
    pkg.native.Problem(scenes[0], device=0).close()
    before = _shared_kb()
    problems = pkg.native.create_problems(scenes, threads=24)
    try:
        for p, s in zip(problems, scenes):
            assert np.array_equal(p.variables()[1], s.points)
    finally:
        for p in problems:
            p.close()
    assert _shared_kb() - before < 4096
