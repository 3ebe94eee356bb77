"""Several large problems created at once still have the host pool's workers: the
share of the creations' CPU time that falls on them.  (Without a GPU a creation
ends after its host plan, which is what is measured here.)  In a process of its
own, where the pool's threads are those that the first creation starts."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

_RUN = """
import os, sys, threading, time
sys.path.insert(0, %r)
import __graft_entry__ as g
pkg = g.load_package()
prob = pkg.synth.generate(pkg.synth.LOOP, n_cam=400, n_pt=60000, seed=pkg.synth.BASE_SEED)

def cpu(tids):
    total = 0
    for t in tids:
        with open("/proc/self/task/%%s/stat" %% t) as f:
            v = f.read().rsplit(")", 1)[1].split()
        total += int(v[11]) + int(v[12])
    return total / os.sysconf("SC_CLK_TCK")

def create():
    try:
        pkg.native.Problem(prob, device=0).close()
    except pkg.native.SgbaError:
        pass  # no GPU: the plan was built

before = set(os.listdir("/proc/self/task"))
create()
workers = set(os.listdir("/proc/self/task")) - before
inside, own = threading.Barrier(3), []

def loop():
    inside.wait()
    for _ in range(8):
        create()
    own.append(time.thread_time())

w0 = cpu(workers)
threads = [threading.Thread(target=loop) for _ in range(3)]
for t in threads:
    t.start()
for t in threads:
    t.join()
print(len(workers), cpu(workers) - w0, sum(own))
"""


@pytest.mark.skipif((os.cpu_count() or 1) < 6, reason="needs cores to spare beside three creations")
def test_workers_run_beside_three_creations(pkg):
    out = subprocess.run([sys.executable, "-c", _RUN % ROOT], capture_output=True, text=True, check=True).stdout.split()
    n, busy, callers = int(out[0]), float(out[1]), float(out[2])
    assert n > 0
    # one region at a time has every worker: a third of the work or more where
    # three creations take turns; next to nothing where the pool is left asleep
    assert busy > 0.25 * callers, (busy, callers)
