"""Several large problems created at once still have the host pool's workers: the
share of the creations' CPU time that falls on them.  (Without a GPU a creation
ends after its host plan, which is what is measured here.)"""
import os
import threading
import time

import pytest


def _cpu(tids):
    total = 0
    for t in tids:
        with open("/proc/self/task/%s/stat" % t) as f:
            v = f.read().rsplit(")", 1)[1].split()
        total += int(v[11]) + int(v[12])
    return total


@pytest.mark.skipif((os.cpu_count() or 1) < 6, reason="needs cores to spare beside three creations")
def test_workers_run_beside_three_creations(pkg):
    prob = pkg.synth.generate(pkg.synth.LOOP, n_cam=400, n_pt=60000, seed=pkg.synth.BASE_SEED)

    def create():
        try:
            pkg.native.Problem(prob, device=0).close()
        except pkg.native.SgbaError:
            pass  # no GPU: the plan was built

    before = set(os.listdir("/proc/self/task"))
    create()  # the pool's threads start with the first creation
    workers = set(os.listdir("/proc/self/task")) - before
    assert workers
    inside = threading.Barrier(3)
    own = []

    def loop():
        inside.wait()
        for _ in range(8):
            create()
        own.append(time.thread_time())

    w0, ticks = _cpu(workers), os.sysconf("SC_CLK_TCK")
    threads = [threading.Thread(target=loop) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    busy = (_cpu(workers) - w0) / ticks
    # one region at a time has every worker: a third of the work or more where
    # three creations take turns; next to nothing where the pool is left asleep
    print("workers %.2f s, callers %.2f s" % (busy, sum(own)))
    assert busy > 0.25 * sum(own), (busy, own)
