"""Two domains of different size stepped and initialised by two host threads: the
library binds a handle to one thread at a time, not the process. The kernels with
dynamic shared memory are shared by the domains; each thread's launches must find
their limit whatever the other asks for. Every state is bitwise that of the same
domain run alone, per phase."""
import threading

import numpy as np
import pytest

import weldformfem_gb300 as wf
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu

INITS, RUNS, STEPS = 150, 8, 2


def domain(n, mode):
    c = W.config(0, scale=n)
    c.perturb, c.top_vz = 0.1, -0.1
    d = wf.Domain(wf.WF_MIXED)
    W.apply(d, c)
    d.set_step_mode(mode)
    d.init()
    return d


# pairs of one kernel with different shared memory: cluster runs of 256-thread
# blocks, tile runs; and one of each
@pytest.mark.parametrize("big,small", [((15, 15, 15), (14, 13, 13)), ((61, 47, 53), (20, 20, 20)),
                                       ((15, 15, 15), (31, 30, 29))])
def test_launches_of_two_threads(big, small):
    errors, done, count = [], threading.Event(), [0]

    def stepping(d):
        try:
            while not done.is_set():
                for _ in range(10):
                    d.run(STEPS)
                    count[0] += STEPS
                d.sync()
        except Exception as e:   # reported by the test's own thread
            errors.append(repr(e))

    def initialising(d):
        try:
            for _ in range(INITS):
                d.init()
                for _ in range(RUNS):
                    d.run(STEPS)
                d.sync()
        except Exception as e:
            errors.append(repr(e))
        done.set()

    a, b = domain(big, 0), domain(small, 0)
    threads = [threading.Thread(target=stepping, args=(a,)),
               threading.Thread(target=initialising, args=(b,))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for d, n, steps in ((a, big, count[0]), (b, small, RUNS * STEPS)):
        want = domain(n, 1)
        want.run(steps)
        want.sync()
        for f in ("x", "v"):
            np.testing.assert_array_equal(d.node_vec(f), want.node_vec(f), err_msg=f)
