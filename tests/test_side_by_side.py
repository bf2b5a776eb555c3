"""Domains stepped side by side by threads of their own. Small boxes' tile runs leave
SMs to each other: four domains take little longer than one (bar 2: they take 1.05
to 1.1 times one domain's time, four times when every launch took all SMs). Each state
is bitwise that of the domain run alone, per phase."""
import threading
import time

import numpy as np
import pytest

import weldformfem_gb300 as wf
from tests import helpers as H
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu

STEPS = 1000
TH = dict(thermal=dict(T0=300.0, k=40.0, cp=450.0, exp=1.1e-5))


def domain(n, extra, mode, k):
    c = W.config(0, scale=n)
    c.perturb, c.top_vz, c.seed = 0.1, -0.1, W.SEED_BASE + k
    d = wf.Domain(wf.WF_MIXED)
    H.setup(d, c, extra)
    d.set_step_mode(mode)
    d.init()
    return d


def together(doms):
    def go(d):
        d.run(STEPS)
        d.sync()

    threads = [threading.Thread(target=go, args=(d,)) for d in doms]
    t = time.perf_counter()
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    return time.perf_counter() - t


@pytest.mark.parametrize("n,extra", [((16, 16, 16), {}), ((18, 18, 18), {}), ((15, 16, 17), TH)])
def test_small_boxes_share_the_gpu(n, extra):
    doms = [domain(n, extra, 0, k) for k in range(4)]
    assert all(d.run_kernels(STEPS) == "tile_run" for d in doms)
    one, four = 1e9, 1e9
    for _ in range(4):
        four = min(four, together(doms))
    ref = [domain(n, extra, 1, k) for k in range(4)]
    for d in ref:
        d.run(4 * STEPS)
        d.sync()
    for a, b in zip(doms, ref):
        for f in ("x", "v"):
            np.testing.assert_array_equal(a.node_vec(f), b.node_vec(f), err_msg=f)
    for _ in range(4):
        one = min(one, together(doms[:1]))
    assert four <= 2.0 * one, (one, four)
