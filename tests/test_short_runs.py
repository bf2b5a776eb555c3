"""Runs of a few steps, as a driver makes them that looks at its results after
every step or two: the automatic mode is not behind the per-phase kernels that it
stands for (step mode 1). Both sides are timed in turn on the same GPU, the
smallest of several repetitions each; bar 1.15 (they are 0.7 to 1.03 of each other;
before their set-up and the reaction's sum were mended, tile runs were at 1.2 to
1.5 for one step)."""
import time

import pytest

import weldformfem_gb300 as wf
from tests import helpers as H
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def domain(n, mode, extra, die):
    c = W.config(2 if die else 0, scale=n)
    c.perturb, c.top_vz = 0.1, -0.02
    if die:
        c.contact["v"] = 0.2
    d = wf.Domain(wf.WF_MIXED)
    H.setup(d, c, extra)
    d.set_step_mode(mode)
    d.init()
    return d


def per_run(d, k, runs=150):
    t = time.perf_counter()
    for _ in range(runs):
        d.run(k)
    d.sync()
    return (time.perf_counter() - t) / runs


TH = dict(thermal=dict(T0=300.0, k=40.0, cp=450.0, exp=1.1e-5))


@pytest.mark.parametrize("n,extra,die", [((20, 20, 20), {}, False), ((30, 30, 30), {}, False),
                                         ((61, 47, 53), {}, True), ((33, 40, 27), TH, False)])
@pytest.mark.parametrize("k", [1, 2, 4])
def test_not_behind_the_phases(n, extra, die, k):
    auto, phases = domain(n, 0, extra, die), domain(n, 1, extra, die)
    best = {0: 1e9, 1: 1e9}
    for d in (auto, phases):
        d.prepare_run(k)
        per_run(d, k)
    for _ in range(7):
        for i, d in ((0, auto), (1, phases)):
            best[i] = min(best[i], per_run(d, k))
    assert best[0] <= 1.15 * best[1], (best[0] * 1e6, best[1] * 1e6)
