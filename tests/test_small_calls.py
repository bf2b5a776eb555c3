"""Small calls beside the step: what a driver makes once per step or per specimen.
Each is bounded by a plain readback on the same domain, whose cost is the copy and
the synchronisation that any such call has (medians of many)."""
import time

import numpy as np
import pytest

import weldformfem_gb300 as wf
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def median(f, n=60):
    t = []
    for _ in range(n):
        a = time.perf_counter()
        f()
        t.append(time.perf_counter() - a)
    return sorted(t)[n // 2]


@pytest.mark.parametrize("prec", [wf.WF_FP64, wf.WF_MIXED])
def test_specimen_reactions(prec):
    """A short history's reaction costs about what a domain's does (0.92; 1.24 to 1.36
    when every call gathered the specimen's column on the device); long and short ones
    are the same values."""
    b = W.ensemble(n_spec=8, nmin=4, nmax=6)
    d = wf.Domain(prec)
    W.apply_batch(d, b)
    d.init()
    d.run(40)
    d.sync()
    one = wf.Domain(prec)
    W.apply(one, W.config(0, scale=(4, 4, 4)))
    one.init()
    one.run(40)
    one.sync()
    assert median(lambda: d.specimen_reaction(3)) <= 1.2 * median(one.reaction)
    short = [d.specimen_reaction(k) for k in range(8)]
    assert all(np.abs(r).max() > 0 for r in short)
    d.run(8300)                             # past 65,536 values: gathered on the device
    for k in range(8):
        long = d.specimen_reaction(k)
        assert long.shape == (8340,)
        np.testing.assert_array_equal(long[:40], short[k])


def test_halo_forces_of_a_small_layer():
    """A layer of 100 hexahedra costs what a reaction readback does, 0.85 to 0.95 of it
    in each direction (the caller's order is made on the device; with scratch from the
    pool and a launch per array it was 1.47 to 1.60)."""
    d = wf.Domain(wf.WF_FP64)
    W.apply(d, W.config(0, scale=(10, 10, 10)))
    d.init()
    d.run(3)
    d.sync()
    plain = median(d.reaction, 100)
    d.step_begin()
    buf = np.zeros(2 * 100 * 24)
    for call in ("wf_get_halo_forces", "wf_set_halo_forces"):
        t = median(lambda: d._call(call, 100, 200, buf), 100)
        assert t <= 1.45 * plain, (call, t, plain)


@pytest.mark.parametrize("prec", [wf.WF_FP64, wf.WF_MIXED])
def test_detj_of_tetrahedra(prec):
    """detJ is formed at the call: 1.33 to 1.35 times a plain field of 576,000 tetrahedra
    (1.55 to 1.59 when the geometry kernel formed the step's adjugates for it as
    well), bar 1.47."""
    d = wf.Domain(prec)
    W.apply(d, W.config(1))
    d.init()
    d.run(2)
    vol = median(lambda: d.elem_scalar("vol"), 80)
    assert median(lambda: d.elem_scalar("detJ"), 80) <= 1.47 * vol
