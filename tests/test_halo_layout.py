"""FP64 halo forces: the caller's order is element by element, the device's row by
row. Ranges of every kind cross unchanged in both directions, with and without
hourglass forces; tetrahedra as well. And they cross at the speed of a copy: a
layer of 128 x 128 hexahedra, 6.3 MB, took 0.06 ms before the device order
changed, 1.1 ms when the host put the rows into order."""
import time

import numpy as np
import pytest

import weldformfem_gb300 as wf
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cid,n,hg", [(0, (7, 5, 3), 0.1), (0, (7, 5, 3), 0.0), (1, (3, 3, 2), 0.0)])
def test_ranges_cross_unchanged(cid, n, hg):
    c = W.config(cid, scale=n)
    c.perturb = 0.1
    d = wf.Domain(wf.WF_FP64)
    W.apply(d, c)
    d.set_hourglass(hg)
    d.init()
    d.run(15)
    d.step_begin()
    w = 3 * d.npe
    full = d.halo_forces(0, d.ne).reshape(2, d.ne, w)
    assert np.abs(full[0]).max() > 0 and (np.abs(full[1]).max() > 0) == (hg > 0 and d.npe == 8)
    rng = np.random.default_rng(W.SEED_BASE)
    for e0, e1 in ((0, 1), (d.ne - 1, d.ne), (4, 4), (3, 36), (0, d.ne)):
        np.testing.assert_array_equal(d.halo_forces(e0, e1).reshape(2, e1 - e0, w), full[:, e0:e1])
        new = rng.standard_normal((2, e1 - e0, w))
        if not full[1].any():
            new[1] = 0.0
        d.set_halo_forces(e0, e1, new)
        full[:, e0:e1] = new
        np.testing.assert_array_equal(d.halo_forces(0, d.ne).reshape(2, d.ne, w), full)


def test_a_layer_crosses_at_the_speed_of_a_copy():
    d = wf.Domain(wf.WF_FP64)
    W.apply(d, W.config(0, scale=(128, 128, 4)))
    d.init()
    d.step_begin()
    m = 128 * 128
    buf = np.zeros(2 * m * 24)
    for call in ("wf_get_halo_forces", "wf_set_halo_forces"):
        t = []
        for _ in range(25):
            a = time.perf_counter()
            d._call(call, m, 2 * m, buf)
            t.append(time.perf_counter() - a)
        assert sorted(t)[12] < 5e-4, (call, sorted(t)[12])
