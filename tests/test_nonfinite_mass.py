"""Lumped masses of tetrahedra whose volume has overflowed: the FP64 step forms
x / c from a reciprocal and a remainder, and keeps the reference's infinity there
(an infinite mass holds its node; a NaN would spread). One node of a block is
carried off at 1e300 m/s; masses, volumes and accelerations against the oracle."""
import numpy as np
import pytest

import weldformfem_gb300 as wf
from oracle import orabind as O
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def run(dom, corner):
    el = W.box_elnod((2, 2, 1), True).astype(np.int32)
    k, j, i = np.meshgrid(np.arange(2), np.arange(3), np.arange(3), indexing="ij")
    x = 1e5 * np.stack([i.ravel(), j.ravel(), k.ravel()], axis=1).astype(float)
    dom.set_mesh(x, el)
    dom.set_materials([dict(model=0, E=200e9, nu=0.3, rho=7850.0, sy0=300e6, H=1e9)])
    dom.add_bcs([(corner, 2, 1e300)])
    dom.set_dt(1.0)
    dom.init()
    dom.step(2)
    return dom.node_scalar("mass"), dom.elem_scalar("vol"), dom.node_vec("a")


@pytest.mark.parametrize("corner", [9, 13, 17])
def test_infinite_volume(corner):
    got, want = run(wf.Domain(wf.WF_FP64), corner), run(O.OracleDomain(), corner)
    assert np.isinf(want[0]).any()
    for g, w in zip(got, want):
        np.testing.assert_array_equal(np.isnan(g), np.isnan(w))
        np.testing.assert_array_equal(np.isinf(g), np.isinf(w))
    assert np.array_equal(got[0], want[0], equal_nan=True)
