"""Tile runs: the automatic mode runs box meshes between the cluster run's size
and the SMs' shared memory as one cooperative launch per 256 steps (reported as
mode 1, whose arithmetic it runs). The state is bitwise that of step mode 1,
across chunks and runs of odd length; the reaction is summed in another order
(FP64 sums of FP32 contributions), 1e-12 relative. Boxes: just above the limit,
flat, long and ragged ones (tiles of one element in a direction, tiles at every
face), with the die, Johnson-Cook, heat and one mass per run."""
import numpy as np
import pytest

import weldformfem_gb300 as wf
from tests import helpers as H
from tests.test_thermal import JC
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def box(n, die=False):
    c = W.config(2 if die else 0, scale=n)
    c.perturb, c.top_vz = 0.1, -15.0
    if die:
        c.contact["v"] = 15.0
    assert c.nel == n and c.n_elem > 6500
    return c


def cases():
    jc = box((21, 20, 17))
    jc.materials = [dict(model=2, E=200e9, nu=0.3, rho=7850.0, sy0=250e6)]
    warm = box((19, 21, 18))
    two = box((17, 23, 19))
    two.materials = [dict(W.STEEL), dict(W.STEEL, sy0=200e6)]
    two.elem_mat = (np.arange(two.n_elem) % 2).astype(np.int32)
    two.mass_mode = 1
    th = dict(T0=300.0, k=40.0, cp=450.0, exp=1.1e-5)
    return {"cube": (box((19, 19, 19)), {}, 300), "flat": (box((67, 53, 2)), {}, 60),
            "long": (box((3, 7, 401)), {}, 60), "thin": (box((1, 97, 71)), {}, 60),
            "die": (box((31, 23, 29), True), {}, 257), "die_flat": (box((83, 81, 1), True), {}, 60),
            "big": (box((61, 47, 53), True), {}, 40), "jc_thermal": (jc, dict(jc=JC, thermal=th), 130),
            "thermal": (warm, dict(thermal=th), 60), "two_masses": (two, {}, 60)}


@pytest.mark.parametrize("name", list(cases()))
def test_tile_run_matches_per_phase_kernels(name):
    case, extra, steps = cases()[name]
    doms = []
    for mode in (1, 0):
        d = wf.Domain(wf.WF_MIXED)
        H.setup(d, case, extra)
        d.set_step_mode(mode)
        d.init()
        d.run(steps - 1)
        d.run(1)
        d.sync()
        doms.append(d)
    a, b = doms
    assert b.step_mode()[0] == 1
    assert a.graph_launches() > 0 and b.graph_launches() == 0
    assert b.launch_count() == 2 + -(-(steps - 1) // 256) + 1   # predictors, chunks
    for f in ("x", "u", "v", "a", "contforce"):
        np.testing.assert_array_equal(b.node_vec(f), a.node_vec(f), err_msg=f)
    np.testing.assert_array_equal(b.node_scalar("mass"), a.node_scalar("mass"))
    for f in ("pl_strain", "vol", "p"):
        np.testing.assert_array_equal(b.elem_scalar(f), a.elem_scalar(f), err_msg=f)
    np.testing.assert_array_equal(b.elem_tensor("tau"), a.elem_tensor("tau"))
    if "thermal" in extra:
        np.testing.assert_array_equal(b.node_scalar("T"), a.node_scalar("T"))
    ra, rb = a.reaction(), b.reaction()
    assert ra.shape == rb.shape == (steps,) and np.abs(ra).max() > 0
    assert H.rel_err(rb, ra) <= 1e-12
