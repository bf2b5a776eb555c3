"""The cluster run with its state in shared memory: where it is chosen, and its
state bit for bit against the per-phase kernels where a thread takes more than one
element or node (blocks of 256 threads; above 4096 elements or nodes on 16 blocks
every loop has a second pass). Box meshes past 4096 nodes take tile runs, so the
meshes here are renumbered, or mode 2 is asked for."""
import numpy as np
import pytest

import weldformfem_gb300 as wf
from tests import helpers as H
from tests.test_thermal import JC
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def domain(n, mode, die=False, law=False, order=None):
    c = W.config(2 if die else 0, scale=n)
    c.perturb, c.top_vz = 0.1, -15.0
    if die:
        c.contact["v"] = 15.0
    if law:
        c.materials = [dict(model=2, E=200e9, nu=0.3, rho=7850.0, sy0=250e6)]
    d = wf.Domain(wf.WF_MIXED)
    if order is None:
        W.apply(d, c)
    else:
        x, el = c.coords(), c.elnod()
        rng = np.random.default_rng(W.SEED_BASE + 7)
        el = el[::-1].copy() if order == "reversed" else el[rng.permutation(len(el))].copy()
        d.set_mesh(x, el)
        W.apply_options(d, c, x=x)
    if law:
        d.set_johnson_cook(0, *JC)
    d.set_step_mode(mode)
    d.init()
    return d


def compare(a, b):
    for f in ("x", "u", "v", "a", "contforce"):
        np.testing.assert_array_equal(b.node_vec(f), a.node_vec(f), err_msg=f)
    np.testing.assert_array_equal(b.node_scalar("mass"), a.node_scalar("mass"))
    for f in ("pl_strain", "vol", "p"):
        np.testing.assert_array_equal(b.elem_scalar(f), a.elem_scalar(f), err_msg=f)
    np.testing.assert_array_equal(b.elem_tensor("tau"), a.elem_tensor("tau"))
    ra, rb = a.reaction(), b.reaction()
    assert ra.shape == rb.shape and np.abs(ra).max() > 0
    assert H.rel_err(rb, ra) <= 1e-12


@pytest.mark.parametrize("n,mode,opts", [
    ((16, 16, 16), 2, {}), ((17, 17, 16), 0, dict(order="reversed")),
    ((18, 18, 18), 0, dict(order="reversed", die=True)), ((18, 18, 18), 2, dict(law=True)),
    ((24, 18, 15), 0, dict(order="reversed", law=True)), ((15, 15, 15), 0, {}),
    ((15, 15, 15), 0, dict(die=True)), ((11, 14, 21), 0, dict(order="scattered"))])
def test_second_passes_are_the_phases(n, mode, opts):
    a, b = domain(n, 1, **opts), domain(n, mode, **opts)
    assert a.run_kernels(70) == "phases" and b.run_kernels(70) == "cluster_smem"
    for k in (70, 9, 60):
        a.run(k)
        b.run(k)
    for d in (a, b):
        d.sync()
    compare(a, b)


def test_limits():
    for n, mode, order, short, least, long in (
            ((10, 10, 10), 0, None, "cluster", 3, "cluster_smem"),
            ((16, 16, 16), 2, None, "cluster", 3, "cluster_smem"),
            ((15, 15, 15), 0, None, "tile_run", 8, "cluster_smem"),      # 4096 nodes
            ((16, 15, 15), 0, None, "tile_run", 8, "tile_run"),
            ((15, 15, 15), 0, "reversed", "phases", 5, "cluster_smem"),
            ((24, 18, 15), 0, "reversed", "phases", 5, "cluster_smem"),  # 6480
            ((19, 19, 19), 0, "reversed", "phases", 5, "phases")):       # 6859
        d = domain(n, mode, order=order)
        for k in (1, 2, 3, 4, 5, 7, 8, 5000):
            assert d.run_kernels(k) == (short if k < least else long), (n, k)
        assert d.step_mode()[0] == (2 if mode == 2 or d.ne <= 3000 else 1)


def test_one_step_at_a_time():
    """Runs of few steps of a small mesh, which take the other kernels."""
    for n, order in (((9, 8, 7), None), ((15, 15, 15), None), ((16, 16, 16), "reversed")):
        a, b = domain(n, 1, order=order), domain(n, 0, order=order)
        for k in (1, 1, 2, 1, 5, 2, 8, 1, 40, 4, 1):
            a.run(k)
            b.run(k)
            b.sync()
        a.sync()
        compare(a, b)
