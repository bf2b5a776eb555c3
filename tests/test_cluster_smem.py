"""Cluster runs with the state in shared memory (hexahedra) against the per-phase
kernels, bit for bit, where their setup can go wrong: one block and every cluster
size, blocks of uneven length, meshes whose numbering scatters a block's nodes
over all blocks, launch chunks of 1024 steps and their remainders, and sizes
around the three block sizes. The reaction sums run in another order (FP64 sums
of FP32 contributions): 1e-12."""

import numpy as np
import pytest

import weldformfem_gb300 as wf
from tests import helpers as H
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu

def compare(setup, runs):
    doms = []
    for mode in (1, 2):
        d = wf.Domain(wf.WF_MIXED)
        setup(d)
        d.set_step_mode(mode)
        d.init()
        for n in runs:
            d.run(n)
        d.sync()
        assert d.step_mode()[0] == mode
        doms.append(d)
    a, b = doms
    for f in ("x", "u", "v", "a", "contforce"):
        np.testing.assert_array_equal(b.node_vec(f), a.node_vec(f), err_msg=f)
    np.testing.assert_array_equal(b.node_scalar("mass"), a.node_scalar("mass"))
    for f in ("pl_strain", "vol", "p"):
        np.testing.assert_array_equal(b.elem_scalar(f), a.elem_scalar(f), err_msg=f)
    np.testing.assert_array_equal(b.elem_tensor("tau"), a.elem_tensor("tau"))
    ra, rb = a.reaction(), b.reaction()
    assert ra.shape == rb.shape == (sum(runs),) and np.abs(ra).max() > 0
    assert H.rel_err(rb, ra) <= 1e-12

@pytest.mark.parametrize("n", [(1, 1, 1), (3, 3, 3), (5, 5, 3), (7, 5, 4), (9, 7, 5), (13, 11, 7),
                               (16, 16, 8), (23, 13, 10)])
@pytest.mark.parametrize("die", [False, True])
def test_sizes(n, die):
    c = W.config(2 if die else 0, scale=n)
    c.perturb, c.top_vz = 0.1, -15.0
    if die:
        c.contact["v"] = 15.0
    compare(lambda d: W.apply(d, c), (70, 1, 130))

def test_scattered_numbering():
    c = W.config(0, scale=(11, 9, 8))
    c.perturb, c.top_vz = 0.1, -15.0
    rng = np.random.default_rng(W.SEED_BASE + 5)
    perm = rng.permutation(c.n_node)
    x = np.empty((c.n_node, 3))
    x[perm] = c.coords()
    el = perm[c.elnod()][rng.permutation(c.n_elem)].astype(np.int32)
    nodes, dims, vals = c.bcs()

    def setup(d):
        d.set_mesh(x, el)
        d.set_materials(c.materials)
        d.add_bcs((perm[nodes], dims, vals))
        d.set_hourglass(0.1)
        d.set_reaction_nodes(perm[c.top_nodes()].astype(np.int32), 2)
        d.set_dt(c.time_step(c.coords()))

    compare(setup, (200,))

def test_chunks():
    c = W.config(0, scale=(4, 4, 4))
    compare(lambda d: W.apply(d, c), (1023, 1024, 1025, 2050))
