"""The FP64 hexahedron kernels against the oracle where they can go wrong: block
edges (1, 31, 32, 33, 127, 128, 129 elements), element volumes inside and
outside the range of the fast two-thirds power, several densities around a node
(lumped-mass shares), and the halo forces of the step halves.

Tolerance 1e-9 of the largest value, 1e-7 for accelerations (the FP64 step's
stated bar, tests/test_parity_fp64.py): the kernel forms the reference's
quantities in another order in FP64, about 1e-15 per operation."""
import numpy as np
import pytest

import weldformfem_gb300 as wf
from oracle import orabind as O
from tests import helpers as H
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def case(n, h, speed=-15.0):
    c = W.Case("box", L=tuple((k + 0.25) * h for k in n), r=h / 2, perturb=0.1,
               seed=W.SEED_BASE + sum(n), hg=0.1, top_vz=speed)
    return c


@pytest.mark.parametrize("n,h", [((1, 1, 1), 1e-3), ((31, 1, 1), 1e-3), ((4, 4, 2), 1e-3),
                                 ((11, 3, 1), 1e-3), ((127, 1, 1), 1e-3), ((8, 4, 4), 1e-3),
                                 ((3, 43, 1), 1e-3),
                                 # volumes 8e-33 (below the fast power's range) and 1e6
                                 ((3, 4, 5), 2e-11), ((3, 4, 5), 1e2)])
def test_hex_step_matches_oracle(n, h):
    c = case(n, h)
    assert c.nel == n
    d, o = wf.Domain(wf.WF_FP64), O.OracleDomain()
    for dom in (d, o):
        W.apply(dom, c)
        dom.init()
        dom.step(60)
    assert d.elem_scalar("pl_strain").max() > 0.0
    for k, v in H.compare_state(d, o).items():
        assert v <= (1e-7 if k in ("a", "fi") else 1e-9), (k, v)
    assert H.rel_err(d.reaction(), o.reaction()) <= 1e-9


def test_halo_forces_are_the_element_forces_of_each_element():
    """Per element and local node: the forces of all elements, added at the
    nodes with the hourglass forces subtracted, are the assembled force."""
    c = case((5, 4, 3), 1e-3)
    d = wf.Domain(wf.WF_FP64)
    W.apply(d, c)
    d.init()
    d.run(20)
    d.step_begin()
    f = d.halo_forces(0, d.ne).reshape(2, d.ne, 8, 3)
    part = d.halo_forces(7, 19).reshape(2, 12, 8, 3)
    np.testing.assert_array_equal(part, f[:, 7:19])
    d.set_halo_forces(7, 19, part)
    np.testing.assert_array_equal(d.halo_forces(0, d.ne).reshape(f.shape), f)
    d.step_end()
    el = d.conn()[0]
    fi = np.zeros((d.nn, 3))
    np.add.at(fi, el.reshape(-1), (f[0] - f[1]).reshape(-1, 3))
    assert H.rel_err(fi, d.node_vec("fi")) <= 1e-12
