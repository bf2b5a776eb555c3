"""Batches of box meshes take corners and node lists from each specimen's box
(mixed precision). Nothing of the arithmetic changes, so the run equals bit for
bit the one that reads the arrays, whatever the specimens' dimensions; a batch
with one specimen in another numbering reads the arrays throughout."""
import numpy as np
import pytest

import weldformfem_gb300 as wf
from weldformfem_gb300 import workloads as W

STEPS = 40


def batch(dims, swap=None):
    """The assembled batch: one block of `dims[i]` hexahedra per specimen, pulled
    at the top; `swap` renumbers two nodes of that specimen."""
    xs, els, eoff, noff, fixed, top = [], [], [0], [0], [], []
    for i, (nx, ny, nz) in enumerate(dims):
        el = W.box_elnod((nx, ny, nz), False).astype(np.int32)
        k, j, a = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1),
                              indexing="ij")
        x = np.stack([1e-3 * a.ravel(), 1.1e-3 * j.ravel(), 0.9e-3 * k.ravel()], axis=1)
        z = x[:, 2].copy()
        if swap == i:
            a, b = 1, len(x) - 2
            el = el.copy()
            x[[a, b]] = x[[b, a]]
            z[[a, b]] = z[[b, a]]
            ia, ib = el == a, el == b
            el[ia], el[ib] = b, a
        fixed += list(noff[-1] + np.where(z < 1e-9)[0])
        top += list(noff[-1] + np.where(z > 0.9e-3 * nz - 1e-9)[0])
        xs.append(x)
        els.append(el + noff[-1])
        eoff.append(eoff[-1] + len(el))
        noff.append(noff[-1] + len(x))
    return np.concatenate(xs), np.concatenate(els).astype(np.int32), eoff, noff, fixed, top


def run(b, box):
    x, el, eoff, noff, fixed, top = b
    ns = len(eoff) - 1
    d = wf.Domain(wf.WF_MIXED)
    d.set_mesh(x, el)
    mats = [dict(model=0, E=200e9 * (1 + 0.05 * k), nu=0.3, rho=7850.0, sy0=300e6, H=1e9)
            for k in range(ns)]
    emat = np.repeat(np.arange(ns, dtype=np.int32), np.diff(eoff))
    d.set_materials(mats, emat)
    d.add_bcs([(int(n), k, 0.0) for n in fixed for k in range(3)]
              + [(int(n), 2, -8.0) for n in top])
    d.set_reaction_nodes(np.array(top, dtype=np.int64), 2)
    d.set_specimens(eoff, noff, np.linspace(4e-8, 6e-8, ns))
    d.set_box_indexing(box)
    d.init()
    d.run(STEPS)
    return ([d.node_vec("u"), d.node_vec("v"), d.elem_scalar("pl_strain")]
            + [d.specimen_reaction(k) for k in range(ns)])


@pytest.mark.gpu
@pytest.mark.parametrize("dims,swap", [
    ([(1, 1, 1)], None),
    ([(1, 1, 1), (1, 1, 7), (9, 1, 1), (1, 6, 2)], None),
    ([(5, 4, 3), (8, 8, 8), (33, 2, 5), (7, 13, 11)], None),
    ([(5, 4, 3), (6, 5, 4), (3, 3, 3)], 1),
])
def test_specimen_boxes_equal_the_arrays(dims, swap):
    b = batch(dims, swap)
    for got, want in zip(run(b, True), run(b, False)):
        assert np.isfinite(want).all()
        np.testing.assert_array_equal(got, want)
