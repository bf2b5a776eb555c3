"""The FP64 triangle-mesh contact search on the GPU against the oracle at the
edges of its chunks of 64 triangles (2, 50, 72, 128 and 162 triangles), with
several triangles within one warp's nodes, with the part and the die away from
the origin (the search works relative to the die's first node), and with a
candidate-node list beside the surface. The search decides in FP64, so the
FP64 bar holds: 1e-9 of the largest value."""
import numpy as np
import pytest

import weldformfem_gb300 as wf
from oracle import orabind as O
from tests import helpers as H
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dens,shift", [(1, 0.0), (5, 0.0), (6, 0.0), (8, 0.0), (9, 0.0),
                                        (6, 2.0), (9, -0.7)])
@pytest.mark.parametrize("hexes", [False, True])
def test_contact_search_matches_oracle(hexes, dens, shift):
    c = W.config(0, scale=(7, 5, 4)) if hexes else W.config(1, scale=(5, 4, 3))
    c.perturb, c.seed, c.bc = 0.1, W.SEED_BASE + dens, "bottom_z"
    x, el = c.coords() + shift, c.elnod()
    top = float(x[:, 2].max())
    xyz, tri = W.axis_plane_mesh((shift - 0.00103, shift - 0.00097, top - 1e-5),
                                 (shift + 0.01, 0.0, 0.0), dens, flip_normals=True)
    doms = (wf.Domain(wf.WF_FP64), O.OracleDomain())
    for d in doms:
        d.set_mesh(x, el)
        W.apply_options(d, c, x=x)
        d.set_contact_trimesh(xyz, tri, [0.0, 0.0, -5.0], 0.1, 0.08, 0.1)
        d.set_end_time(1e-5)
        d.init()
        d.step(120)
    d, o = doms
    assert o.reaction().max() > 0.0
    for f in ("u", "v", "contforce"):
        assert H.rel_err(d.node_vec(f), o.node_vec(f)) <= 1e-9, f
    assert H.rel_err(d.reaction(), o.reaction()) <= 1e-9
    assert H.rel_err(d.trimesh_nodes(), o.trimesh_nodes()) <= 1e-12
