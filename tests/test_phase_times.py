"""Times of the mixed per-phase kernels, against each other on the same GPU (the
smallest of several phase-timed runs).

A box of 2.05 M hexahedra: node update / elements, bar 1.10. It is 1.06; 1.13 when
the thermal gather stood in the common node kernel and prescribed velocities were
loaded ahead of the arithmetic. A renumbered mesh of 729,000, read through the
connectivity: geometry / node update, bar 0.42. It is 0.40; 0.44 with the additions
packed in pairs, for which those kernels have no registers."""
import pytest

import weldformfem_gb300 as wf
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def phases(n, renumbered):
    c = W.config(0, scale=n)
    c.perturb, c.top_vz = 0.1, -0.02
    d = wf.Domain(wf.WF_MIXED)
    x = c.coords()
    d.set_mesh(x, c.elnod()[::-1].copy() if renumbered else c.elnod())
    W.apply_options(d, c, x=x)
    d.set_step_mode(1)
    d.set_phase_timing(True)
    d.init()
    best = None
    for _ in range(8):
        d.run(40)
        d.sync()
        ms, steps = d.phase_times()
        t = ms / steps
        best = t if best is None else [min(a, b) for a, b in zip(best, t)]
    return dict(zip(("geometry", "nodal", "elements", "nodes"), best))


def test_node_update_of_a_box():
    t = phases((160, 160, 80), False)
    assert t["nodes"] <= 1.10 * t["elements"], t


def test_geometry_through_the_connectivity():
    t = phases((90, 90, 90), True)
    assert t["geometry"] <= 0.42 * t["nodes"], t
