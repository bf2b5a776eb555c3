"""Device memory of an FP64 domain: the step's scratch is the element and hourglass
forces, and what the geometry phase leaves for the element phase lies in those.
Bytes an element of a block of 96^3 hexahedra (1027; 1102 with an array of its own for
the adjugates) and of tetrahedra (470; 528), in a process of its own. And a read-back of detJ, which runs the geometry kernel, leaves the element
forces of the step as they were."""
import os
import subprocess
import sys

import numpy as np
import pytest

import weldformfem_gb300 as wf
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
import torch
import weldformfem_gb300 as wf
from weldformfem_gb300 import workloads as W
c = W.config({cid}, scale={n})
w = wf.Domain(wf.WF_FP64)
W.apply(w, W.config({cid}, scale=(2, 2, 2)))
w.init()
w.sync()
before = torch.cuda.mem_get_info()[0]
d = wf.Domain(wf.WF_FP64)
W.apply(d, c)
d.init()
d.run(2)
d.sync()
print((before - torch.cuda.mem_get_info()[0]) / c.n_elem)
"""


@pytest.mark.parametrize("cid,n,most", [(0, (96, 96, 96), 1060.0), (1, (40, 40, 60), 500.0)])
def test_bytes_an_element(cid, n, most):
    r = subprocess.run([sys.executable, "-c", SRC.format(cid=cid, n=n)], cwd=ROOT,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert float(r.stdout.split()[-1]) <= most


@pytest.mark.parametrize("cid", [0, 1])
def test_detj_leaves_the_forces(cid):
    c = W.config(cid, scale=(5, 4, 3))
    d = wf.Domain(wf.WF_FP64)
    W.apply(d, c)
    d.init()
    assert not d.halo_forces(0, d.ne).any()     # no step yet
    d.elem_scalar("detJ")
    assert not d.halo_forces(0, d.ne).any()
    d.run(30)
    f = d.halo_forces(0, d.ne)
    assert np.abs(f).max() > 0
    detj = d.elem_scalar("detJ")
    np.testing.assert_array_equal(d.halo_forces(0, d.ne), f)
    assert (detj > 0).all()
