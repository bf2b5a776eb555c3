"""Node lists by position. The mixed step keeps the node -> element lists of 8192
nodes of tetrahedra and more by position, unless a list is much longer than the
mean. A block of tetrahedra alone takes them; with a fan of tetrahedra around an
edge beside it (its two axis nodes belong to 80 elements each) the same block
reads the lists laid end to end. Both add the same entries in the same order, so
the block's state is the same bit for bit."""
import numpy as np
import pytest

import weldformfem_gb300 as wf
from weldformfem_gb300 import workloads as W

FAN = 80


def block(n):
    nx, ny, nz = n
    el = W.box_elnod(n, True).astype(np.int32)
    k, j, i = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij")
    x = 1e-3 * np.stack([i.ravel(), 1.1 * j.ravel(), 0.9 * k.ravel()], axis=1)
    return x, el


def fan():
    a = 2 * np.pi * np.arange(FAN) / FAN
    ring = np.stack([0.02 * np.cos(a), 0.02 * np.sin(a), np.full(FAN, 2e-3)], axis=1)
    x = np.concatenate([[[0.0, 0.0, 0.0], [0.0, 0.0, 4e-3]], ring]) + [0.2, 0.0, 0.0]
    r = 2 + np.arange(FAN)
    el = np.stack([np.zeros(FAN), r, 2 + (r - 1) % FAN, np.ones(FAN)], axis=1)
    return x, el.astype(np.int32)


def run(n, with_fan, steps=25):
    x, el = block(n)
    nn, ne = len(x), len(el)
    bottom = np.where(x[:, 2] < 1e-9)[0]
    top = np.where(x[:, 2] > 0.9e-3 * n[2] - 1e-9)[0]
    if with_fan:
        fx, fe = fan()
        v = np.einsum("ij,ij->i", np.cross(fx[fe[:, 1]] - fx[fe[:, 0]], fx[fe[:, 2]] - fx[fe[:, 0]]),
                      fx[fe[:, 3]] - fx[fe[:, 0]])
        assert (v > 0).all() and np.bincount(fe.ravel()).max() == FAN
        x, el = np.concatenate([x, fx]), np.concatenate([el, fe + nn])
    d = wf.Domain(wf.WF_MIXED)
    d.set_mesh(x, el)
    d.set_materials([dict(model=0, E=200e9, nu=0.3, rho=7850.0, sy0=300e6, H=1e9)])
    d.add_bcs([(int(i), k, 0.0) for i in bottom for k in range(3)]
              + [(int(i), 2, -12.0) for i in top])
    d.set_dt(2e-8)
    d.init()
    d.run(steps)
    return ([d.node_vec(f)[:nn] for f in ("x", "u", "v", "a")]
            + [d.elem_scalar("pl_strain")[:ne]])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(20, 20, 22), (3, 5, 341)])
def test_lists_by_position_equal_the_lists(n):
    assert np.prod(np.array(n) + 1) >= 8192
    a, b = run(n, False), run(n, True)
    assert np.abs(a[1]).max() > 0.0
    for got, want in zip(a, b):
        assert np.isfinite(want).all()
        np.testing.assert_array_equal(got, want)
