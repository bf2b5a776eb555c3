"""Which kernels a run launches and how the mixed kernels index the mesh, on both
sides of every limit. wf_get_step_mode names the arithmetic; these are the
kernels."""
import numpy as np
import pytest

import weldformfem_gb300 as wf
from tests import helpers as H
from tests import test_node_lists as NL
from tests import test_specimen_box as SB
from weldformfem_gb300 import workloads as W

pytestmark = pytest.mark.gpu

TH = dict(thermal=dict(T0=300.0, k=40.0, cp=450.0, exp=1.1e-5))
LONG = 1000


def domain(n, prec=wf.WF_MIXED, cid=0, mode=0, extra=None, energy=False, renumber=False):
    c = W.config(cid, scale=n)
    d = wf.Domain(prec)
    if renumber:
        x = c.coords()
        d.set_mesh(x, c.elnod()[::-1].copy())
        W.apply_options(d, c, x=x)
    else:
        H.setup(d, c, extra or {})
    if energy:
        d.set_energy_history(True)
    d.set_step_mode(mode)
    d.init()
    return d


def test_automatic_choice():
    for n, kernels in (((10, 10, 10), "cluster_smem"),      # at most 3000 hexahedra
                       ((15, 20, 10), "cluster_smem"),
                       ((19, 19, 19), "tile_run"), ((61, 47, 53), "tile_run"),
                       ((80, 80, 80), "phases"),            # past the SMs' shared memory
                       ((256, 256, 4), "sweep")):
        d = domain(n)
        assert d.run_kernels(LONG) == kernels, n
    assert domain((10, 10, 10), energy=True).run_kernels(LONG) == "phases"
    assert domain((20, 20, 20), energy=True).run_kernels(LONG) == "phases"
    assert domain((20, 20, 20), prec=wf.WF_FP64).run_kernels(LONG) == "phases"
    assert domain((20, 20, 20), renumber=True).run_kernels(LONG) == "phases"
    assert domain((8, 8, 8), cid=1).run_kernels(LONG) == "phases"     # 3072 tetrahedra
    assert domain((7, 7, 7), cid=1).run_kernels(LONG) == "cluster"    # 2058
    # heat: through L2 for small meshes, tiles to two passes of the elements
    assert domain((10, 10, 10), extra=TH).run_kernels(LONG) == "cluster"
    assert domain((33, 40, 27), extra=TH).run_kernels(LONG) == "tile_run"
    assert domain((62, 60, 60), extra=TH).run_kernels(LONG) == "phases"


def test_a_chosen_mode_is_what_runs():
    d = domain((20, 20, 20))
    for mode, kernels in ((1, "phases"), (2, "cluster"), (4, "sweep"), (5, "flow"), (0, "tile_run")):
        d.set_step_mode(mode)
        assert d.run_kernels(LONG) == kernels
    assert domain((10, 10, 10), mode=3).run_kernels(LONG) == "tiled"
    d.set_phase_timing(True)
    assert d.run_kernels(LONG) == "phases"


def test_calls_that_are_refused():
    d = wf.Domain(wf.WF_MIXED)
    for call in (lambda: d.run_kernels(1), d.index_tables):
        with pytest.raises(wf.WfError) as e:
            call()
        assert e.value.status == wf.WF_ERR_STATE
    d = domain((3, 3, 3))
    with pytest.raises(wf.WfError) as e:
        d.run_kernels(-1)
    assert e.value.status == wf.WF_ERR_ARG


def tets(n, fan):
    x, el = NL.block(n)
    if fan:
        fx, fe = NL.fan()
        x, el = np.concatenate([x, fx]), np.concatenate([el, fe + len(x)])
    d = wf.Domain(wf.WF_MIXED)
    d.set_mesh(x, el)
    d.set_materials([dict(model=0, E=200e9, nu=0.3, rho=7850.0, sy0=300e6, H=1e9)])
    d.set_dt(2e-8)
    d.init()
    return d


def test_lists_by_position():
    for n in ((20, 20, 22), (3, 5, 341)):
        assert 8 <= tets(n, False).index_tables()[0] <= 64
        assert tets(n, True).index_tables()[0] == 0        # a list of 80 entries
    assert tets((5, 5, 5), False).index_tables()[0] == 0   # below 8192 nodes
    assert domain((20, 20, 20)).index_tables() == (0, False)


@pytest.mark.parametrize("dims,swap,on", [([(5, 4, 3), (8, 8, 8)], None, True),
                                          ([(1, 1, 1)], None, True),
                                          ([(5, 4, 3), (6, 5, 4)], 1, False)])
def test_specimen_boxes(dims, swap, on):
    x, el, eoff, noff, _, _ = SB.batch(dims, swap)
    for box in (True, False):
        d = wf.Domain(wf.WF_MIXED)
        d.set_mesh(x, el)
        d.set_materials([dict(model=0, E=200e9, nu=0.3, rho=7850.0, sy0=300e6, H=1e9)])
        d.set_specimens(eoff, noff, np.full(len(dims), 4e-8))
        d.set_box_indexing(box)
        d.init()
        assert d.index_tables() == (0, on and box)
        assert d.run_kernels(LONG) == "phases"
