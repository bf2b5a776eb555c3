"""The work that users of this framework have it do, as cases to be timed.

A pass is what a program does between building its mesh and looking at its
results: wf_init on the described domain (the preamble of the reference's
SolveChungHulbert), a run of explicit steps, and the readback of the fields
into the program's own buffers. Three kinds differ:
  die_mesh  a part under a rigid triangle-mesh die; the domain is initialised
            once and a pass is the next output interval of the run
  solve     one whole call, from host arrays to results, domain included
  adjoint   forward with checkpoints and the gradient of the reaction history

Sizes: the named configurations of weldformfem_gb300.workloads (the 10^3 cube,
the 576,000 tetrahedra, the 256 x 256 x 128 block under a die, the ensemble of
cubes of 6 to 40 elements per edge, the 32^3 octants), scaled blocks between
them and ragged ones. Materials are the workloads' steel, or a Johnson-Cook
steel with heat; tool speeds are those of drop forging (10 to 20 m/s), so the
plastic return runs from the first steps. The seed moves the interior nodes,
the tool speed and the material constants.

The mixed step computes and keeps its fields in 32 bits (the library hands
them out widened to 64); the cases take them as 32-bit arrays, the FP64 step's
as 64-bit ones.
"""
import math
import random

import numpy as np
import torch

import weldformfem_gb300 as wf
from weldformfem_gb300 import workloads as W

STEEL = dict(model=0, E=200e9, nu=0.3, rho=7850.0, sy0=300e6, H=1e9)
# B n C eps0 m Tm Tt T; C ln(rate) stays above -1 at the rates ahead of the first stress wave
JC = [400e6, 0.35, 0.005, 1.0, 1.0, 1500.0, 20.0, 300.0]
RHO_B = 0.8182                                            # Chung-Hulbert spectral radius


def _case(name, kind, prec, nx, ny, nz, steps, **more):
    c = dict(kind=kind, prec=prec, nx=nx, ny=ny, nz=nz, steps=steps, **more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a coupon or one forming cell: the smallest runs, bound by latency
        _case("cube_1k_mixed", "box", "mixed", 10, 10, 10, 1000),
        # the same at the reference's precision
        _case("cube_1k_fp64", "box", "fp64", 10, 10, 10, 200),
        # an ordinary part of odd size under a flat die, production precision
        _case("block_152k_die_mixed", "die", "mixed", 61, 47, 53, 200),
        # the largest: the headline block under a flat die with friction
        _case("block_8m_die_mixed", "die", "mixed", 256, 256, 128, 100),
        # the reference's own element type at its headline size
        _case("tets_576k_mixed", "tets", "mixed", 40, 40, 60, 200),
        # a million hexahedra at the reference's precision
        _case("block_1m_die_fp64", "die", "fp64", 128, 128, 64, 20),
        # a forging: tetrahedra under a triangle-mesh die with friction and heat
        _case("forging_tets_fp64", "die_mesh", "fp64", 20, 20, 30, 60),
        # rate- and temperature-dependent steel with heat conduction, odd size
        _case("jc_thermal_mixed", "thermal", "mixed", 33, 40, 27, 200),
        # an ensemble of specimens in one domain (calibration, sampling)
        _case("ensemble_128_mixed", "ensemble", "mixed", 40, 40, 40, 100, nspec=128),
        # material identification: reaction history and its gradient
        _case("adjoint_32cube_fp64", "adjoint", "fp64", 32, 32, 32, 64),
        # one whole call from host arrays to results
        _case("solve_2m_mixed", "solve", "mixed", 160, 160, 80, 20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the listed kinds over their whole range of sizes."""
    kind = rng.choice(["box", "box", "die", "die", "tets", "die_mesh", "thermal", "ensemble",
                       "adjoint", "solve"])
    prec = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "adjoint":
        n = [_log_int(rng, 6, 36) for _ in range(3)]
        return _case("", kind, "fp64", *n, rng.randint(20, 64))
    if kind == "ensemble":
        return _case("", kind, "mixed", 40, 40, 40, rng.randint(20, 100),
                     nspec=_log_int(rng, 8, 128))
    most = {"box": 4e6, "die": 8e6, "tets": 1e5, "die_mesh": 1.2e4, "thermal": 5e5,
            "solve": 2e6}[kind]
    if prec == "fp64":
        most = min(most, 1e6)
    cells = math.exp(rng.uniform(math.log(300.0), math.log(most)))
    side = cells ** (1.0 / 3.0)
    fx, fy = rng.uniform(0.6, 1.6), rng.uniform(0.6, 1.6)
    n = [max(3, int(side * fx)), max(3, int(side * fy)), max(3, int(side / (fx * fy)))]
    if rng.random() < 0.5:
        n = [v | 1 for v in n]
    cells = n[0] * n[1] * n[2] * (6 if kind in ("tets", "die_mesh") else 1)
    budget = 1.6e7 if prec == "fp64" else 4e8
    steps = int(min(1000 if prec == "mixed" else 200, max(20, budget / cells)))
    if kind == "solve":
        steps = 20
    return _case("", kind, prec, *n, steps)


# ---- inputs --------------------------------------------------------------------


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _box(nx, ny, nz, h, tets, perturb, gen, dev):
    """Box mesh in the AddBoxLength numbering, interior nodes moved by up to
    perturb * h: coordinates [nn, 3] (float64), connectivity (int32), and the
    grid indices of the nodes."""
    ax = [torch.arange(n + 1, device=dev) for n in (nx, ny, nz)]
    kk, jj, ii = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    ii, jj, kk = ii.reshape(-1), jj.reshape(-1), kk.reshape(-1)
    x = torch.stack([ii, jj, kk], 1).to(torch.float64) * h
    inside = ((ii > 0) & (ii < nx) & (jj > 0) & (jj < ny) & (kk > 0) & (kk < nz))
    move = torch.rand(x.shape, generator=gen, device=dev, dtype=torch.float64) * 2.0 - 1.0
    x = x + move * inside[:, None] * (perturb * h)
    ex, ey, ez = (torch.arange(n, device=dev) for n in (nx, ny, nz))
    px, pxy = nx + 1, (nx + 1) * (ny + 1)
    n0 = (ex[None, None, :] + px * ey[None, :, None] + pxy * ez[:, None, None]).reshape(-1)
    off = torch.tensor([0, 1, 1 + px, px, pxy, pxy + 1, pxy + px + 1, pxy + px], device=dev)
    el = n0[:, None] + off[None, :]
    if tets:
        split = torch.tensor([[0, 1, 3, 5], [1, 2, 3, 5], [0, 5, 3, 4], [4, 5, 3, 7],
                              [5, 6, 3, 7], [5, 2, 3, 6]], device=dev)
        el = el[:, split].reshape(-1, 4)
    return x, el.to(torch.int32), (ii, jj, kk)


def _edges(npe):
    if npe == 8:
        return [(0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5),
                (2, 6), (3, 7)]
    return [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]


def _shortest_edge(x, el):
    el = el.long()
    best = math.inf
    for a, b in _edges(el.shape[1]):
        d = x[el[:, b]] - x[el[:, a]]
        best = min(best, float((d * d).sum(1).min().sqrt()))
    return best


def _specimens(nspec):
    """Elements per edge of each specimen, U{6..40}: the case's, not the seed's."""
    r = random.Random(1000 + nspec)
    return [r.randint(6, 40) for _ in range(nspec)]


def _model(case, seed):
    """Everything that describes the inputs of a case, on the device."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 7919 + 17)
    r = random.Random(int(seed))
    kind = case["kind"]
    if kind == "ensemble":
        return _ensemble(case, gen, r, dev)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    tets = kind in ("tets", "die_mesh")
    h = {"tets": 5e-4, "die_mesh": 5e-4, "die": 1e-3, "solve": 1e-3}.get(kind, 0.01 / max(nx, ny, nz))
    x, el, (ii, jj, kk) = _box(nx, ny, nz, h, tets, 0.15 if tets else 0.1, gen, dev)
    m = dict(x=x, el=el, h=h, hg=0.0 if tets else 0.1, speed=r.uniform(14.0, 18.0),
             mats=[dict(STEEL, sy0=300e6 * r.uniform(0.8, 1.0))], emat=None, spec=None,
             thermal=None, jc=None, plane=None, die=None)
    top = torch.nonzero(kk == nz).reshape(-1)
    m["top"] = top
    if kind in ("die", "solve", "die_mesh"):
        conds = [(kk == 0, 2, 0.0)]
    else:
        conds = [(ii == 0, 0, 0.0), (jj == 0, 1, 0.0), (kk == 0, 2, 0.0),
                 (kk == nz, 2, -m["speed"])]
    nodes = [torch.nonzero(c).reshape(-1) for c, _, _ in conds]
    m["bc_node"] = torch.cat(nodes)
    m["bc_dim"] = torch.cat([torch.full_like(n, c[1]) for n, c in zip(nodes, conds)])
    m["bc_val"] = torch.cat([torch.full(n.shape, c[2], dtype=torch.float64, device=dev)
                             for n, c in zip(nodes, conds)])
    if kind in ("die", "solve"):
        m["plane"] = dict(z0=nz * h, vz=-m["speed"], k=10.0 * STEEL["E"] * h, mu=0.1)
    if kind == "die_mesh":
        # a square plate of triangles just above the part's top, its edges off
        # the part's nodes
        L = 1.37 * h * max(nx, ny)
        xyz, tri = W.axis_plane_mesh((-0.153 * L, -0.147 * L, nz * h - 1e-6), (0.847 * L, 0.0, 0.0),
                                     7, flip_normals=True)
        m["die"] = dict(xyz=xyz, tri=tri, vel=[0.0, 0.0, -m["speed"]], mu_s=0.1, mu_d=0.08,
                        pf=0.1, end_t=1e-5, hc=2.0e6, T=600.0)
        m["thermal"] = dict(T0=20.0, k=50.0, cp=460.0, exp=1.2e-5)
    if kind == "thermal":
        m["mats"] = [dict(model=2, E=200e9, nu=0.3, rho=7850.0, sy0=250e6 * r.uniform(0.9, 1.1))]
        m["jc"] = JC
        m["thermal"] = dict(T0=300.0, k=40.0, cp=450.0, exp=1.1e-5)
    if kind == "adjoint":
        octant = ((torch.arange(nx, device=dev) >= nx // 2)[None, None, :] * 1
                  + (torch.arange(ny, device=dev) >= ny // 2)[None, :, None] * 2
                  + (torch.arange(nz, device=dev) >= nz // 2)[:, None, None] * 4)
        m["emat"] = octant.reshape(-1).to(torch.int32)
        m["mats"] = [dict(STEEL, E=200e9 * r.uniform(0.8, 1.2), sy0=300e6 * r.uniform(0.8, 1.2),
                          H=1e9 * r.uniform(0.8, 1.2)) for _ in range(8)]
        m["seed_R"] = np.random.default_rng(int(seed)).uniform(0.5, 1.5, case["steps"])
    m["dt"] = 0.3 * _shortest_edge(x, el) / math.sqrt(200e9 * 1.2 / 7850.0)
    return m


def _ensemble(case, gen, r, dev):
    xs, els, dts, mats, top, spec = [], [], [], [], [], []
    bn, bd, bv, eoff, noff = [], [], [], [0], [0]
    for n in _specimens(case["nspec"]):
        h = 0.01 / n
        x, el, (ii, jj, kk) = _box(n, n, n, h, False, 0.05, gen, dev)
        mats.append(dict(model=0, E=r.uniform(70e9, 210e9), nu=0.3, rho=7850.0,
                         sy0=r.uniform(200e6, 300e6), H=r.uniform(0.2e9, 2e9)))
        vz = -r.uniform(12.0, 18.0)
        base = noff[-1]
        for c, dim, val in [(ii == 0, 0, 0.0), (jj == 0, 1, 0.0), (kk == 0, 2, 0.0), (kk == n, 2, vz)]:
            at = torch.nonzero(c).reshape(-1)
            bn.append(at + base)
            bd.append(torch.full_like(at, dim))
            bv.append(torch.full(at.shape, val, dtype=torch.float64, device=dev))
        top.append(torch.nonzero(kk == n).reshape(-1) + base)
        xs.append(x)
        els.append(el + base)
        dts.append(0.3 * _shortest_edge(x, el) / math.sqrt(mats[-1]["E"] / 7850.0))
        eoff.append(eoff[-1] + el.shape[0])
        noff.append(base + x.shape[0])
    emat = torch.repeat_interleave(torch.arange(len(mats), device=dev),
                                   torch.tensor(np.diff(eoff), device=dev)).to(torch.int32)
    return dict(x=torch.cat(xs), el=torch.cat(els), hg=0.1, mats=mats, emat=emat,
                bc_node=torch.cat(bn), bc_dim=torch.cat(bd), bc_val=torch.cat(bv),
                top=torch.cat(top), spec=(eoff, noff, np.array(dts)), dt=None, thermal=None,
                jc=None, plane=None, die=None)


# ---- one pass through the library ---------------------------------------------------


def _host(t, dtype):
    return np.ascontiguousarray(t.cpu().numpy().astype(dtype, copy=False))


def _describe(d, s):
    """The calls between a mesh and wf_init, as a driver makes them."""
    m = s["m"]
    d.set_mesh(s["x"], s["el"])
    d.set_materials(m["mats"], s["emat"])
    d.add_bcs(s["bcs"])
    if m["hg"]:
        d.set_hourglass(m["hg"])
    if m["jc"]:
        d.set_johnson_cook(0, *m["jc"])
    if m["thermal"]:
        t = m["thermal"]
        d.set_thermal(True, t["T0"])
        d.set_material_thermal(0, t["k"], t["cp"], t["exp"])
    if m["plane"]:
        p = m["plane"]
        d.set_contact_plane(p["z0"], p["vz"], p["k"], p["mu"], s["top"])
    elif m["die"]:
        p = m["die"]
        d.set_contact_trimesh(p["xyz"], p["tri"], p["vel"], p["mu_s"], p["mu_d"], p["pf"])
        d.set_contact_heat(p["hc"], p["T"])
        d.set_end_time(p["end_t"])
    else:
        d.set_reaction_nodes(s["top"], 2)
    if m["spec"]:
        d.set_specimens(*m["spec"])
    else:
        d.set_dt(m["dt"])


def prepare(case, seed):
    m = _model(case, seed)
    mixed = case["prec"] == "mixed"
    s = dict(case=case, m=m, x=_host(m["x"], np.float64), el=_host(m["el"], np.int32),
             emat=None if m["emat"] is None else _host(m["emat"], np.int32),
             top=_host(m["top"], np.int32),
             bcs=(_host(m["bc_node"], np.int64), _host(m["bc_dim"], np.int32),
                  _host(m["bc_val"], np.float64)))
    nn, ne = s["x"].shape[0], s["el"].shape[0]
    for k in ("x", "el", "top", "bc_node", "bc_dim", "bc_val", "emat"):
        m[k] = None   # the host copies are the user's
    s["prec"] = wf.WF_MIXED if mixed else wf.WF_FP64
    if case["kind"] == "adjoint":
        s["buf"] = {}
    else:
        # the program's result buffers, written once so that their pages exist
        s["buf"] = {"u": torch.zeros(nn, 3, dtype=torch.float64),
                    "v": torch.zeros(nn, 3, dtype=torch.float64),
                    "pl": torch.zeros(ne, dtype=torch.float64)}
        if m["thermal"]:
            s["buf"]["T"] = torch.zeros(nn, dtype=torch.float64)
        if mixed:
            s["buf32"] = {k: torch.zeros_like(v, dtype=torch.float32) for k, v in s["buf"].items()}
    if case["kind"] != "solve":
        s["dom"] = wf.Domain(s["prec"])
        _describe(s["dom"], s)
    if case["kind"] == "die_mesh":
        s["dom"].init()
    return s


def _read(d, s):
    """The fields into the program's buffers; the reaction history."""
    b = s["buf"]
    d.node_vec("u", out=b["u"].numpy().reshape(-1))
    d.node_vec("v", out=b["v"].numpy().reshape(-1))
    L = wf.lib()
    if L.wf_get_elem_scalar(d.h, wf.ELEM_SCALAR["pl_strain"], b["pl"].numpy()):
        raise RuntimeError("wf_get_elem_scalar failed")
    if "T" in b and L.wf_get_node_scalar(d.h, wf.NODE_SCALAR["T"], b["T"].numpy()):
        raise RuntimeError("wf_get_node_scalar failed")
    if s["m"]["spec"]:
        R = np.stack([d.specimen_reaction(k) for k in range(len(s["m"]["mats"]))])
    else:
        R = d.reaction()
    out = dict(b)
    if "buf32" in s:
        for k, v in s["buf32"].items():
            v.copy_(b[k])
        out = dict(s["buf32"])
        R = R.astype(np.float32)
    out["reaction"] = R
    return out


def run(state):
    s, case = state, state["case"]
    if case["kind"] == "adjoint":
        d = s["dom"]
        d.init()
        d.adjoint_forward(case["steps"])
        R = d.reaction()
        return dict(reaction=R, grad=d.adjoint_backward(s["m"]["seed_R"]))
    if case["kind"] == "solve":
        d = wf.Domain(s["prec"])
        _describe(d, s)
        d.init()
        # the stable step from the mesh as it is on the device (0.3 h_min / c)
        d.set_dt(0.3 * d.min_edge_length() / math.sqrt(200e9 * 1.2 / 7850.0))
        d.run(case["steps"])
        out = _read(d, s)
        d.close()
        return out
    d = s["dom"]
    if case["kind"] != "die_mesh":
        d.init()
    d.run(case["steps"])
    return _read(d, s)


# ---- what a pass cannot do without --------------------------------------------------


def work(case):
    """Bytes: every step reads and writes the state of an explicit step once
    (positions, velocities, accelerations, displacements; stress and plastic
    strain; the total strain the FP64 step keeps; tetrahedra's connectivity),
    the fields are read back once. Operations: of the element kinematics,
    stress return, forces and the node update."""
    fp = 8 if case["prec"] == "fp64" else 4
    tets = case["kind"] in ("tets", "die_mesh")
    if case["kind"] == "ensemble":
        n = _specimens(case["nspec"])
        ne, nn = sum(k ** 3 for k in n), sum((k + 1) ** 3 for k in n)
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        ne, nn = nx * ny * nz * (6 if tets else 1), (nx + 1) * (ny + 1) * (nz + 1)
    elem = 2 * 7 * fp + (16 if tets else 0) + (2 * 6 * 8 if fp == 8 else 0)
    # x (mixed: compensated pairs), v, previous a; FP64 also u
    node = 2 * (3 * 8 + 3 * 4 + 3 * 4) if fp == 4 else 2 * 4 * 3 * 8
    flops = ne * (350 if tets else 700) + nn * 60
    if case["kind"] in ("thermal", "die_mesh"):
        node += 2 * 8
        flops += ne * 150
    passes = case["steps"] * (3.0 if case["kind"] == "adjoint" else 1.0)
    out = 0 if case["kind"] == "adjoint" else nn * 6 * 8 + ne * 8
    return {"bytes": float(passes * (ne * elem + nn * node) + out), "flops": float(passes * flops)}


# ---- the same in 64 bits, in plain torch ----------------------------------------------

_HEX = [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1),
        (-1, 1, 1)]
_HG = [[1, 1, -1, -1, -1, -1, 1, 1], [1, -1, -1, 1, -1, 1, 1, -1], [1, -1, 1, -1, 1, -1, 1, -1],
       [-1, 1, -1, 1, 1, -1, 1, -1]]


def _surface(x, el):
    """External nodes, their shares of the external face areas and the mean
    least height of their elements (tetrahedra)."""
    nn, dev = x.shape[0], x.device
    faces = el[:, torch.tensor([[0, 1, 2], [0, 1, 3], [1, 2, 3], [0, 2, 3]], device=dev)].reshape(-1, 3)
    key = torch.sort(faces, 1)[0]
    key = (key[:, 0] * nn + key[:, 1]) * nn + key[:, 2]
    _, inv, cnt = torch.unique(key, return_inverse=True, return_counts=True)
    faces = faces[cnt[inv] == 1]
    p = x[faces]
    share = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]).norm(dim=1) * 0.5 / 3.0
    area = torch.zeros(nn, dtype=torch.float64, device=dev)
    area.index_add_(0, faces.reshape(-1), share.repeat_interleave(3))
    hmin = torch.full((el.shape[0],), 1e6, dtype=torch.float64, device=dev)
    for i, f in enumerate([(1, 2, 3), (0, 2, 3), (0, 1, 3), (0, 1, 2)]):
        q = [x[el[:, k]] for k in f]
        n = torch.linalg.cross(q[1] - q[0], q[2] - q[0])
        ar = n.norm(dim=1)
        hgt = ((x[el[:, i]] - q[0]) * n).sum(1).abs() / ar
        hmin = torch.where((ar >= 1e-12) & (hgt < hmin), hgt, hmin)
    length = torch.zeros(nn, dtype=torch.float64, device=dev)
    count = torch.zeros_like(length)
    length.index_add_(0, el.reshape(-1), hmin.repeat_interleave(4))
    count.index_add_(0, el.reshape(-1), torch.ones_like(hmin).repeat_interleave(4))
    return faces.unique(), area, length / count


class _Reference:
    """The explicit step of a model in 64-bit torch (out of place where a
    gradient passes). theta: E, sigma_y0, H per material, for the gradient."""

    def __init__(self, m, theta=None):
        x, el = m["x"], m["el"].long()
        dev, f8 = x.device, torch.float64
        self.m, self.x, self.el, self.npe = m, x, el, el.shape[1]
        nn, ne = x.shape[0], el.shape[0]
        self.nn, self.ne = nn, ne
        if theta is None:
            theta = torch.tensor([[q["E"], q["sy0"], q.get("H", 0.0)] for q in m["mats"]], dtype=f8,
                                 device=dev)
        E, sy0, H = theta[:, 0], theta[:, 1], theta[:, 2]
        nu = torch.tensor([q["nu"] for q in m["mats"]], dtype=f8, device=dev)
        rho = torch.tensor([q["rho"] for q in m["mats"]], dtype=f8, device=dev)
        K, G = E / (3.0 * (1.0 - 2.0 * nu)), E / (2.0 * (1.0 + nu))
        cs = torch.sqrt(K / rho)
        pick = (lambda t: t[m["emat"].long()]) if m["emat"] is not None else (lambda t: t[0])
        self.K, self.G, self.cs, self.sy0, self.H, self.E = map(pick, (K, G, cs, sy0, H, E))
        # the reference keeps one density for all elements: every material's is the same here
        self.rho = float(m["mats"][0]["rho"])
        if m["spec"]:
            eoff, noff, dts = m["spec"]
            dts = torch.tensor(dts, dtype=f8, device=dev)
            idx = torch.arange(len(dts), device=dev)
            self.spec_n = torch.repeat_interleave(idx, torch.tensor(np.diff(noff), device=dev))
            self.dt_e = torch.repeat_interleave(dts, torch.tensor(np.diff(eoff), device=dev))
            self.dt = dts[self.spec_n][:, None]
        else:
            self.dt = self.dt_e = m["dt"]
        self.alpha = (2.0 * RHO_B - 1.0) / (1.0 + RHO_B)
        self.beta = (5.0 - 3.0 * RHO_B) / ((1.0 + RHO_B) ** 2 * (2.0 - RHO_B))
        self.gamma = 1.5 - self.alpha
        self.fixed = torch.zeros(nn, 3, dtype=torch.bool, device=dev)
        self.bval = torch.zeros(nn, 3, dtype=f8, device=dev)
        self.fixed[m["bc_node"], m["bc_dim"]] = True
        self.bval[m["bc_node"], m["bc_dim"]] = m["bc_val"]
        if self.npe == 8:
            self.D = 0.125 * torch.tensor(_HEX, dtype=f8, device=dev)       # [8, 3]
            self.hgv = torch.tensor(_HG, dtype=f8, device=dev)              # [4, 8]
            self.w = 8.0
        else:
            self.D = torch.tensor([[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], dtype=f8, device=dev)
            self.w = 1.0 / 6.0
        zero = lambda *n: torch.zeros(*n, dtype=f8, device=dev)  # noqa: E731
        self.u, self.pa = zero(nn, 3), zero(nn, 3)
        # only the last dimension's velocity conditions survive the preamble
        self.v = self.bval * torch.tensor([0.0, 0.0, 1.0], dtype=f8, device=dev)
        self.tau, self.pls = zero(ne, 6), zero(ne)
        self.cf, self.ut = zero(nn, 3), zero(nn, 3)
        self.s0 = self.gather(self.volume(self.kin()[1])[:, None].expand(ne, self.npe))
        self.time, self.R = 0.0, []
        if m["thermal"]:
            self.T = torch.full((nn,), m["thermal"]["T0"], dtype=f8, device=dev)
            self.dte, self.qc = zero(ne * self.npe), zero(nn)
        if m["die"]:
            p = m["die"]
            self.ext, self.area, self.nodlen = _surface(x, el)
            self.dx = torch.tensor(p["xyz"], dtype=f8, device=dev)
            self.tri = torch.tensor(p["tri"], device=dev).long()
            self.dvel = torch.tensor(p["vel"], dtype=f8, device=dev)

    def gather(self, f):
        """Element-node values summed at the nodes."""
        out = torch.zeros((self.nn,) + tuple(f.shape[2:]), dtype=torch.float64, device=f.device)
        return out.index_add(0, self.el.reshape(-1), f.reshape((-1,) + tuple(f.shape[2:])))

    def kin(self):
        """dN/dx detJ [ne, 3, npe] and detJ."""
        J = torch.einsum("am,eak->emk", self.D, self.x[self.el])
        r0, r1, r2 = J[:, 0], J[:, 1], J[:, 2]
        A = torch.stack([torch.linalg.cross(r1, r2), torch.linalg.cross(r2, r0),
                         torch.linalg.cross(r0, r1)], 2)     # adj(J): [e, k, m]
        det = (r0 * A[:, :, 0]).sum(1)
        return torch.einsum("ekm,am->eka", A, self.D), det

    def volume(self, det):
        return det * self.w

    def step(self):
        m, el, dt, fx = self.m, self.el, self.dt, self.fixed
        vp = torch.where(fx, self.bval, self.v + (1.0 - self.gamma) * dt * self.pa)
        B, det = self.kin()
        vol = self.volume(det)
        vn = self.gather(vol[:, None].expand(self.ne, self.npe))
        jr, mass = vn / self.s0, vn / self.npe * self.rho
        L = torch.einsum("eia,eak->eik", B, vp[el]) / det[:, None, None]
        s = [L[:, 0, 0], L[:, 1, 1], L[:, 2, 2], 0.5 * (L[:, 1, 0] + L[:, 0, 1]),
             0.5 * (L[:, 2, 1] + L[:, 1, 2]), 0.5 * (L[:, 2, 0] + L[:, 0, 2])]
        w01, w12, w02 = (0.5 * (L[:, 1, 0] - L[:, 0, 1]), 0.5 * (L[:, 2, 1] - L[:, 1, 2]),
                         0.5 * (L[:, 2, 0] - L[:, 0, 2]))
        if m["thermal"]:
            c = m["thermal"]["exp"] * self.dte[el].mean(1)
            s = [s[0] - c, s[1] - c, s[2] - c] + s[3:]
        Ja = jr[el].mean(1)
        p = -self.K * (torch.where(Ja < 0.0, torch.full_like(Ja, 0.2), Ja) - 1.0)
        t = list(self.tau.unbind(1))
        c = (s[0] + s[1] + s[2]) / 3.0
        g2, de = 2.0 * self.G, self.dt_e
        # tau W^T + W tau with the reference's tensor product
        spin = [2.0 * (t[3] * w01 + t[5] * w02),
                (t[3] * w01 - t[4] * w12) + (w12 * t[4] - w01 * t[3]),
                (t[5] * w02 + t[4] * w12) - (w02 * t[5] + w12 * t[4]),
                (t[0] * w01 - t[5] * w12) + (w01 * t[1] + w02 * t[4]),
                (t[3] * w02 + t[1] * w12) + (w12 * t[2] - w01 * t[5]),
                (t[0] * w02 + t[3] * w12) + (w01 * t[4] + w02 * t[2])]
        t = [t[k] + ((s[k] - (c if k < 3 else 0.0)) * g2 + spin[k]) * de for k in range(6)]
        tr = (t[0] + t[1] + t[2]) / 3.0
        dev = [t[0] - tr, t[1] - tr, t[2] - tr]
        J2 = 0.5 * (dev[0] ** 2 + dev[1] ** 2 + dev[2] ** 2 + 2.0 * (t[3] ** 2 + t[4] ** 2 + t[5] ** 2))
        # sqrt(3 J2), with a finite slope at zero stress
        eq = torch.where(J2 > 0.0, torch.sqrt(3.0 * torch.where(J2 > 0.0, J2, torch.ones_like(J2))),
                         torch.zeros_like(J2))
        if m["jc"]:
            Bj, n, C, e0, mj, Tm, Tt, _ = m["jc"]
            rate = torch.sqrt(0.5 * ((s[0] - s[1]) ** 2 + (s[1] - s[2]) ** 2 + (s[2] - s[0]) ** 2)
                              + 3.0 * (s[3] ** 2 + s[4] ** 2 + s[5] ** 2))
            th = 1.0 - ((self.T[el].mean(1) - Tt) / (Tm - Tt)) ** mj
            sr = torch.where(rate == 0.0, torch.full_like(rate, 1e-5), rate)
            sy = (self.sy0 + Bj * self.pls ** n) * (1.0 + C * torch.log(sr / e0)) * th
            lim = torch.clamp(rate, max=1e6)
            one = torch.where(self.pls > 0.0, self.pls, torch.ones_like(self.pls))
            Ht = torch.where(self.pls > 0.0,
                             n * Bj * one ** (n - 1.0) * (1.0 + C * torch.log(lim / e0)) * th,
                             (self.E * 0.1).expand_as(one))
        else:
            sy, Ht = self.sy0 + self.H * self.pls, self.H
        on = sy < eq
        safe = torch.where(on, eq, torch.ones_like(eq))
        dg = torch.where(on, (eq - sy) / (3.0 * self.G + Ht), torch.zeros_like(eq))
        fac = 1.0 - 3.0 * self.G * dg / safe
        t = [torch.where(on, dev[k] * fac, t[k]) for k in range(3)] + \
            [torch.where(on, t[k] * fac, t[k]) for k in range(3, 6)]
        self.tau, self.pls = torch.stack(t, 1), self.pls + dg
        sg = [t[0] - p, t[1] - p, t[2] - p] + t[3:]
        S = torch.stack([torch.stack([sg[0], sg[3], sg[5]], 1), torch.stack([sg[3], sg[1], sg[4]], 1),
                         torch.stack([sg[5], sg[4], sg[2]], 1)], 1)
        f = torch.einsum("eia,eik->eak", B, S) * self.w
        if m["hg"]:
            hm = torch.einsum("ja,eak->ejk", self.hgv, vp[el])
            ch = m["hg"] * vol ** 0.6666666 * self.rho * 0.25 * self.cs
            f = f + torch.einsum("ja,ejk->eak", self.hgv, hm) * ch[:, None, None]
        fi = self.gather(f)
        cf, r = None, None
        if m["plane"]:
            cf, r = self.plane(vp, mass)
        elif m["die"]:
            cf, r = self.press(vp, mass)
        else:
            r = fi[m["top"], 2]
            r = torch.zeros(len(m["mats"]), dtype=torch.float64, device=r.device).index_add(
                0, self.spec_n[m["top"]], r) if m["spec"] else r.sum()
        self.R.append(r)
        if m["thermal"]:
            th = m["thermal"]
            fh = dg / torch.where(on, sy, torch.ones_like(dg))
            ii = [fh * (sg[0] - 0.5 * (sg[1] + sg[2])), fh * (sg[1] - 0.5 * (sg[0] + sg[2])),
                  fh * (sg[2] - 0.5 * (sg[0] + sg[1]))] + [1.5 * fh * sg[k] for k in (3, 4, 5)]
            q = 0.9 * (sg[0] * ii[0] + sg[1] * ii[1] + sg[2] * ii[2]
                       + 2.0 * (sg[3] * ii[3] + sg[4] * ii[4] + sg[5] * ii[5])) / self.dt_e
            grad = torch.einsum("eia,ea->ei", B, self.T[el])
            KT = torch.einsum("eia,ei->ea", B, grad) * (th["k"] / det * self.w)[:, None]
            mi = mass[el]
            rate = -KT / mi + (0.9 * q * vol / self.npe)[:, None] / (mi * th["cp"])
            self.dte = rate.reshape(-1)
            self.T = self.T + (self.gather(rate) + self.qc / (mass * th["cp"])) * self.dt
        a = -fi / mass[:, None]
        if cf is not None:
            a = a + cf / mass[:, None]
        a = torch.where(fx, torch.zeros_like(a), a)
        a = (a - self.alpha * self.pa) / (1.0 - self.alpha)
        v = torch.where(fx, self.bval, vp + self.gamma * dt * a)
        du = dt * (self.v + (0.5 - self.beta) * dt * self.pa) + self.beta * dt * dt * a
        self.x, self.u, self.v, self.pa = self.x + du, self.u + du, v, a
        if m["die"]:
            p = m["die"]
            ramp = math.sqrt(self.time / (0.01 * p["end_t"])) if self.time < 0.01 * p["end_t"] else 1.0
            self.dx = self.dx + ramp * self.dvel * self.dt
        self.time += self.dt if not m["spec"] else 0.0

    def plane(self, vp, mass):
        """The flat die: penalty, damping, Coulomb friction on the top nodes."""
        p, at, dt = self.m["plane"], self.m["top"], self.dt
        gap = p["z0"] + p["vz"] * self.time - self.x[at, 2]
        hit, mt, vt = gap < 0.0, mass[at], vp[at]
        k = torch.clamp(0.2 * mt / (dt * dt), max=p["k"])
        fz = k * gap - 0.2 * 2.0 * mt * torch.sqrt(k / mt) * vt[:, 2]
        ut = self.ut[at][:, :2] + vt[:, :2] * dt
        ft = -k[:, None] * ut
        most = p["mu"] * fz.abs()
        slide = ~(ft.norm(dim=1) <= most)
        sp = vt[:, :2].norm(dim=1)
        dirn = vt[:, :2] / torch.where(sp > 0.0, sp, torch.ones_like(sp))[:, None]
        ft = torch.where(slide[:, None], -most[:, None] * dirn, ft)
        ut = torch.where(slide[:, None], torch.zeros_like(ut), ut)
        self.ut = self.ut.clone()
        self.ut[at, :2] = torch.where(hit[:, None], ut, self.ut[at][:, :2])
        cf = torch.zeros_like(vp)
        cf[at] = torch.where(hit[:, None], torch.cat([ft, fz[:, None]], 1), torch.zeros_like(vt))
        return cf, (fz.abs() * hit).sum()

    def press(self, vp, mass):
        """The triangle-mesh die: every external node against the triangles in
        order; the first one it is behind, with its projection inside, acts."""
        d, dt = self.m["die"], self.dt
        P = self.dx[self.tri]
        n = torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
        n = n / n.norm(dim=1, keepdim=True)
        pp = (P[:, 2] * n).sum(1)
        at = self.ext
        x, v, mt = self.x[at], vp[at], mass[at]
        dd = x @ n.T - pp
        ok = dd < 0.0
        Q = x[:, None, :] - n[None] * dd[:, :, None]
        for a in range(3):
            e1 = P[:, (a + 1) % 3] - P[:, a]
            ok &= ~((torch.linalg.cross(e1[None].expand_as(Q), Q - P[None, :, a]) * n[None]).sum(2) < 0.0)
        hit = ok.any(1)
        j = ok.int().argmax(1)
        n, dd = n[j], dd.gather(1, j[:, None])[:, 0]
        vn = (v * n).sum(1)
        k = torch.minimum(0.2 * mt / (dt * dt), self.m["mats"][0]["E"] * self.area[at] / self.nodlen[at])
        sc = -(d["pf"] * k * dd + 0.2 * 2.0 * mt * torch.sqrt(k / mt) * vn)
        fn = sc.abs()
        vt = v - n * vn[:, None]
        ut = self.ut[at] + vt * dt
        ft = -k[:, None] * ut
        slide = ~(ft.norm(dim=1) <= d["mu_s"] * fn)
        ft = torch.where(slide[:, None], -vt * (d["mu_d"] * fn / vt.norm(dim=1))[:, None], ft)
        ut = torch.where(slide[:, None], torch.zeros_like(ut), ut)
        self.ut, self.cf = self.ut.clone(), self.cf.clone()
        self.ut[at] = torch.where(hit[:, None], ut, self.ut[at])
        self.cf[at] = torch.where(hit[:, None], n * sc[:, None] + ft, self.cf[at])
        self.qc = self.qc.clone()
        self.qc[at] = torch.where(hit, d["hc"] * self.area[at] * (d["T"] - self.T[at]), self.qc[at])
        return self.cf, (fn * hit).sum()


def exact(case, seed):
    m = _model(case, seed)
    if case["kind"] == "adjoint":
        theta = torch.tensor([[q["E"], q["sy0"], q["H"]] for q in m["mats"]], dtype=torch.float64,
                             device=m["x"].device, requires_grad=True)
        ref = _Reference(m, theta)
        for _ in range(case["steps"]):
            ref.step()
        R = torch.stack(ref.R)
        (R * torch.tensor(m["seed_R"], device=R.device)).sum().backward()
        return dict(reaction=R.detach().cpu(), grad=theta.grad.cpu())
    with torch.no_grad():
        ref = _Reference(m)
        for _ in range(case["steps"]):
            ref.step()
    out = dict(u=ref.u, v=ref.v, pl=ref.pls)
    if m["thermal"]:
        out["T"] = ref.T
    R = torch.stack(ref.R)
    out["reaction"] = R.T.contiguous() if m["spec"] else R
    return {k: v.cpu() for k, v in out.items()}
