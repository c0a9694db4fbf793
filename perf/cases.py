"""What is timed: the calls a MAESTROeX step makes into this library, through its public entry
points (``maestroex_gb300.stage``), over the sizes and options such steps use.

Families (one or two listed cases each; ``draw`` gives more of the same ranges):

* ``ppm``      Maestro::PPM on one box, called box by box from an MFIter loop: the smallest call.
* ``stage2d``  the whole stage in 2-D (y radial), replayed as a CUDA graph.
* ``stage3d``  the whole stage on one plane-parallel level: a small test problem launched
               kernel by kernel, limited slopes (ppm_type 0) on ragged boxes with walls, the
               species-streamed form, and the 256^3 production step.
* ``amr``      the stage on a two-level hierarchy: uneven boxes, refined bubbles.
* ``sphere``   the full star on uniform radial bins (the reference's default).
* ``edge``     MakeEdgeScal alone, conservative or advective, on caller FABs.
* ``velocity`` VelocityAdvance + UpdateVel.
* ``mac``      the MAC projection to 1e-10.
* ``adjoint``  the multi-step adjoint: forward and reverse, state (and velocity) gradient.

Fields are the seeded atmospheres of ``maestroex_gb300.configs``, formed on the device.
"""
import math

import numpy as np
import torch

from maestroex_gb300 import capi, configs
from maestroex_gb300.basestate import cell_to_edge
from maestroex_gb300.params import FIRSTSPEC, INTERIOR, OUTFLOW, PI, RHO, RHOH, SLIPWALL, SYMMETRY, TEMP, make_params
from maestroex_gb300.stage import (MultiFab, ScalarAdvectionStage, StageBuffers, amr_buffers, make_amr_stage,
                                   make_stage)

L, GRAV = configs.L_DOMAIN, configs.GRAV
H = 0.25 * L
# boundary types lo / hi: "open" periodic sides, a wall below and outflow above (the planar
# workloads); "walls" symmetry, slip walls and outflow mixed; "periodic" everywhere
BCS = {
    "open": ((INTERIOR, INTERIOR, SLIPWALL), (INTERIOR, INTERIOR, OUTFLOW)),
    "walls": ((OUTFLOW, SYMMETRY, SLIPWALL), (OUTFLOW, SLIPWALL, OUTFLOW)),
    "periodic": ((INTERIOR,) * 3, (INTERIOR,) * 3),
}


# ---------------------------------------------------------------- inputs
def _outer(fz, fy, fx):
    return fz[:, None, None] * fy[None, :, None] * fx[None, None, :]


def _tensor(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _modes(rng, x):
    """A smooth field of unit RMS: eight seeded Fourier modes on the cell centres x."""
    f = 0.0
    for _ in range(8):
        k, p, a = rng.integers(1, 5, size=3), rng.uniform(0, 2 * math.pi, size=3), rng.normal()
        c = [torch.cos(2 * math.pi * int(k[d]) / L * x[d] + float(p[d])) for d in range(3)]
        f = f + float(a) * _outer(c[2], c[1], c[0])
    return f / f.square().mean().sqrt()


def atmosphere(n, nspec, seed, bc, w0_amp=1.0e4, rho_pert=1.0e-5, gravity=True, gpi_amp=1.0e-5, cfl=0.7):
    """The plane-parallel atmosphere of configs.planar_config with its fields formed on the
    device: a dict for make_stage / StageBuffers without the layout and the options."""
    rng = np.random.default_rng(seed)
    dx = tuple(L / v for v in n)
    x = [(torch.arange(n[d], dtype=torch.float64, device="cuda") + 0.5) * dx[d] for d in range(3)]
    shape = (n[2], n[1], n[0])
    r = (np.arange(n[2]) + 0.5) * dx[2]
    rho0 = 1.0e7 * np.exp(-r / H)
    p0 = rho0 * abs(GRAV) * H
    lo, hi = BCS[bc]
    X = torch.zeros((nspec,) + shape, dtype=torch.float64, device="cuda")
    for s in range(nspec):
        for _ in range(6):
            w, c, a = rng.uniform(0.05, 0.2) * L, rng.uniform(0, L, size=3), rng.uniform(0.2, 1.0)
            g = []
            for d in range(3):
                dd = x[d] - float(c[d])
                if lo[d] == INTERIOR:
                    dd = dd - L * torch.round(dd / L)
                g.append(torch.exp(-(dd * dd) / (w * w)))
            X[s] += float(a) * _outer(g[2], g[1], g[0])
    X.clamp_(min=1.0e-10)
    X /= X.sum(0, keepdim=True)
    r3 = _tensor(rho0)[:, None, None]
    rho = r3 * (1.0 + rho_pert * _modes(rng, x))
    rhoh = rho * (1.0e17 + 1.0e16 * _modes(rng, x))
    rhoh0 = rhoh.mean(dim=(1, 2)).cpu().numpy()
    sold = torch.zeros((4 + nspec,) + shape, dtype=torch.float64, device="cuda")
    sold[RHO], sold[RHOH], sold[TEMP], sold[PI] = rho, rhoh, 1.0e8, 0.0
    torch.mul(X, rho[None], out=sold[FIRSTSPEC:])
    del X
    # u = curl A of eight modes, w = 0 on the z walls
    u = torch.zeros((3,) + shape, dtype=torch.float64, device="cuda")
    for _ in range(8):
        k, p, a = rng.integers(1, 5, size=3), rng.uniform(0, 2 * math.pi, size=3), rng.normal(size=3)
        cx, cy, cz = 2 * math.pi * k[0] / L, 2 * math.pi * k[1] / L, math.pi * k[2] / L
        Cx, Sx = torch.cos(cx * x[0] + p[0]), torch.sin(cx * x[0] + p[0])
        Cy, Sy = torch.cos(cy * x[1] + p[1]), torch.sin(cy * x[1] + p[1])
        Cz, Sz, Czp = torch.cos(cz * x[2]), torch.sin(cz * x[2]), torch.cos(cz * x[2] + p[2])
        u[0] += a[2] * _outer(Czp, -cy * Sy, Cx) - a[1] * _outer(cz * Cz, Cy, Cx)
        u[1] += a[0] * _outer(cz * Cz, Cy, Cx) - a[2] * _outer(Czp, Cy, -cx * Sx)
        u[2] += a[1] * _outer(Sz, Cy, -cx * Sx) - a[0] * _outer(Sz, -cy * Sy, Cx)
    u *= 0.01 * math.sqrt(5.0 / 3.0 * abs(GRAV) * H) / u.abs().max()
    re = np.arange(n[2] + 1) * dx[2]
    w0 = np.zeros(n[2] + 1)
    if w0_amp:
        w0 = sum(rng.normal() * np.sin(m * math.pi * re / L) for m in range(1, 5))
        w0 *= w0_amp / np.abs(w0).max()
        w0[0] = 0.0
    gpi = torch.zeros((3,) + shape, dtype=torch.float64, device="cuda")
    if gpi_amp:
        for d in range(3):
            gpi[d] = gpi_amp * abs(GRAV) * r3 * _modes(rng, x)
    um = [float(u[d].abs().max()) for d in range(3)]
    um[2] += float(np.abs(w0).max())
    return dict(
        n=n, dx=dx, nspec=nspec, bc_lo=lo, bc_hi=hi, dt=cfl * min(dx[d] / um[d] for d in range(3)),
        rel_eps=1.0e-8 * max(um), base_cutoff_density=1.0e3, buoyancy_cutoff_factor=5.0, uold=u, sold=sold, gpi=gpi,
        thermal=torch.zeros((1,) + shape, dtype=torch.float64, device="cuda"), rho0_old=rho0, rho0_new=rho0,
        rhoh0_old=rhoh0, rhoh0_new=rhoh0, p0_old=p0, p0_new=p0, psi=np.zeros(n[2]),
        grav_cell=np.full(n[2], GRAV if gravity else 0.0), w0_force=np.zeros(n[2]), w0=w0,
        rho0_predicted_edge=cell_to_edge(rho0))


def _size(case):
    return tuple(case["n%s" % d] for d in "xyz")


def _boxes(case):
    """The level's boxes: tiles of `grid`, or with `uneven` a seeded split of the domain."""
    n = _size(case)
    if case.get("uneven"):
        return configs.uneven_boxes(n, list(range(8, 8 * (max(n) // 8) + 1, 8)) + [v for v in n if v % 8],
                                    np.random.default_rng(case["uneven"]), p_stop=0.1)
    return configs.tile_boxes(n, case["grid"])


def _faces(rng, n, d, scale, wall_lo, wall_hi, periodic, smooth=None):
    """A face field of direction d: seeded noise (plus a smooth part), the two copies of a
    periodic face equal, no flow through walls."""
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 62)))
    m = [n[e] + (1 if e == d else 0) for e in range(3)]
    u = scale * (0.5 + 0.1 * torch.randn((1, m[2], m[1], m[0]), dtype=torch.float64, device="cuda", generator=g))
    v = u.movedim(3 - d, -1)
    if periodic:
        v[..., -1] = v[..., 0]
    if wall_lo:
        v[..., 0] = 0.0
    if wall_hi:
        v[..., -1] = 0.0
    return u


# ---------------------------------------------------------------- the families
def _prepare_ppm(case, seed):
    n, t, um = _size(case), case["ppm_type"], case["umac"]
    rng = np.random.default_rng(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    dom = tuple(v + 8 for v in n)
    cfg = dict(n=dom, dx=tuple(L / v for v in dom), nspec=1, ppm_type=t, bc_lo=(INTERIOR,) * 3, bc_hi=(INTERIOR,) * 3,
               dt=0.5 * L / max(dom) / 1.0e6, rel_eps=1.0e-2, base_cutoff_density=1.0e3)
    bx = (4, 4, 4) + tuple(3 + v for v in n)
    gr = 3 if t == 2 else 2
    x = [(torch.arange(-gr, n[d] + gr, dtype=torch.float64, device="cuda") + 0.5) / n[d] * L for d in range(3)]
    s = (1.0e7 * torch.exp(-x[2] / H)[:, None, None] * (1.0 + 0.1 * _modes(rng, x)))[None].contiguous()
    vel = []
    for d in range(3):
        m = [n[e] + (1 if um and e == d else 0) for e in range(3)]
        vel.append(3.0e5 * torch.randn((1, m[2], m[1], m[0]), dtype=torch.float64, device="cuda", generator=g))
    Ip = torch.empty((3, n[2], n[1], n[0]), dtype=torch.float64, device="cuda")
    return dict(st=ScalarAdvectionStage(make_params(cfg)), bx=bx, s=s, s_lo=[4 - gr] * 3, vel=vel, umac=um, Ip=Ip,
                Im=torch.empty_like(Ip), cfg=cfg)


def _run_ppm(q):
    q["st"].ppm(q["bx"], q["s"], q["s_lo"], 0, q["vel"], [q["bx"][:3]] * 3, q["umac"], (0,) * 6, q["Ip"], q["Im"])
    return {"Ip": q["Ip"], "Im": q["Im"]}


def _prepare_stage2d(case, seed):
    cfg = configs.planar_config_2d(n=(case["nx"], case["ny"]), nspec=case["nspec"], ppm_type=case["ppm_type"],
                                   max_grid=case["grid"], seed=seed, rho_pert=1.0e-5)
    return dict(st=make_stage(cfg), buf=StageBuffers(cfg).load(cfg), mode=capi.MODE_GRAPH)


def _prepare_stage3d(case, seed):
    cfg = atmosphere(_size(case), case["nspec"], seed, case["bc"])
    cfg.update(ppm_type=case["ppm_type"], boxes=_boxes(case))
    q = dict(st=make_stage(cfg), buf=StageBuffers(cfg, edges=case["edges"]).load(cfg),
             mode=capi.MODE_GRAPH if case["graph"] else capi.MODE_BATCHED)
    return q


def _stage_out(b):
    out = {"snew": b.snew.data, "sold": b.sold.data, "umac": [m.data for m in b.umac], "eta": b.eta.data}
    if b.sedge is not None:
        out.update(sedge=[m.data for m in b.sedge], sflux=[m.data for m in b.sflux])
    return out


def _run_stage(q):
    b = q["buf"]
    q["st"].stage_forward(b.uold, b.sold, b.gpi, b.snew, b.umac, b.sedge, b.sflux, b.eta, thermal=b.thermal,
                          mode=q["mode"])
    return _stage_out(b)


def _prepare_amr(case, seed):
    n0, rng = case["nx"], np.random.default_rng(case["layout"])
    n = (n0,) * 3
    cfg = atmosphere(n, case["nspec"], seed, "open")
    for k in ("uold", "sold", "gpi", "thermal"):
        cfg[k] = cfg[k].cpu().numpy()
    cfg.update(ppm_type=case["ppm_type"], dt=0.5 * cfg["dt"],
               boxes=configs.uneven_boxes(n, [16, 32, 48, 64, 96, 128], rng, p_stop=0.5))
    # level 1: the same atmosphere on the fine radial grid, its state injected from level 0
    fine = atmosphere((8, 8, 2 * n0), 1, seed, "open")
    w0 = np.zeros(2 * n0 + 1)
    w0[0::2], w0[1::2] = cfg["w0"], 0.5 * (cfg["w0"][:-1] + cfg["w0"][1:])
    lev1 = {k: fine[k] for k in ("rho0_old", "rho0_new", "p0_old", "p0_new", "psi", "grav_cell", "w0_force",
                                 "rho0_predicted_edge")}
    lev1.update(n=(2 * n0,) * 3, dx=tuple(v / 2 for v in cfg["dx"]), inject=True, w0=w0,
                rhoh0_old=np.repeat(cfg["rhoh0_old"], 2), rhoh0_new=np.repeat(cfg["rhoh0_new"], 2),
                boxes=configs.bubble_boxes(n, nbubbles=3, cover=case["cover"], block_edges=(8, 16, 24, 32),
                                           max_edge=32, rng=rng))
    cfg["levels"] = [{k: cfg[k] for k in configs.LEVEL_KEYS}, lev1]
    return dict(st=make_amr_stage(cfg), bufs=amr_buffers(cfg, edges=case["edges"]))


def _run_amr(q):
    q["st"].stage_forward_levels(q["bufs"], mode=capi.MODE_GRAPH)
    return [_stage_out(b) for b in q["bufs"]]


def _prepare_sphere(case, seed):
    n = case["nx"]
    cfg = configs.spherical_config(n=n, nspec=case["nspec"], ppm_type=case["ppm_type"], max_grid=case["grid"],
                                   seed=seed, exact=case["exact_bins"])
    return dict(st=make_stage(cfg), buf=StageBuffers(cfg).load(cfg), mode=capi.MODE_GRAPH)


def _prepare_edge(case, seed):
    n, bc = _size(case), case["bc"]
    cfg = atmosphere(n, case["nspec"], seed, bc)
    cfg.update(ppm_type=case["ppm_type"], boxes=_boxes(case))
    rng = np.random.default_rng(seed + 1)
    b, ng, lo, hi = cfg["boxes"], 4 if case["ppm_type"] == 2 else 3, cfg["bc_lo"], cfg["bc_hi"]
    umax = float(cfg["uold"].abs().max())

    def grown(a, g):  # the domain array with g ghost cells: periodic images, or the end cells
        for d in range(3):
            m, i = a.shape[3 - d], torch.arange(-g, a.shape[3 - d] + g, device="cuda")
            per = lo[d] == INTERIOR
            m = n[d] if per else m
            a = a.index_select(3 - d, i % m if per else i.clamp(0, m - 1))
        return a

    def multifab(a, g, nodal=-1):
        p, mf = grown(a, g), MultiFab(b, a.shape[0], g, nodal=nodal)
        for f, l, h in zip(mf.fabs, mf.los, mf.his):
            f.copy_(p[(slice(None),) + tuple(slice(l[d] + g, h[d] + g + 1) for d in (2, 1, 0))])
        return mf

    # the MAC velocity: the mean of the cell velocity on the faces, with seeded noise on it
    um = []
    for d in range(3):
        per = lo[d] == INTERIOR
        u = _faces(rng, n, d, 0.2 * umax, not per and lo[d] != OUTFLOW, not per and hi[d] != OUTFLOW, per)
        v, c = u.movedim(3 - d, -1), cfg["uold"][d:d + 1].movedim(3 - d, -1)
        v[..., 1:-1] += 0.5 * (c[..., 1:] + c[..., :-1])
        if per:
            v[..., 0] += 0.5 * (c[..., 0] + c[..., -1])
            v[..., -1] = v[..., 0]
        um.append(u)
    force = torch.zeros_like(cfg["sold"])
    if case["conservative"]:
        start, num = RHO, 1
    else:
        start, num = FIRSTSPEC, case["nspec"]
        cfg["sold"][start:] /= cfg["sold"][RHO].clone()
    force[start:start + num] = 1.0e-3 / cfg["dt"] * cfg["sold"][start:start + num]
    q = dict(st=make_stage(cfg), state=multifab(cfg["sold"], ng), umac=[multifab(um[d], 1, d) for d in range(3)],
             force=multifab(force, 1), sedge=[MultiFab(b, 4 + case["nspec"], 0, nodal=d) for d in range(3)],
             start=start, num=num, cons=int(case["conservative"]))
    if case.get("keep"):
        q["domain"] = (cfg, um, force)
    return q


def _run_edge(q):
    q["st"].make_edge_scal(q["state"], q["sedge"], q["umac"], q["force"], 0, q["start"], q["start"], q["num"],
                           q["cons"])
    c = slice(q["start"], q["start"] + q["num"])
    return [[f[c] for f in m.fabs] for m in q["sedge"]]


def _prepare_velocity(case, seed):
    cfg = atmosphere(_size(case), 2, seed, case["bc"])
    cfg.update(ppm_type=case["ppm_type"], boxes=_boxes(case))
    st, b = make_stage(cfg), cfg["boxes"]
    buf = StageBuffers(cfg, edges=False).load(cfg)
    st.advance_premac(buf.uold, buf.sold, buf.gpi, buf.umac)
    q = dict(st=st, uold=buf.uold, sold=buf.sold, gpi=buf.gpi, umac=buf.umac, unew=MultiFab(b, 3, buf.sold.ng),
             rhohalf=MultiFab(b, 1, 0).from_domain((1.0 + 1.0e-4) * cfg["sold"][RHO:RHO + 1]),
             uedge=[MultiFab(b, 3, 0, nodal=d) for d in range(3)])
    return q


def _run_velocity(q):
    q["st"].velocity_advance(q["uold"], q["sold"], q["rhohalf"], q["gpi"], q["umac"], q["unew"], q["uedge"])
    return {"unew": q["unew"].data, "uedge": [m.data for m in q["uedge"]]}


def _mac_inputs(case, seed):
    n, bc = _size(case), case["bc"]
    cfg = atmosphere(n, 2, seed, bc, w0_amp=0.0, rho_pert=1.0e-3)
    cfg.update(ppm_type=1, boxes=_boxes(case))
    rng = np.random.default_rng(seed + 1)
    lo, hi = cfg["bc_lo"], cfg["bc_hi"]
    umax = float(cfg["uold"].abs().max())
    um = [_faces(rng, n, d, umax, lo[d] not in (INTERIOR, OUTFLOW), hi[d] not in (INTERIOR, OUTFLOW),
                 lo[d] == INTERIOR) for d in range(3)]
    beta0 = cfg["rho0_old"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    noise = torch.randn(cfg["thermal"].shape, dtype=torch.float64, device="cuda", generator=g)
    macrhs = 1.0e-3 * umax / cfg["dx"][0] * _tensor(beta0)[:, None, None] * noise
    return cfg, um, beta0, macrhs


def _prepare_mac(case, seed):
    cfg, um, beta0, macrhs = _mac_inputs(case, seed)
    b = cfg["boxes"]
    ustar = [MultiFab(b, 1, 1, nodal=d).from_domain(um[d]) for d in range(3)]
    return dict(st=make_stage(cfg), ustar=ustar, umac=[MultiFab(b, 1, 1, nodal=d) for d in range(3)],
                rhs=MultiFab(b, 1, 0).from_domain(macrhs), rho=MultiFab(b, 1, 0).from_domain(cfg["sold"][RHO:RHO + 1]),
                beta0=beta0, phi=MultiFab(b, 1, 0))


def _run_mac(q):
    for u, v in zip(q["umac"], q["ustar"]):  # the projection works in place on this step's Utilde*
        u.data.copy_(v.data)
    q["st"].mac_project(q["umac"], q["rhs"], q["rho"], q["beta0"], macphi=q["phi"])
    return {"umac": [[f[:, 1:-1, 1:-1, 1:-1] for f in m.fabs] for m in q["umac"]], "phi": q["phi"].fabs}


def _prepare_adjoint(case, seed):
    n, bc, nspec = _size(case), case["bc"], case["nspec"]
    cfg = atmosphere(n, nspec, seed, bc, w0_amp=0.0 if case["grad_u"] else 1.0e4, rho_pert=1.0e-2, gravity=False,
                     gpi_amp=0.0, cfl=0.5)
    cfg.update(ppm_type=case["ppm_type"], boxes=_boxes(case), evolve_base_state=0)
    b, ns = cfg["boxes"], 4 + nspec
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn(cfg["sold"].shape, dtype=torch.float64, device="cuda", generator=g)
    w[RHO], w[TEMP], w[PI] = 0.0, 0.0, 0.0
    return dict(st=make_stage(cfg), uold=MultiFab(b, 3, 0).from_domain(cfg["uold"]),
                sold=MultiFab(b, ns, 0).from_domain(cfg["sold"]), weight=MultiFab(b, ns, 0).from_domain(w),
                grad=MultiFab(b, ns, 0), sfin=MultiFab(b, ns, 0),
                gu=MultiFab(b, 3, 0) if case["grad_u"] else None, steps=case["steps"], ckpt=case["ckpt"])


def _run_adjoint(q):
    J, _ = q["st"].stage_adjoint(q["uold"], q["sold"], q["weight"], q["steps"], q["ckpt"], grad_s=q["grad"],
                                 sfinal=q["sfin"], grad_u=q["gu"])
    return {"J": J, "grad_s": q["grad"].data, "sfinal": q["sfin"].data,
            "grad_u": None if q["gu"] is None else q["gu"].data}


PREPARE = {"ppm": _prepare_ppm, "stage2d": _prepare_stage2d, "stage3d": _prepare_stage3d, "amr": _prepare_amr,
           "sphere": _prepare_sphere, "edge": _prepare_edge, "velocity": _prepare_velocity, "mac": _prepare_mac,
           "adjoint": _prepare_adjoint}
RUN = {"ppm": _run_ppm, "stage2d": _run_stage, "stage3d": _run_stage, "amr": _run_amr, "sphere": _run_stage,
       "edge": _run_edge, "velocity": _run_velocity, "mac": _run_mac, "adjoint": _run_adjoint}


def prepare(case, seed):
    q = PREPARE[case["family"]](case, seed)
    q["family"] = case["family"]
    return q


def run(state):
    return RUN[state["family"]](state)


# ---------------------------------------------------------------- the cases
def listed():
    def cube(n, **kw):
        return dict(nx=n, ny=n, nz=n, **kw)

    return [
        # one box of an MFIter loop: 32^3 cells grown by one, traced with the MAC velocity
        cube(34, name="ppm_box_34", family="ppm", ppm_type=1, umac=1),
        # the 2-D reference problem: one 256 x 256 box, 3 species
        dict(name="stage2d_256", family="stage2d", nx=256, ny=256, nz=1, nspec=3, ppm_type=1, grid=256),
        # a small test problem, kernels launched one by one: latency and launches
        cube(32, name="stage3d_32_batched", family="stage3d", nspec=3, ppm_type=1, bc="open", grid=16, graph=False,
             edges=True),
        # limited slopes on uneven boxes, symmetry / wall / outflow faces
        dict(name="stage3d_slopes_ragged", family="stage3d", nx=72, ny=56, nz=88, nspec=5, ppm_type=0, bc="walls",
             uneven=2, graph=False, edges=True),
        # an ordinary step of a 13-species network, ppm_type 2, no edge states asked for
        cube(128, name="stage3d_128_streamed", family="stage3d", nspec=13, ppm_type=2, bc="open", grid=64, graph=True,
             edges=False),
        # the production step (the benchmark's workload)
        cube(256, name="stage3d_256", family="stage3d", nspec=13, ppm_type=1, bc="open", grid=64, graph=True,
             edges=True),
        # two levels: uneven level-0 boxes, refined bubbles
        cube(96, name="amr_96", family="amr", nspec=13, ppm_type=2, layout=4, cover=0.06, edges=True),
        # the full star on one level, uniform radial bins
        cube(96, name="sphere_96", family="sphere", nspec=21, ppm_type=2, grid=32, exact_bins=False),
        # MakeEdgeScal alone: the density in conservative form
        dict(name="edge_conservative", family="edge", nx=96, ny=80, nz=112, nspec=2, ppm_type=1, bc="periodic",
             grid=48, conservative=True),
        # the velocity update of the same step
        cube(128, name="velocity_128", family="velocity", ppm_type=1, bc="open", grid=64),
        # the MAC projection of the production step
        cube(256, name="mac_256", family="mac", bc="open", grid=128),
        # sensitivities: four steps, states stored every two, state and velocity gradient
        cube(64, name="adjoint_64", family="adjoint", nspec=3, ppm_type=1, bc="periodic", grid=32, steps=4, ckpt=2,
             grad_u=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tile(rng, n, most=10000):
    """A box edge that leaves no sliver narrower than 4 cells and makes at most `most` boxes."""
    ok = [g for g in (16, 24, 32, 48, 64, 96, 128) if all(v % g == 0 or v % g >= 4 for v in n) and
          math.prod(-(-v // g) for v in n) <= most]
    return rng.choice(ok or [max(n)])


def draw(rng):
    f = rng.choice(sorted(PREPARE))
    c = dict(family=f)
    if f == "ppm":
        c.update(nx=_log(rng, 8, 128), ny=_log(rng, 8, 128), nz=_log(rng, 8, 128), ppm_type=rng.choice([1, 2]),
                 umac=rng.choice([0, 1]))
    elif f == "stage2d":
        n = (_log(rng, 32, 1024), _log(rng, 32, 1024))
        c.update(nx=n[0], ny=n[1], nz=1, nspec=rng.choice([2, 3, 13]), ppm_type=rng.choice([0, 1, 2]),
                 grid=rng.choice([max(n), _tile(rng, n)]))
    elif f in ("stage3d", "edge", "velocity"):
        top = {"stage3d": 160, "edge": 192, "velocity": 192}[f]
        n = tuple(_log(rng, 20, top) for _ in range(3))
        c.update(nx=n[0], ny=n[1], nz=n[2], ppm_type=rng.choice([0, 1, 1, 2] if f == "stage3d" else [1, 2]),
                 bc=rng.choice(sorted(BCS)), grid=_tile(rng, n, 18 if f == "edge" else 10000))
        if f != "velocity":
            c.update(nspec=rng.choice([2, 3, 5, 13]))
        if f == "stage3d":
            if c["bc"] == "periodic":
                c["bc"] = "open"  # an atmosphere is not periodic in z
            c.update(graph=rng.random() < 0.5, edges=rng.random() < 0.5)
        if f == "edge":
            c.update(conservative=rng.random() < 0.5)
        if f == "velocity":
            c["bc"] = rng.choice(["open", "walls"])
    elif f == "amr":
        c.update(nx=rng.choice([48, 64, 80, 96, 112]), nspec=rng.choice([3, 5, 13]), ppm_type=rng.choice([1, 2]),
                 layout=rng.randrange(1000), cover=round(rng.uniform(0.02, 0.1), 3), edges=rng.random() < 0.5)
        c.update(ny=c["nx"], nz=c["nx"])
    elif f == "sphere":
        n = 8 * rng.randrange(4, 14)
        c.update(nx=n, ny=n, nz=n, nspec=rng.choice([3, 13, 21]), ppm_type=rng.choice([1, 2]), grid=_tile(rng, (n,)),
                 exact_bins=rng.random() < 0.5)
    elif f == "mac":
        n = 16 * rng.randrange(2, 13)
        c.update(nx=n, ny=n, nz=n, bc="open", grid=-(-n // 32) * 16)
    else:
        n = tuple(4 * _log(rng, 5, 20) for _ in range(3))
        gu = rng.random() < 0.5
        c.update(nx=n[0], ny=n[1], nz=n[2], nspec=rng.choice([2, 3, 5]), ppm_type=1,
                 bc="periodic" if gu else rng.choice(["periodic", "open"]), grid=_tile(rng, n), steps=4,
                 ckpt=rng.choice([2, 4]), grad_u=gu)
    return c


def _cells(case):
    c = case["nx"] * case["ny"] * case["nz"]
    if case["family"] == "amr":
        c += int(8 * case["cover"] * 1.6 * c)  # the blocks that hold the bubbles
    return c


def work(case):
    """Doubles read and written once per cell (inputs, then outputs), and the FP64 operations
    of the method: per component and direction, PPM (slope 3, interface 8, limiter and tracing
    15; twice that for ppm_type 2's fourth-order limiter), the two transverse states (2 x 8) and the edge state (14)."""
    f, n, t = case["family"], _cells(case), case.get("ppm_type", 1)
    ns, nd = case.get("nspec", 0), 2 if case["family"] == "stage2d" else 3
    ppm = {0: 12, 1: 26, 2: 52}[t]
    comp = nd * (ppm + 30)
    if f == "ppm":
        return {"bytes": 8 * n * (1 + 3 + 6), "flops": n * 3 * ppm}
    if f in ("stage2d", "stage3d", "amr", "sphere"):
        nscal = 4 + ns
        b = nd + nscal + nd + 1 + nscal + nd + 1 + (2 * nd * (2 + ns) if case.get("edges", True) else 0)
        return {"bytes": 8 * n * b, "flops": n * ((ns + 2 + nd) * comp + 25 * ns)}
    if f == "edge":
        num = 1 if case["conservative"] else ns
        return {"bytes": 8 * n * (2 * num + 3 + 3 * num), "flops": n * num * (comp + 18)}
    if f == "velocity":
        return {"bytes": 8 * n * (3 + 1 + 1 + 3 + 3 + 3 + 9), "flops": n * (3 * comp + 40)}
    if f == "mac":  # about 12 cycles of 4 sweeps and a residual, 13 operations a cell
        return {"bytes": 8 * n * (3 + 1 + 1 + 3 + 1), "flops": n * 12 * 5 * 13 * 8 / 7}
    one = n * ((ns + 2 + nd) * comp + 25 * ns)
    return {"bytes": 8 * n * (3 + 2 * (4 + ns) + 2 * (4 + ns) + (3 if case["grad_u"] else 0)),
            "flops": 3 * case["steps"] * one}


# ---------------------------------------------------------------- in plain torch
def _sh(a, d, m):
    """a shifted: element i holds a(i + m) along direction d (x = 0), wrapping around."""
    return torch.roll(a, -m, dims=a.dim() - 1 - d)


def _ppm1(s, d, ulo, uhi, dt, dx, eps):
    """Ip, Im of PPM (ppm_type 1) along d away from boundaries; ulo / uhi: the tracing velocity
    on the low / high side of each cell."""
    sm1, sp1 = _sh(s, d, -1), _sh(s, d, 1)
    c, l, r = 0.5 * (sp1 - sm1), 2.0 * (s - sm1), 2.0 * (sp1 - s)
    dv = torch.copysign(torch.minimum(c.abs(), torch.minimum(l.abs(), r.abs())), c)
    dv = torch.where((l > 0) == (r > 0), dv, torch.zeros_like(dv))
    dv = torch.where((l == 0) | (r == 0), torch.zeros_like(dv), dv)
    f = 0.5 * (s + sm1) - (dv - _sh(dv, d, -1)) / 6.0
    f = torch.maximum(f, torch.minimum(s, sm1))
    sm = torch.minimum(f, torch.maximum(s, sm1))
    sp = _sh(sm, d, 1)
    a, q = sp - s, s - sm
    flat = ~(((a > 0) & (q > 0)) | ((a < 0) & (q < 0)))
    steep_p, steep_m = a.abs() >= 2.0 * q.abs(), q.abs() >= 2.0 * a.abs()
    sp2 = torch.where(flat, s, torch.where(steep_p, 3.0 * s - 2.0 * sm, sp))
    sm2 = torch.where(flat, s, torch.where(steep_m & ~steep_p, 3.0 * s - 2.0 * sp, sm))
    s6 = 6.0 * s - 3.0 * (sm2 + sp2)
    sg = uhi.abs() * dt / dx
    Ip = torch.where(uhi > eps, sp2 - 0.5 * sg * (sp2 - sm2 - (1.0 - 2.0 / 3.0 * sg) * s6), s)
    sg = ulo.abs() * dt / dx
    Im = torch.where(ulo < -eps, sm2 + 0.5 * sg * (sp2 - sm2 + (1.0 - 2.0 / 3.0 * sg) * s6), s)
    return Ip, Im


def _exact_ppm(case, seed):
    if case["ppm_type"] != 1:
        return None
    q = _prepare_ppm(case, seed)
    n, cfg, s = _size(case), q["cfg"], q["s"][0]
    inner = (slice(2, -2),) * 3
    out = {"Ip": torch.empty_like(q["Ip"]), "Im": torch.empty_like(q["Im"])}
    for d in range(3):
        v = q["vel"][d][0]
        full = torch.zeros((2,) + tuple(s.shape), dtype=torch.float64, device="cuda")
        for side in (0, 1):
            full[side][inner] = v.narrow(2 - d, side if case["umac"] else 0, n[d])
        Ip, Im = _ppm1(s, d, full[0], full[1], cfg["dt"], cfg["dx"][d], cfg["rel_eps"])
        out["Ip"][d], out["Im"][d] = Ip[inner], Im[inner]
    return out


def _exact_edge(case, seed):
    """MakeEdgeScal on a periodic domain, conservative, ppm_type 1."""
    if case["ppm_type"] != 1 or case["bc"] != "periodic" or not case["conservative"]:
        return None
    cfg, um, force = _prepare_edge(dict(case, keep=True), seed)["domain"]
    n, dt, dx, eps = cfg["n"], cfg["dt"], cfg["dx"], cfg["rel_eps"]
    s, f = cfg["sold"][RHO], force[RHO]
    u = [um[d][0].narrow(2 - d, 0, n[d]) for d in range(3)]  # the low face of each cell
    du = [_sh(u[d], d, 1) - u[d] for d in range(3)]
    divu = (du[0] + du[1] + du[2]) / dx[0]

    def upwind(v, l, r, tie):
        return torch.where(v.abs() > tie, torch.where(v > 0, l, r), 0.5 * (l + r))

    lr = []
    for d in range(3):
        Ip, Im = _ppm1(s, d, u[d], _sh(u[d], d, 1), dt, dx[d], eps)
        lr.append((Ip, Im))  # at the cell: its high-side and low-side state
    simh = [upwind(u[d], _sh(lr[d][0], d, -1), lr[d][1], 0.0) for d in range(3)]
    qf = {}
    for d in range(3):
        for t in range(3):
            if t == d:
                continue
            w = simh[t] * u[t]
            c = -dt / 3.0 / dx[t] * (_sh(w, t, 1) - w) - dt / 3.0 * s * divu + dt / 3.0 / dx[t] * s * du[t]
            qf[d, t] = upwind(u[d], _sh(lr[d][0] + c, d, -1), lr[d][1] + c, eps)
    out = []
    for d in range(3):
        t1, t2 = [t for t in range(3) if t != d]
        c = 0.5 * dt * f - 0.5 * dt / dx[d] * s * du[d]
        for a, b in ((t1, t2), (t2, t1)):
            w = qf[a, b] * u[a]
            c = c - 0.5 * dt / dx[a] * (_sh(w, a, 1) - w)
        e = upwind(u[d], _sh(lr[d][0] + c, d, -1), lr[d][1] + c, eps)
        e = torch.cat([e, e.narrow(2 - d, 0, 1)], dim=2 - d)
        out.append([e[None][(slice(None),) + tuple(slice(b[k], b[3 + k] + (2 if k == d else 1)) for k in (2, 1, 0))]
                    for b in cfg["boxes"]])
    return out


def _exact_mac(case, seed):
    """The projection by conjugate gradients on the discrete system (diagonal
    preconditioner), to 1e-15 of the right-hand side."""
    cfg, um, beta0, macrhs = _mac_inputs(case, seed)
    n, dx, lo, hi = cfg["n"], cfg["dx"], cfg["bc_lo"], cfg["bc_hi"]
    rho = cfg["sold"][RHO]
    b0 = np.asarray(beta0)
    e = np.empty(n[2] + 1)
    e[2:-2] = 7.0 / 12.0 * (b0[2:-1] + b0[1:-2]) - 1.0 / 12.0 * (b0[3:] + b0[:-3])
    e[2:-2] = np.clip(e[2:-2], np.minimum(b0[1:-2], b0[2:-1]), np.maximum(b0[1:-2], b0[2:-1]))
    e[0], e[1], e[-2], e[-1] = b0[0], 0.5 * (b0[0] + b0[1]), 0.5 * (b0[-1] + b0[-2]), b0[-1]
    bz = [_tensor(b0)[:, None, None], _tensor(b0)[:, None, None], _tensor(e)[:, None, None]]

    def ends(a, d):  # the neighbours beyond the two ends of direction d
        x = 2 - d
        first, last = a.narrow(x, 0, 1), a.narrow(x, n[d] - 1, 1)
        return (last, first) if lo[d] == INTERIOR else (first, last)

    B, kind = [], []
    for d in range(3):
        a, z = ends(rho, d)
        B.append(bz[d] * bz[d] / (0.5 * (torch.cat([a, rho], 2 - d) + torch.cat([rho, z], 2 - d))))
        kind.append("per" if lo[d] == INTERIOR else (lo[d] == OUTFLOW, hi[d] == OUTFLOW))

    def grad(p, d):
        x = 2 - d
        if kind[d] == "per":
            a, z = ends(p, d)
        else:  # Dirichlet 0 on the face through the ghost -phi, Neumann otherwise
            a, z = [(-1.0 if dirichlet else 1.0) * p.narrow(x, i, 1) for dirichlet, i in
                    zip(kind[d], (0, n[d] - 1))]
        return (torch.cat([p, z], x) - torch.cat([a, p], x)) / dx[d]

    def diff(v, d):
        return (v.narrow(2 - d, 1, n[d]) - v.narrow(2 - d, 0, n[d])) / dx[d]

    def apply(p):
        return sum(diff(-B[d] * grad(p, d), d) for d in range(3))

    bu = [um[d][0] * bz[d] for d in range(3)]
    rhs = macrhs[0] - sum(diff(bu[d], d) for d in range(3))
    diag = 0.0
    for d in range(3):
        w, x = B[d] / (dx[d] * dx[d]), 2 - d
        if kind[d] != "per":
            w = w.clone()
            for dirichlet, i in zip(kind[d], (0, n[d])):
                w.narrow(x, i, 1).mul_(2.0 if dirichlet else 0.0)
        diag = diag + w.narrow(x, 0, n[d]) + w.narrow(x, 1, n[d])
    p, r = torch.zeros_like(rhs), rhs.clone()
    z = r / diag
    d_, rz = z.clone(), (r * z).sum()
    goal = 1.0e-15 * float(rhs.norm())
    for it in range(20000):
        Ad = apply(d_)
        a = rz / (d_ * Ad).sum()
        p += a * d_
        r -= a * Ad
        if it % 50 == 49 and float(r.norm()) <= goal:
            break
        z = r / diag
        rz, old = (r * z).sum(), rz
        d_ = z + (rz / old) * d_
    out = []
    for d in range(3):
        u = (bu[d] - B[d] * grad(p, d)) / bz[d]
        out.append([u[None][(slice(None),) + tuple(slice(b[k], b[3 + k] + (2 if k == d else 1)) for k in (2, 1, 0))]
                    for b in cfg["boxes"]])
    return {"umac": out, "phi": [p[None, b[2]:b[5] + 1, b[1]:b[4] + 1, b[0]:b[3] + 1] for b in cfg["boxes"]]}


def exact(case, seed):
    """The single functions in plain torch; the whole stages, the velocity update and the
    adjoint, which chain dozens of them, have no value here."""
    f = {"ppm": _exact_ppm, "edge": _exact_edge, "mac": _exact_mac}.get(case["family"])
    return f(case, seed) if f else None
