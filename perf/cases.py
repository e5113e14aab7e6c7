"""Performance cases: what a program that uses this library has it do.

Each case goes through the public entry points (functor calls, steppers,
ensembles, the octree far field, the shallow-water sums, the network's
gradient) on meshes and initial conditions of the kind the configurations and
tests use, with the particles turned by a seeded rotation and the vorticity
made of seeded Gaussian vortices.  ``exact`` restates the same sums and
updates in plain torch FP64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from lpm_gb300 import core
from lpm_gb300 import functors as F
from lpm_gb300.bve import BVERK4, BVESphere
from lpm_gb300.ensemble import BVEEnsemble, random_vortex_params
from lpm_gb300.farfield import NNORM, NPARAM, FarField
from lpm_gb300.ic2d import Incompressible2D, Incompressible2DRK2

MESH = {"icos": core.MESH_ICOS_TRI, "cubed": core.MESH_CUBED_SPHERE, "quad": core.MESH_QUAD_RECT}
PREC = {"fp64": core.FP64, "fp32c": core.FP32C, "chord64": core.FP64_CHORD}
MASKED = core.STEP_SKIP_MASKED_TARGETS
PLANE_RADIUS = 4.0
PSE_EPS = 0.25
EXACT_PAIRS = 4e10  # above this the plain FP64 sum takes too long


def listed():
    return [
        # the smallest call a host program makes: one functor launch of a
        # coarse run, in the default precision; latency
        dict(name="functor_small", kind="sums", mesh="icos", level=2, prec="fp64", eps=0.0,
             faces=False, psi=False, ntgt=0, soa=False),
        # initialisation and output of a run: velocity and stream function on
        # vertices and faces, default precision
        dict(name="solve_fp64", kind="sums", mesh="cubed", level=5, prec="fp64", eps=0.0,
             faces=True, psi=True, ntgt=0, soa=False),
        # velocity and stream function at a ragged number of passive tracers
        # and on the faces, smoothed kernel, FP32 compensated, SoA arrays
        dict(name="tracers_fp32c", kind="sums", mesh="icos", level=6, prec="fp32c", eps=0.01,
             faces=True, psi=True, ntgt=100003, soa=True),
        # a step of the FP64 validation run (Rossby-Haurwitz class, level 4)
        dict(name="rk4_fp64", kind="rk4", level=4, prec="fp64", eps=0.0, reproject=False),
        # a step of the high-resolution FP32 compensated run; the largest case
        dict(name="rk4_fp32c", kind="rk4", level=7, prec="fp32c", eps=0.01, reproject=True),
        # planar dipoles: a Heun step with velocity and stream function
        dict(name="rk2_plane_fp32c", kind="rk2", mesh="quad", level=7, prec="fp32c", eps=0.05),
        # an ensemble of small problems of uneven size advanced together
        dict(name="ensemble_fp32c", kind="ensemble", problems=32, lo=3, hi=5, eps=0.01),
        # the octree far field as a function call: new positions every call
        dict(name="farfield_velocity", kind="ffvel", level=6, theta=0.4),
        # a step whose evaluations use the far field with the learned
        # correction
        dict(name="farfield_rk4_net", kind="ffrk4", level=7, theta=0.5, net=True),
        # spherical shallow water: vertex and face sums, FP32 compensated
        dict(name="swe_sphere_fp32c", kind="swe", mesh="icos", level=6, prec="fp32c", eps=0.01),
        # planar shallow water with particle strength exchange, FP64
        dict(name="swe_plane_fp64", kind="swe", mesh="quad", level=5, prec="fp64", eps=0.02),
        # training direction of the correction network: forward and backward
        dict(name="network_gradient", kind="grad", rows=16384),
    ]


def draw(rng):
    kind = rng.choice(["sums", "sums", "sums", "rk4", "rk4", "rk2", "ensemble", "ffvel", "ffrk4",
                       "swe", "swe", "grad"])
    eps = rng.choice([0.0, round(10 ** rng.uniform(-2.5, -1), 5)])
    if kind == "sums":
        mesh, prec = rng.choice(["icos", "cubed", "quad"]), rng.choice(["fp64", "fp64", "fp32c", "chord64"])
        top = {"icos": 6, "cubed": 6, "quad": 6}[mesh] + (prec == "fp32c")
        # divided icosahedral faces coincide with their central child: face
        # targets there need eps > 0
        faces = rng.random() < 0.5
        if faces and mesh == "icos" and eps == 0.0:
            eps = 0.01
        return dict(kind=kind, mesh=mesh, level=rng.randint(1, top - (prec != "fp32c")), prec=prec,
                    eps=eps, faces=faces, psi=rng.random() < 0.5,
                    ntgt=rng.choice([0, int(10 ** rng.uniform(0, 4.5))]), soa=rng.random() < 0.5)
    if kind == "rk4":
        prec = rng.choice(["fp64", "fp32c", "fp32c", "chord64"])
        return dict(kind=kind, level=rng.randint(2, 6 if prec == "fp32c" else 5), prec=prec,
                    eps=eps if prec != "fp32c" else max(eps, 0.005), reproject=rng.random() < 0.5)
    if kind == "rk2":
        mesh, prec = rng.choice(["icos", "cubed", "quad"]), rng.choice(["fp64", "fp32c"])
        return dict(kind=kind, mesh=mesh, level=rng.randint(2, 6 if prec == "fp32c" else 4),
                    prec=prec, eps=max(eps, 0.01))
    if kind == "ensemble":
        return dict(kind=kind, problems=rng.randint(2, 48), lo=rng.randint(2, 4),
                    hi=rng.randint(4, 5), eps=max(eps, 0.005))
    if kind in ("ffvel", "ffrk4"):
        c = dict(kind=kind, level=rng.randint(4, 7), theta=round(rng.uniform(0.3, 0.55), 3))
        if kind == "ffrk4":
            c["net"] = rng.random() < 0.4
        return c
    if kind == "swe":
        mesh, prec = rng.choice(["icos", "quad"]), rng.choice(["fp64", "fp32c"])
        return dict(kind=kind, mesh=mesh, level=rng.randint(2, 6 if prec == "fp32c" else 4),
                    prec=prec, eps=max(eps, 0.01))
    return dict(kind=kind, rows=128 * int(2 ** rng.uniform(0, 8)))


# ---- inputs ----------------------------------------------------------------

_contexts = {}


def _ctx(prec):
    """One context per precision for the whole process, as a program keeps."""
    if prec not in _contexts:
        _contexts[prec] = core.Context(0, precision=PREC[prec])
    return _contexts[prec]


def _dev():
    return torch.device("cuda", 0)


def _rng(seed):
    return np.random.default_rng(seed)


def _turn(rng, x):
    """Sphere points after a seeded solid rotation (unit length kept)."""
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    y = x @ (q * np.sign(np.diag(r)))
    return y / np.linalg.norm(y, axis=1, keepdims=True)


def _mesh(case, seed):
    """Positions (rotated / shifted), areas, mask and vorticity, on the host."""
    rng = _rng(seed)
    plane = case.get("mesh") == "quad"
    vx, fx, fa, fm = core.build_mesh(MESH[case.get("mesh", "icos")], case["level"],
                                     PLANE_RADIUS if plane else 1.0)
    if plane:
        shift = rng.uniform(-0.01, 0.01, 2)
        vx, fx = vx + shift, fx + shift
        c, s = rng.uniform(-2, 2, (4, 2)), rng.uniform(0.5, 1.0, 4)
        a = rng.uniform(-3, 3, 4)

        def field(x):
            return sum(k * np.exp(-((x - p) ** 2).sum(1) / w**2) for k, p, w in zip(a, c, s))
    else:
        both = _turn(rng, np.concatenate([vx, fx]))
        vx, fx = both[: len(vx)], both[len(vx):]
        prm = random_vortex_params(rng)

        def field(x):
            return core.eval_ic(core.IC_MULTI_GAUSSIAN, prm, x)
    return dict(vx=vx, fx=fx, fa=fa, fm=fm, vz=field(vx), fz=field(fx), field=field, rng=rng)


def _up(a, soa=False):
    t = torch.from_numpy(np.ascontiguousarray(a)).to(_dev())
    return t.t().contiguous().t() if soa and t.dim() == 2 else t


def _bve(case, seed, ctx):
    m = _mesh(dict(case, mesh="icos"), seed)
    sph = BVESphere(case["level"], ctx=ctx)
    sph.vert_x, sph.face_x = _up(m["vx"]), _up(m["fx"])
    sph.rel_vort_verts, sph.rel_vort_faces = _up(m["vz"]), _up(m["fz"])
    return sph


def _bve_velocity(sph, ctx, eps):
    """Velocities of the initial state with smoothing eps."""
    if eps == 0.0:
        sph.init_velocity()
    else:
        F.ic2d_passive_sums(ctx, sph.velocity_verts, None, sph.vert_x, sph.face_x,
                            sph.rel_vort_faces, sph.face_area, sph.face_mask, eps)
        F.ic2d_active_sums(ctx, sph.velocity_faces, None, sph.face_x, sph.rel_vort_faces,
                           sph.face_area, sph.face_mask, eps, self_rule=1)
    sph.velocity_faces[sph.face_mask.bool()] = 0.0  # divided faces are not moved


def _swe_fields(case, seed):
    m = _mesh(case, seed)
    rng = m["rng"]
    nf = len(m["fx"])
    sig = m["fz"][::-1].copy() * 0.5 if nf else m["fz"]
    h = lambda x: 1.0 + 0.1 * np.sin(x[:, 0] + 2 * x[:, 1]) + 0.01 * rng.uniform()
    return dict(m, fs=sig, vh=h(m["vx"]), fh=h(m["fx"]))


RK_DT = {2: 0.02, 3: 0.01, 4: 0.01, 5: 0.005, 6: 0.005, 7: 0.002}


def _network(seed):
    """Weights of the size and scale an initialised network has, and the
    input normalisation; a small output scale, as the residual has."""
    rng = _rng(seed)
    w = np.zeros(NPARAM, np.float32)
    o = 0
    for rows, cols, live, bias in ((128, 48, 127, 40), (128, 128, 127, 127), (128, 128, 127, 127),
                                   (16, 128, 3, 127)):
        k = 1.0 / math.sqrt(40 if cols == 48 else 127)
        a = rng.uniform(-k, k, (rows, cols))
        a[live:] = 0.0
        a[:, bias] = 0.0
        w[o:o + a.size] = a.ravel()
        o += a.size
    norm = np.zeros(NNORM, np.float32)
    norm[48:48 + 41] = 1.0
    norm[96] = 1e-3
    return w, norm


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sums":
        ctx = _ctx(case["prec"])
        m = _mesh(case, seed)
        nd = m["vx"].shape[1]
        if case["ntgt"]:
            x = m["rng"].normal(size=(case["ntgt"], nd))
            m["vx"] = (x / np.linalg.norm(x, axis=1, keepdims=True) if nd == 3
                       else m["rng"].uniform(-PLANE_RADIUS, PLANE_RADIUS, x.shape))
        soa = case["soa"]
        s = dict(case=case, ctx=ctx, x=_up(m["vx"], soa), y=_up(m["fx"], soa), z=_up(m["fz"]),
                 a=_up(m["fa"]), m=_up(m["fm"]))
        for k, n in (("x", len(m["vx"])), ("y", len(m["fx"]))):
            s["u" + k] = _up(np.zeros((n, nd)), soa)
            s["p" + k] = _up(np.zeros(n)) if case["psi"] else None
        return s
    if kind == "rk4":
        ctx = _ctx(case["prec"])
        sph = _bve(case, seed, ctx)
        _bve_velocity(sph, ctx, case["eps"])
        flags = MASKED | (core.STEP_REPROJECT if case["reproject"] else 0)
        st = BVERK4(RK_DT[case["level"]], sph, precision=PREC[case["prec"]], eps=case["eps"],
                    flags=flags)
        return dict(case=case, sph=sph, st=st)
    if kind == "rk2":
        ctx = _ctx(case["prec"])
        ic = Incompressible2D(MESH[case["mesh"]], case["level"], radius=PLANE_RADIUS
                              if case["mesh"] == "quad" else 1.0, eps=case["eps"],
                              coriolis=(0.0, 0.1) if case["mesh"] == "quad" else None, ctx=ctx)
        m = _mesh(case, seed)
        ic.vert_x, ic.face_x = _up(m["vx"]), _up(m["fx"])
        ic.rel_vort_passive, ic.rel_vort_active = _up(m["vz"]), _up(m["fz"])
        ic.init_direct_sums()
        return dict(case=case, ic=ic, st=Incompressible2DRK2(0.005, ic, precision=PREC[case["prec"]]))
    if kind == "ensemble":
        rng = _rng(seed)
        levels = [case["lo"] + p % (case["hi"] - case["lo"] + 1) for p in range(case["problems"])]
        e = BVEEnsemble(levels, [random_vortex_params(rng) for _ in levels], 0.005, eps=case["eps"],
                        precision=core.FP32C, flags=MASKED | core.STEP_REPROJECT, ctx=_ctx("fp32c"))
        e.velocity()
        return dict(case=case, e=e)
    if kind == "ffvel":
        m = _mesh(case, seed)
        x = _up(np.concatenate([m["vx"], m["fx"][m["fm"] == 0]]))
        return dict(case=case, ff=FarField(theta=case["theta"], ctx=_ctx("chord64")), x=x,
                    u=torch.zeros_like(x), y=_up(m["fx"]), z=_up(m["fz"]), a=_up(m["fa"]),
                    m=_up(m["fm"]))
    if kind == "ffrk4":
        ctx = _ctx("chord64")
        sph = _bve(case, seed, ctx)
        ff = FarField(theta=case["theta"], ctx=ctx, rho_min=min(0.25, case["theta"]))
        if case["net"]:
            ff.set_weights(*_network(seed))
            ff.set_network(True)
        # the velocities of the initial state, FP32 compensated
        _bve_velocity(sph, _ctx("fp32c"), 0.01)
        st = BVERK4(RK_DT[case["level"]], sph, precision=core.FP64_CHORD, eps=0.01,
                    flags=MASKED | core.STEP_REPROJECT)
        st.set_farfield(ff)
        return dict(case=case, sph=sph, st=st, ff=ff)
    if kind == "swe":
        m = _swe_fields(case, seed)
        s = {k: _up(m[k]) for k in ("vx", "fx", "fz", "fs", "fa", "fm", "vh", "fh")}
        return dict(s, case=case, ctx=_ctx(case["prec"]))
    if kind == "grad":
        ff = FarField(ctx=_ctx("fp32c"))
        ff.set_weights(*_network(seed))
        rng = _rng(seed + 1)
        return dict(case=case, ff=ff, x=rng.normal(size=(case["rows"], 48)).astype(np.float32),
                    y=rng.normal(size=(case["rows"], 3)).astype(np.float32))
    raise ValueError(kind)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "sums":
        ctx, src = s["ctx"], (s["y"], s["z"], s["a"], s["m"])
        if s["y"].shape[1] == 3 and case["eps"] == 0.0:
            if case["psi"]:
                F.bve_vertex_solve(ctx, s["px"], s["ux"], s["x"], *src)
                if case["faces"]:
                    F.bve_face_solve(ctx, s["py"], s["uy"], *src)
            else:
                F.bve_vertex_velocity(ctx, s["ux"], s["x"], *src)
                if case["faces"]:
                    F.bve_face_velocity(ctx, s["uy"], *src)
        else:
            F.ic2d_passive_sums(ctx, s["ux"], s["px"], s["x"], *src, case["eps"])
            if case["faces"]:
                F.ic2d_active_sums(ctx, s["uy"], s["py"], *src, case["eps"])
        return [s["ux"], s["px"]] + ([s["uy"], s["py"]] if case["faces"] else [])
    if kind in ("rk4", "ffrk4"):
        sph = s["sph"]
        s["st"].advance_timestep(sph)
        return [sph.vert_x, sph.rel_vort_verts, sph.velocity_verts, sph.face_x, sph.rel_vort_faces,
                sph.velocity_faces]
    if kind == "rk2":
        ic = s["ic"]
        ic.advance_timestep(s["st"])
        return [ic.vert_x, ic.rel_vort_passive, ic.velocity_passive, ic.stream_fn_passive, ic.face_x,
                ic.rel_vort_active, ic.velocity_active, ic.stream_fn_active]
    if kind == "ensemble":
        e = s["e"]
        e.advance_timestep()
        return [e.vx, e.vzeta, e.vvel, e.fx, e.fzeta, e.fvel]
    if kind == "ffvel":
        s["ff"].velocity(s["u"], s["x"], s["y"], s["z"], s["a"], s["m"], 0.01)
        return s["u"]
    if kind == "swe":
        ctx, eps = s["ctx"], case["eps"]
        if s["vx"].shape[1] == 3:
            src = (s["fx"], s["fz"], s["fs"], s["fa"], s["fm"], eps)
            return [F.swe_sphere_vertex_sums(ctx, s["vx"], *src), F.swe_sphere_face_sums(ctx, *src)]
        src = (s["fx"], s["fz"], s["fs"], s["fa"], s["fm"], s["fh"], eps, PSE_EPS)
        return [F.swe_plane_vertex_sums(ctx, s["vx"], s["vh"], *src), F.swe_plane_face_sums(ctx, *src)]
    return s["ff"].grad(s["x"], s["y"])


# ---- what a pass cannot do without ------------------------------------------

def _counts(mesh, level):
    nv, nf = core.mesh_sizes(MESH[mesh], level)
    leaves = {"icos": 20, "cubed": 6, "quad": 4}[mesh] * 4**level
    return nv, nf, leaves


def _sum_work(nt, nf, ns, nd, flops_per_pair, outs):
    return nt * 8 * (nd + outs) + nf * (8 * (nd + 2) + 1), float(nt) * ns * flops_per_pair


def work(case):
    kind = case["kind"]
    if kind == "grad":
        n = case["rows"]
        return {"bytes": n * 4 * 51 + 4 * NPARAM * 2, "flops": 6.0 * n * NPARAM}
    if kind == "ensemble":
        b = f = 0
        for p in range(case["problems"]):
            nv, nf, ns = _counts("icos", case["lo"] + p % (case["hi"] - case["lo"] + 1))
            b += (nv + nf) * 8 * 14
            f += 4.0 * (nv + ns) * ns * 24
        return {"bytes": b, "flops": f}
    mesh = case.get("mesh", "icos")
    nv, nf, ns = _counts(mesh, case["level"])
    nd = 2 if mesh == "quad" else 3
    pair = (16 if nd == 2 else 24)
    if kind == "sums":
        fl = pair + (4 if case["psi"] else 0)
        nt = (case["ntgt"] or nv) + (nf if case["faces"] else 0)
        b, f = _sum_work(nt, nf, ns, nd, fl, nd + case["psi"])
    elif kind == "rk4":
        b, f = (nv + nf) * 8 * 14, 4.0 * (nv + ns) * ns * 24
    elif kind == "rk2":
        b, f = (nv + nf) * 8 * 14, float(nv + nf) * ns * (2 * pair + 4)
    elif kind == "ffvel":
        # every target against the cells and leaves it meets: O(log n) cells
        # of about 250 flops and a neighbourhood of sources
        b, f = _sum_work(nv + ns, nf, 1, nd, 0, 3)
        f = (nv + ns) * (150 * 250.0 + 1500 * 24)
    elif kind == "ffrk4":
        b = (nv + nf) * 8 * 14
        f = 4 * (nv + ns) * (150 * 250.0 + 1500 * 24 + (80 * 2.0 * NPARAM if case["net"] else 0))
    else:
        b, f = _sum_work(nv + nf, nf, ns, nd, 71.0 if nd == 3 else 70.0, 4 if nd == 3 else 10)
    return {"bytes": b, "flops": f}


# ---- the same in plain FP64 ---------------------------------------------------

def _half_defect(x):
    """(1 - |x|^2) / 2 with the squares taken exactly (split products)."""
    c = x * 134217729.0
    hi = c - (c - x)
    lo = x - hi
    s = torch.ones(x.shape[0], dtype=torch.float64, device=x.device)
    e = torch.zeros_like(s)
    for k in range(x.shape[1]):
        p = x[:, k] * x[:, k]
        pe = ((hi[:, k] * hi[:, k] - p) + 2 * hi[:, k] * lo[:, k]) + lo[:, k] * lo[:, k]
        t = s - p
        e = e + ((s - (t + p)) - pe)
        s = t
    return 0.5 * (s + e)


def _pair_sums(x, y, g, eps, psi, chord, own=None):
    """Velocity (and stream function) at x from strengths g at y.  own: source
    index skipped by each target (-1: none).  chord: 1 - x.y taken as
    |x - y|^2 / 2 whatever the lengths."""
    nd = x.shape[1]
    u, p = torch.empty_like(x), torch.empty(x.shape[0], dtype=x.dtype, device=x.device)
    cx, cy = (0.0, 0.0) if chord or nd == 2 else (_half_defect(x), _half_defect(y))
    rows = max(1, int(4e7 // max(1, y.shape[0])))
    for i in range(0, x.shape[0], rows):
        xi = x[i:i + rows]
        d = [xi[:, k:k + 1] - y[None, :, k] for k in range(nd)]
        q = d[0] * d[0]
        for k in range(1, nd):
            q = q + d[k] * d[k]
        if nd == 3:
            q = 0.5 * q
            if not chord:
                q = q + (cx[i:i + rows, None] + cy[None, :])
        q = q + eps * eps
        gq = g[None, :] / q
        lg = torch.log(q) if psi else None
        if own is not None:
            r = (own[i:i + rows] >= 0).nonzero()[:, 0]
            gq[r, own[i:i + rows][r]] = 0.0
            if psi:
                lg[r, own[i:i + rows][r]] = 0.0
        w = [(gq * dk).sum(1) for dk in d]
        if nd == 3:
            u[i:i + rows] = torch.linalg.cross(xi, torch.stack(w, 1)) / (4 * math.pi)
        else:
            u[i:i + rows] = torch.stack([-w[1], w[0]], 1) / (2 * math.pi)
        if psi:
            p[i:i + rows] = -(lg @ g) / (4 * math.pi)
    return u, (p if psi else None)


def _slots(mask):
    """Leaf slots, and for each slot its index among them or -1."""
    leaf = (mask == 0).nonzero()[:, 0]
    own = torch.full((mask.shape[0],), -1, dtype=torch.int64, device=mask.device)
    own[leaf] = torch.arange(leaf.shape[0], device=mask.device)
    return leaf, own


def _exact_rk4(vx, vz, fx, fz, fa, fm, dt, eps, chord, reproject, Omega=2 * math.pi):
    leaf, own = _slots(fm)
    nv = vx.shape[0]
    self_idx = torch.cat([torch.full((nv,), -1, dtype=torch.int64, device=vx.device), own[leaf]])
    area = fa[leaf]

    def velocity(x, zl):
        return _pair_sums(x, x[nv:], zl * area, eps, False, chord, self_idx)[0]

    x0, z0 = torch.cat([vx, fx[leaf]]), torch.cat([vz, fz[leaf]])
    tend = lambda u: -2.0 * Omega * u[:, 2] * dt
    u = velocity(x0, z0[nv:])
    xs, zs = [dt * u], [tend(u)]
    for c in (0.5, 0.5, 1.0):
        u = velocity(x0 + c * xs[-1], (z0 + c * zs[-1])[nv:])
        xs.append(dt * u)
        zs.append(tend(u))
    x = x0 + ((xs[0] + xs[3]) / 6 + (xs[1] + xs[2]) / 3)
    if reproject:
        x = x / x.norm(dim=1, keepdim=True)
    z3 = torch.cat([zs[2][:nv], zs[3][nv:]])  # faces take stage 4 twice, as the reference does
    z = z0 + ((zs[0] + zs[3]) / 6 + (zs[1] + z3) / 3)
    u = velocity(x, z[nv:])
    fx, fz = fx.clone(), fz.clone()
    fu = torch.zeros_like(fx)
    fx[leaf], fz[leaf], fu[leaf] = x[nv:], z[nv:], u[nv:]
    return [x[:nv], z[:nv], u[:nv], fx, fz, fu]


def _exact_rk2(s, case, dt=0.005):
    ic = s["ic"]
    leaf, own = _slots(ic.face_mask)
    nv, area, nd = ic.n_vertices_host(), ic.face_area[leaf], ic.ndim
    chord = case["prec"] != "fp64"
    x = torch.cat([ic.vert_x, ic.face_x])
    z = torch.cat([ic.rel_vort_passive, ic.rel_vort_active])
    f = (lambda u: -2.0 * ic.cor_param * u[:, 2]) if nd == 3 else (lambda u: -ic.cor_param * u[:, 1])

    def sums(x, z, psi):
        return _pair_sums(x, x[nv:][leaf], z[nv:][leaf] * area, case["eps"], psi, chord)

    u, _ = sums(x, z, False)
    x1, z1 = dt * u, f(u)
    u, _ = sums(x + x1, z + dt * z1, False)
    z = z + 0.5 * dt * (z1 + f(u))
    x = x + 0.5 * (x1 + dt * u)
    u, p = sums(x, z, True)
    return [x[:nv], z[:nv], u[:nv], p[:nv], x[nv:], z[nv:], u[nv:], p[nv:]]


def _exact_swe_sphere(x, y, rot, pot, eps):
    u = torch.empty_like(x)
    dd = torch.empty(x.shape[0], dtype=x.dtype, device=x.device)
    cx, cy = _half_defect(x), _half_defect(y)
    eye = torch.eye(3, dtype=x.dtype, device=x.device)
    rows = max(1, int(1e7 // y.shape[0]))
    for i in range(0, x.shape[0], rows):
        xi = x[i:i + rows]
        d = xi[:, None, :] - y[None]
        one_s = 0.5 * (d * d).sum(2) + (cx[i:i + rows, None] + cy[None])  # 1 - x.y
        D = one_s + eps * eps
        i1 = 1.0 / (4 * math.pi * D)
        sz, ss = rot * i1, pot * i1
        R, Q = sz / D, ss / D
        c = -torch.linalg.cross(xi[:, None, :].expand_as(d), d)  # x cross y
        v = eps * eps * xi[:, None, :] + d
        w = one_s[..., None] * xi[:, None, :] - d  # y - (x.y) x
        u[i:i + rows] = (c * sz[..., None] + w * ss[..., None]).sum(1)
        M = torch.einsum("tsi,tsj->tij", c * R[..., None], v) - torch.einsum("tsi,tsj->tij", v * Q[..., None], w)
        Y = (sz[..., None] * y[None]).sum(1)
        z = torch.zeros_like(Y[:, 0])
        M = M + torch.stack([z, -Y[:, 2], Y[:, 1], Y[:, 2], z, -Y[:, 0], -Y[:, 1], Y[:, 0], z], 1).view(-1, 3, 3)
        M = M - (ss * (1.0 - one_s)).sum(1)[:, None, None] * (eye - xi[:, :, None] * xi[:, None, :])
        dd[i:i + rows] = (M * M.transpose(1, 2)).sum((1, 2))
    return {"u": u, "ddot": dd}


def _exact_swe_plane(x, sx, y, rot, pot, area, sy, eps, pse):
    n = x.shape[0]
    o = torch.empty(n, 9, dtype=x.dtype, device=x.device)
    rows = max(1, int(2e7 // y.shape[0]))
    for i in range(0, n, rows):
        d0, d1 = x[i:i + rows, :1] - y[None, :, 0], x[i:i + rows, 1:] - y[None, :, 1]
        r2 = d0 * d0 + d1 * d1
        q = r2 + eps * eps
        a, b = rot / q, pot / q
        ax, bx = a / q, b / q
        p2 = r2 / pse**2
        lap = (40 * (1 - p2) + 10 * p2**2 - (2.0 / 3.0) * p2**3) * torch.exp(-p2) / math.pi
        lg = -torch.log(q) / (4 * math.pi)
        A, B = a.sum(1) / (2 * math.pi), b.sum(1) / (2 * math.pi)
        o[i:i + rows] = torch.stack([
            (b * d0 - a * d1).sum(1) / (2 * math.pi), (a * d0 + b * d1).sum(1) / (2 * math.pi),
            (ax * d0 * d1 - bx * d0 * d0).sum(1) / math.pi + B,
            (ax * d1 * d1 - bx * d0 * d1).sum(1) / math.pi - A,
            (-ax * d0 * d0 - bx * d0 * d1).sum(1) / math.pi + A,
            (-ax * d0 * d1 - bx * d1 * d1).sum(1) / math.pi + B,
            ((sy[None] - sx[i:i + rows, None]) * area * lap).sum(1) / pse**2,
            lg @ rot, lg @ pot], 1)
    return {"u": o[:, :2], "ddot": o[:, 2] ** 2 + 2 * o[:, 3] * o[:, 4] + o[:, 5] ** 2,
            "du1dx1": o[:, 2], "du1dx2": o[:, 3], "du2dx1": o[:, 4], "du2dx2": o[:, 5],
            "laps": o[:, 6], "psi": o[:, 7], "phi": o[:, 8]}


def _exact_grad(s):
    bf = lambda a: torch.from_numpy(a).to(_dev()).to(torch.bfloat16).double()
    w, norm = s["ff"].get_weights()
    p = bf(w).requires_grad_(True)
    h, y, o = bf(s["x"]), torch.from_numpy(s["y"]).to(_dev()).double(), 0
    for rows, cols in ((128, 48), (128, 128), (128, 128), (16, 128)):
        z = h @ p[o:o + rows * cols].view(rows, cols).t()
        o += rows * cols
        if rows == 128:  # unit 127 is the constant 1
            z = torch.nn.functional.silu(z)
            h = torch.cat([z[:, :127], torch.ones_like(z[:, :1])], 1)
    loss = ((z[:, :3] - y) ** 2).sum() / y.shape[0]
    return torch.autograd.grad(loss, p)[0]


def exact(case, seed):
    kind = case["kind"]
    w = work(case)["flops"]
    if kind in ("sums", "rk4", "rk2", "swe", "ensemble") and w / 24 > EXACT_PAIRS:
        return None
    if kind == "ffrk4" or (kind == "ffvel" and case["level"] > 6):
        return None
    if kind in ("rk4", "ensemble"):
        if kind == "rk4":
            m = _mesh(dict(case, mesh="icos"), seed)
            t = [_up(m[k]) for k in ("vx", "vz", "fx", "fz", "fa", "fm")]
            return _exact_rk4(*t, RK_DT[case["level"]], case["eps"], case["prec"] != "fp64",
                              case["reproject"])
        rng = _rng(seed)
        parts = []
        for p in range(case["problems"]):
            vx, fx, fa, fm = core.build_mesh(core.MESH_ICOS_TRI, case["lo"] + p % (case["hi"] - case["lo"] + 1), 1.0)
            prm = random_vortex_params(rng)
            vz, fz = (core.eval_ic(core.IC_MULTI_GAUSSIAN, prm, x) for x in (vx, fx))
            parts.append(_exact_rk4(*(_up(a) for a in (vx, vz, fx, fz, fa, fm)), 0.005, case["eps"],
                                    True, True))
        return [torch.cat(x) for x in zip(*parts)]
    s = prepare(case, seed)
    if kind == "grad":
        return _exact_grad(s)
    if kind == "rk2":
        return _exact_rk2(s, case)
    if kind == "swe":
        leaf, own = _slots(s["fm"])
        y, a = s["fx"][leaf], s["fa"][leaf]
        rot, pot = s["fz"][leaf] * a, s["fs"][leaf] * a
        if y.shape[1] == 3:
            return [_exact_swe_sphere(x, y, -rot, -pot, case["eps"]) for x in (s["vx"], s["fx"])]
        return [_exact_swe_plane(x, h, y, rot, pot, a, s["fh"][leaf], case["eps"], PSE_EPS)
                for x, h in ((s["vx"], s["vh"]), (s["fx"], s["fh"]))]
    leaf, own = _slots(s["m"])
    y, g = s["y"][leaf], (s["z"] * s["a"])[leaf]
    if kind == "ffvel":
        return _pair_sums(s["x"], y, g, 0.01, False, True)[0]
    chord = case["prec"] != "fp64"
    out = list(_pair_sums(s["x"], y, g, case["eps"], case["psi"], chord))
    if case["faces"]:
        out += _pair_sums(s["y"], y, g, case["eps"], case["psi"], chord,
                          own if case["eps"] == 0.0 else None)
    return out
