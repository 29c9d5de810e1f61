"""The work that users of this framework have it do, through its public entry points.

Kinds of calls (``case["kind"]``):

* ``assemble``  one ``assembleLinearSystem`` on a state that is new to the
  context: element assembly, static condensation and scatter, the call every
  Newton iteration of a reference driver makes.  ``source`` says where the state
  is: on the device, or in pinned host memory (``assemble_from_host``).
* ``newton``    ``getQ`` and one step of ``solveNonlinearProblem`` with GMRES.
* ``dirk``      one time step of an unsteady run (three implicit stages).
* ``batch``     one Newton iteration of many independent solves packed into one
  context, the inner call of the solve server.
* ``graph``     one assembly pass over meshes of mixed order as one graph launch.

Sizes are those of the benchmark's tasks and of the solve server's requests
(256 to 16,384 triangles, orders 1 to 3; meshes of orders 1 to 4; tetrahedra up
to order 3), 3D meshes smaller than the benchmark's so that several states fit
a device.  ``exact`` restates the discretisation in plain torch, FP64.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from hfem_b200.batch import BatchSolver
from hfem_b200.batched import MixedOrderAssembly
from hfem_b200.core import HDGSolver
from hfem_b200.gen.master import make_master
from hfem_b200.gen.mesh import build_mesh
from hfem_b200.gen.problem import Problem, ns2d_channel, ns3d_box, ns3d_tgv, with_models
from hfem_b200.gen.state import init_uhat, make_udg

F64 = torch.float64


# ------------------------------------------------------------------- the cases
def _assemble(name, nd, p, n, bounded=False, stab=0, visc=0, mode=0, source="device"):
    return dict(name=name, kind="assemble", nd=nd, p=p, n=n, bounded=bounded, stab=stab, visc=visc, mode=mode,
                source=source)


def listed():
    return [
        # the smallest solves of a server: a few hundred linear triangles, bound by launches and latency
        _assemble("assemble 2d p1 288", 2, 1, 12),
        # the 2D benchmark mesh, 32 x 32 x 2 quadratic triangles
        _assemble("assemble 2d p2 2048", 2, 2, 32),
        # a walled channel with the Roe tensor and Sutherland's law, cubic triangles on an odd grid
        _assemble("assemble 2d p3 channel roe", 2, 3, 45, bounded=True, stab=2, visc=1),
        # a large mesh of the highest order
        _assemble("assemble 2d p4 7938", 2, 4, 63),
        # 3D flow on quadratic tetrahedra, the state arriving from host memory each pass
        _assemble("assemble 3d p2 host", 3, 2, 9, source="host"),
        # the headline workload's elements (cubic tetrahedra), FP64
        _assemble("assemble 3d p3 13182", 3, 3, 13),
        # the same elements in mixed precision
        _assemble("assemble 3d p3 mixed", 3, 3, 9, mode=1),
        # one Newton step of the 2D benchmark mesh, block-Jacobi GMRES
        dict(name="newton 2d p2 bj", kind="newton", nd=2, p=2, n=32, bounded=False, stab=0, visc=0, precond=2, mode=0),
        # the same step with the BILU0 preconditioner
        dict(name="newton 2d p2 bilu0", kind="newton", nd=2, p=2, n=32, bounded=False, stab=0, visc=0, precond=0,
             mode=0),
        # a Taylor-Green time step, DIRK(3,3), FP32 preconditioner with FP64 refinement
        dict(name="dirk 3d p3 tgv", kind="dirk", p=3, n=6, mode=2),
        # one iteration of the solve server's quadratic group: eight requests of uneven size
        dict(name="batch 2d p2 x8", kind="batch", p=2, count=8, lo=256, hi=2048, mix=11),
        # meshes of orders 1 to 4 and uneven size in one graph
        dict(name="graph 2d p1-4 x12", kind="graph", count=12, lo=256, hi=4096, mix=5),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["assemble"] * 6 + ["newton"] * 3 + ["batch", "graph", "dirk"])
    if kind in ("assemble", "newton"):
        nd = rng.choice([2, 2, 3])
        p = rng.choice([1, 2, 3, 4] if nd == 2 else [1, 2, 3])
        if kind == "assemble":
            top = {(2, 1): 100, (2, 2): 90, (2, 3): 75, (2, 4): 60, (3, 1): 16, (3, 2): 13, (3, 3): 11}[nd, p]
        else:
            top = {(2, 1): 48, (2, 2): 40, (2, 3): 24, (2, 4): 20, (3, 1): 8, (3, 2): 6, (3, 3): 5}[nd, p]
        n = max(3, round(_log(rng, 10 if nd == 2 else 3, top)))
        bounded = rng.random() < 0.3
        stab, visc = (rng.choice([(2, 0), (2, 1), (1, 0), (0, 1)]) if rng.random() < 0.3 else (0, 0))
        c = dict(kind=kind, nd=nd, p=p, n=n, bounded=bounded, stab=stab, visc=visc, re=round(_log(rng, 50, 500), 2))
        if kind == "assemble":
            return dict(c, mode=rng.choice([0, 0, 0, 1, 3]), source=rng.choice(["device", "device", "host"]))
        return dict(c, bounded=False, precond=2 if nd == 3 or rng.random() < 0.7 else 0, mode=rng.choice([0, 0, 2]))
    if kind == "dirk":
        return dict(kind=kind, p=rng.choice([1, 2, 3]), n=rng.choice([3, 4, 5]), mode=rng.choice([0, 2]),
                    dt=round(_log(rng, 0.003, 0.03), 4))
    hi = rng.choice([1024, 2048, 4096])
    c = dict(kind=kind, count=rng.randint(2, 12), lo=256, hi=hi, mix=rng.randint(0, 10 ** 6))
    return c if kind == "graph" else dict(c, p=rng.choice([1, 2, 3]))


# ------------------------------------------------------------------ the inputs
@functools.lru_cache(maxsize=64)
def _grid(nd, p, n, length, bounded):
    m = make_master(nd, p)
    return m, build_mesh(m, n, length, periodic=not bounded)


def _physics(nd, p, n, bounded, stab, visc, seed, mach=None, re=None):
    """A problem of the generator's kinds on a cached grid, its state from the seed."""
    length, dt = (10.0, 0.1) if nd == 2 else (1.0, 0.01)
    m, mesh = _grid(nd, p, n, length, bounded)
    mach = mach or (0.5 if nd == 2 else 0.3)
    re = re or (100.0 if nd == 2 else 400.0)
    if nd == 2:
        udg = make_udg(m, mesh, "vortex", 1.4, mach, seed=seed, noise=1e-3, centre=(5.0, 5.0))
    else:
        udg = make_udg(m, mesh, "fourier", 1.4, mach, seed=seed)
    sh = np.zeros_like(udg)
    sh[:, :nd + 2] = udg[:, :nd + 2] / dt
    prob = Problem(name="case", master=m, mesh=mesh, param=np.array([1.4, 0.0, re, 0.72, mach, 2.0]), tdep=1,
                   fc_u=1.0 / dt, fc_q=1.0, time=0.0, udg=udg, uh=init_uhat(m, mesh, udg), sh=sh, dt=dt)
    if bounded:
        few = (ns2d_channel if nd == 2 else ns3d_box)(n=1, porder=1, mach=mach)
        prob.bcm, prob.bcs = few.bcm, few.bcs
    return with_models(prob, conv_stab=stab, viscosity_model=visc)


def _tgv(case, seed):
    p = ns3d_tgv(n=case["n"], porder=case["p"])
    noise = np.random.default_rng(seed).uniform(-1e-4, 1e-4, size=p.udg[:, :5].shape)
    p.udg[:, :5] += noise * np.abs(p.udg[:, :5]).max()
    p.uh = init_uhat(p.master, p.mesh, p.udg)
    p.sh[:] = 0.0
    return p


def _mix(case, seed):
    """Uneven independent problems, as requests arrive: sizes, Re and Mach from the mix, states from the seed."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for i in range(case["count"]):
        ne = math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
        order = case.get("p") or 1 + i % 4
        out.append(_physics(2, order, max(3, round(math.sqrt(ne / 2))), False, 0, 0, 1000 * seed + i,
                            mach=float(rng.uniform(0.2, 0.7)), re=float(rng.uniform(50, 500))))
    return out


def _problems(case, seed):
    if case["kind"] == "dirk":
        return [_tgv(case, seed)]
    if case["kind"] in ("batch", "graph"):
        return _mix(case, seed)
    return [_physics(case["nd"], case["p"], case["n"], case["bounded"], case["stab"], case["visc"], seed,
                     re=case.get("re"))]


def prepare(case, seed):
    probs = _problems(case, seed)
    kind = case["kind"]
    for p in probs:
        if kind in ("assemble", "graph"):          # a state as a time step leaves it: q consistent with u and uhat
            u, uh, sh = (torch.as_tensor(a, device="cuda") for a in (p.udg, p.uh, p.sh))
            p.udg = _with_q(_tables(p, "cuda"), p, u, uh, sh).cpu().numpy()
    st = dict(kind=kind, case=case, views=None)
    if kind == "graph":
        st["graph"] = MixedOrderAssembly(probs, tune=False)
        groups = [b.s for b in st["graph"].solvers]
    elif kind == "batch":
        st["batch"] = BatchSolver(probs)
        groups = [st["batch"].s]
    else:
        s = HDGSolver(probs[0])
        s.set_precision(case["mode"])
        groups = [s]
    st["solvers"] = groups
    place = (lambda a: torch.from_numpy(a).pin_memory()) if case.get("source") == "host" else \
        (lambda a: torch.as_tensor(a, device="cuda"))
    st["inputs"] = [tuple(place(np.ascontiguousarray(a)) for a in (s.prob.udg, s.prob.uh, s.prob.sh)) for s in groups]
    return st


def _views(st, names):
    """The contexts' device buffers, taken once as a program that keeps a context does.  A view does not own its
    memory, so each one carries the context (and the graph or batch around it) it belongs to."""
    if st["views"] is None:
        st["views"] = [{k: s.device_tensor(k) for k in names} for s in st["solvers"]]
        for s, group in zip(st["solvers"], st["views"]):
            for t in group.values():
                t.owner = (s, st.get("graph"), st.get("batch"))
    return st["views"]


SYSTEM = ("Hg", "Rg", "DinvF", "DinvRu")


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "assemble":
        s = st["solvers"][0]
        ptrs = [t.data_ptr() for t in st["inputs"][0]]
        if case["source"] == "host":
            rn = s.assemble_from_host(*ptrs)
        else:
            s.set_solution_device(*ptrs)
            rn = s.assembleLinearSystem()
        return {"rnorm": rn, **_views(st, SYSTEM)[0]}
    for s, inp in zip(st["solvers"], st["inputs"]):
        s.set_solution_device(*[t.data_ptr() for t in inp])
    if kind == "graph":
        st["graph"].launch()
        return {"rnorm": st["graph"].finish(), "systems": _views(st, SYSTEM)}
    s = st["solvers"][0]
    if kind == "dirk":
        p = s.prob
        s.set_physics(p.param, p.tdep, p.fc_u, p.fc_q, 0.0)
    s.getQ()
    if kind == "newton":
        _, hist = s.solveNonlinearProblem(newton_tol=1e-10, maxiter=1, precond=case["precond"])
        out = {"rnorms": hist}
    elif kind == "batch":
        b = st["batch"]
        old, new = b.newton_iteration(1e-10, np.ones(b.n, dtype=bool))
        out = {"rnorms": np.stack([old, new])}
    else:
        s.solveUnsteadyStep(case.get("dt", s.prob.dt))
        out = {}
    return {**out, **_views(st, ("udg", "uh"))[0]}


# -------------------------------------------------------------------- the work
def _counts(nd, p, ne, nf, nblk):
    """Bytes and FLOPs of one assembly: inputs read, the condensed system and the update's blocks written once;
    element quadrature, LU and the two condensation products.  Also the bytes of the block matrix and one vector."""
    m = make_master(nd, p)
    ncu, ndf = nd + 2, m.npf * m.nfe
    n, nb, bsz = m.npv * ncu, ncu * ndf, ncu * m.npf
    nc = ncu * (nd + 1)
    flops = 2.0 * m.npv * m.ngv * (nd + 1) * ncu * (1 + ncu * m.npv + ncu * ndf) \
        + 2.0 * m.npf * m.ngf * m.nfe * ncu * ncu * (2 * m.npf + m.npv + ndf) \
        + (2.0 / 3.0) * n ** 3 + 2.0 * n * n * nb + 2.0 * nb * nb * n + 2.0 * n * n + 2.0 * nb * n
    state = 8.0 * (2 * ne * m.npv * nc + ne * m.npv * nd + nf * bsz)
    system = 8.0 * (nblk * bsz * bsz + nf * bsz + ne * n * (nb + 1))
    return flops * ne, state, system, 8.0 * nblk * bsz * bsz, 8.0 * nf * bsz


# GMRES iterations of one Newton step on these workloads (block Jacobi, BILU0) and Newton iterations of a DIRK step
ITS_BJ, ITS_BILU0, DIRK_NEWTON = 60, 13, 6


def work(case):
    kind = case["kind"]
    if kind in ("batch", "graph"):
        rng = np.random.default_rng(case["mix"])
        sizes = []
        for i in range(case["count"]):
            ne = math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
            rng.uniform(size=2)
            n = max(3, round(math.sqrt(ne / 2)))
            sizes.append((2, case.get("p") or 1 + i % 4, 2 * n * n))
    else:
        nd = 3 if kind == "dirk" else case["nd"]
        sizes = [(nd, case["p"], (2 if nd == 2 else 6) * case["n"] ** nd)]
    b = f = 0.0
    for nd, p, ne in sizes:
        nf = ne * (nd + 1) // 2
        fl, state, system, mat, vec = _counts(nd, p, ne, nf, nf * (2 * nd + 1))
        if kind in ("assemble", "graph"):
            f, b = f + fl, b + state + system
            continue
        its = ITS_BILU0 if case.get("precond") == 0 else ITS_BJ
        steps = DIRK_NEWTON if kind == "dirk" else 1
        # per Newton iteration: two state passes, the system written and read once, one matrix product per iteration
        b += steps * (2 * state + 2 * system + its * (mat + vec))
        f += steps * (fl + its * mat / 4.0)
    return {"bytes": b, "flops": f}


# ------------------------------------------------- the discretisation in 64 bits
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _tables(p, dev):
    """Geometry, basis tables and the q-equation matrices of every element."""
    m, me = p.master, p.mesh
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device=dev)  # noqa: E731
    nd, perm = m.nd, torch.as_tensor(m.perm.astype(np.int64), device=dev)
    phi, phig, psi, psig = t(m.shapvl), t(m.shapvg), t(m.shapfc), t(m.shapfg)      # (node, point, deriv)
    x = t(me.dgnodes)                                                              # (ne, nd, npv)
    J = torch.einsum("eda,agr->egdr", x, phi[:, :, 1:])
    jac = torch.linalg.det(J)
    X = torch.linalg.inv(J).transpose(2, 3) * jac[..., None, None]                 # X[d, r] = jac dxi_r/dx_d
    xf = x[:, :, perm]                                                             # (ne, nd, nfe, npf)
    T = torch.einsum("edfm,mqr->efqdr", xf, psi[:, :, 1:])
    nv = torch.stack([T[..., 1, 0], -T[..., 0, 0]], -1) if nd == 2 else torch.linalg.cross(T[..., 0], T[..., 1])
    jf = nv.norm(dim=-1)
    nl = nv / jf[..., None]
    M = p.fc_q * torch.einsum("bg,ag,eg->eba", phig[:, :, 0], phi[:, :, 0], jac)
    C = torch.einsum("bgr,ag,egdr->edba", phig[:, :, 1:], phi[:, :, 0], X)
    Ef = torch.einsum("kq,jq,efq,efqd->edfkj", psig[:, :, 0], psi[:, :, 0], jf, nl)
    ne, npv, ndf = me.ne, m.npv, m.npf * m.nfe
    E = torch.zeros(ne, nd, npv, ndf, dtype=F64, device=dev)
    for f in range(m.nfe):
        E[:, :, perm[f], f * m.npf:(f + 1) * m.npf] = Ef[:, :, f]
    MC = torch.linalg.solve(M[:, None], torch.cat([C, E], -1))
    return dict(nd=nd, perm=perm, phi=phi, phig=phig, psi=psi, psig=psig, jac=jac, X=X, jf=jf, nl=nl, M=M,
                MC=MC[..., :npv], ME=MC[..., npv:], elcon=torch.as_tensor(me.elcon.astype(np.int64), device=dev))


def _with_q(T, p, udg, uh, sh):
    """udg with q = sh_q + M^-1 (C u - E uhat) on every element."""
    nd, ncu = T["nd"], T["nd"] + 2
    ne, _, npv = udg.shape
    u, uhe = udg[:, :ncu], uh[T["elcon"]]
    q = torch.einsum("edba,eca->edcb", T["MC"], u) - torch.einsum("edbf,efc->edcb", T["ME"], uhe)
    q = q + sh[:, ncu:].reshape(ne, nd, ncu, npv) / p.fc_q
    return torch.cat([u, q.reshape(ne, nd * ncu, npv)], 1)


def _viscosity(P, w, nd):
    gam, mach, S, T0, b = P[0], P[4], 111.0, 300.0, 100.0
    ke = (w[..., 1:nd + 1] ** 2).sum(-1)
    Tm = (w[..., nd + 1] - 0.5 * ke / w[..., 0]) / (gam * (gam - 1) * mach * mach * w[..., 0])
    a = (S + T0) * Tm ** 1.5 / (S + T0 * Tm)
    return 0.5 - math.atan(b) / math.pi + a * (torch.atan(b * a) / math.pi + 0.5)


def _flux(P, w, nd, visc):
    """Navier-Stokes flux (..., nd, ncu) of w = (u, q_1, ..., q_nd)."""
    ncu, gam, re, pr = nd + 2, P[0], P[2], P[3]
    r, mom, E = w[..., 0], w[..., 1:nd + 1], w[..., nd + 1]
    q = w[..., ncu:].reshape(*w.shape[:-1], nd, ncu)
    v = mom / r[..., None]
    p = (gam - 1) * (E - 0.5 * (v * mom).sum(-1))
    dv = (q[..., 1:nd + 1] - v[..., None, :] * q[..., :1]) / r[..., None, None]      # [d, i] = dv_i/dx_d
    eye = torch.eye(nd, dtype=F64, device=w.device)
    div = dv.diagonal(dim1=-2, dim2=-1).sum(-1)
    mu = _viscosity(P, w, nd)[..., None, None] if visc else 1.0
    tau = mu * (dv + dv.transpose(-1, -2) - (2.0 / 3.0) * div[..., None, None] * eye) / re
    fm = v[..., :, None] * mom[..., None, :] + p[..., None, None] * eye + tau
    heat = q[..., nd + 1] / r[..., None] - E[..., None] * q[..., 0] / (r * r)[..., None] - (dv * v[..., None, :]).sum(-1)
    fe = (E + p)[..., None] * v + (tau * v[..., None, :]).sum(-1) \
        + gam / (re * pr) * (mu[..., 0] if visc else 1.0) * heat
    return torch.cat([mom[..., None], fm, fe[..., None]], -1)


def _stab(P, nl, uh, v, nd, method):
    """The stabilization tensor at uh applied to v: constant, Lax-Friedrichs or Roe."""
    if method == 0:
        return P[5] * v
    gam, g1, b = P[0], P[0] - 1.0, 10.0
    if method == 1 and nd == 2:            # the 2D Lax-Friedrichs routine evaluates a fixed state
        st = torch.tensor([1.0, 0.9994, 0.0349, 1.7858e4], dtype=F64, device=v.device).expand_as(uh)
        uh = st
    r, uv = uh[..., 0], uh[..., 1:nd + 1] / uh[..., :1]
    af, un = 0.5 * (uv ** 2).sum(-1), (nl * uv).sum(-1)
    p = g1 * (uh[..., nd + 1] - r * af)
    c2 = gam * p / r
    c = torch.sqrt(c2)
    if method == 1:
        return torch.where(un >= 0, un + c, c - un)[..., None] * v
    h = uh[..., nd + 1] / r + p / r
    smooth = lambda x: 2.0 * (x * (torch.atan(b * x) / math.pi + 0.5) - math.atan(b) / math.pi + 0.5) - x  # noqa: E731
    l1, l2, l3 = smooth(un + c), smooth(un - c), smooth(un)
    s1, s2 = 0.5 * (l1 + l2) - l3, 0.5 * (l1 - l2)
    av = af * v[..., 0] - (uv * v[..., 1:nd + 1]).sum(-1) + v[..., nd + 1]
    bv = (nl * v[..., 1:nd + 1]).sum(-1) - un * v[..., 0]
    c1, c3 = g1 * s1 * av / c2 + s2 * bv / c, g1 * s2 * av / c + s1 * bv
    one = torch.ones_like(r)
    return l3[..., None] * v + c1[..., None] * torch.cat([one[..., None], uv, h[..., None]], -1) \
        + c3[..., None] * torch.cat([torch.zeros_like(one)[..., None], nl.expand_as(uv), un[..., None]], -1)


def _fhat(p, z, nl, nd):
    """Trace flux of z = (u, q, uh)."""
    ncu = nd + 2
    nc = ncu * (nd + 1)
    u, q, uh = z[..., :ncu], z[..., ncu:nc], z[..., nc:]
    f = _flux(p.param, torch.cat([uh, q], -1), nd, p.viscosity_model)
    return (f * nl[..., None]).sum(-2) + _stab(p.param, nl, uh, u - uh, nd, p.conv_stab)


def _fbou(p, z, nl, nd, kind, ui):
    """Boundary flux of z = (u, q, uh): no-slip wall 2, Dirichlet 5, extrapolation 6, slip wall 7."""
    ncu = nd + 2
    u, uh = z[..., :ncu], z[..., ncu * (nd + 1):]
    if kind == 5:
        return p.param[5] * (ui - uh)
    if kind == 6:
        return u - uh
    if kind == 7:
        mom = u[..., 1:nd + 1]
        return torch.cat([u[..., :1], mom - nl * (nl * mom).sum(-1, keepdim=True), u[..., nd + 1:]], -1) - uh
    if kind == 2:
        return torch.cat([u[..., :1] - uh[..., :1], -uh[..., 1:nd + 1], _fhat(p, z, nl, nd)[..., nd + 1:]], -1)
    raise ValueError(f"boundary condition {kind}")


def _jacobian(f, z):
    """f(z) and its derivative along every component of z (last axis), by forward mode."""
    cols, val = [], None
    for k in range(z.shape[-1]):
        t = torch.zeros_like(z)
        t[..., k] = 1.0
        val, d = torch.func.jvp(f, (z,), (t,))
        cols.append(d)
    return val, torch.stack(cols, -1)


def _blocks(p, T, udg, uh, sh, e0, e1):
    """Element blocks D, F, K, H, Ru, Rh of elements e0..e1-1, and Rh with fhat on every face."""
    nd, perm, phi, phig, psi, psig = (T[k] for k in ("nd", "perm", "phi", "phig", "psi", "psig"))
    ncu, npv = nd + 2, phi.shape[0]
    nc, ndf = ncu * (nd + 1), T["elcon"].shape[1]
    nfe, npf = perm.shape
    s = slice(e0, e1)
    ne, nd1 = e1 - e0, nd + 1
    jac, X, jf, nl, w = T["jac"][s], T["X"][s], T["jf"][s], T["nl"][s], udg[s]
    uhe = uh[T["elcon"][s]]
    # volume
    wg = torch.einsum("eca,ag->egc", w, phi[:, :, 0])
    src = torch.einsum("eca,ag->egc", sh[s, :ncu], phi[:, :, 0]) - p.fc_u * wg[..., :ncu]
    f, df = _jacobian(lambda z: _flux(p.param, z, nd, p.viscosity_model), wg)
    pulled = torch.cat([(src * jac[..., None])[:, :, None], torch.einsum("egdj,egdr->egrj", f, X)], 2)
    dsrc = torch.zeros(ne, jac.shape[1], ncu, nc, dtype=F64, device=w.device)
    for j in range(ncu):
        dsrc[..., j, j] = -p.fc_u
    dpull = torch.cat([(dsrc * jac[..., None, None])[:, :, None], torch.einsum("egdjc,egdr->egrjc", df, X)], 2)
    Ru = torch.einsum("igr,egrj->eji", phig, pulled)                               # row i + npv j
    Y = -torch.einsum("igr,egrjc->eigjc", phig, dpull)
    Y = Y.reshape(ne, npv, Y.shape[2], ncu, nd1, ncu)                              # (e, i, g, j, d', k)
    dphi = torch.einsum("edba,bg->egda", T["MC"][s], phi[:, :, 0])
    dpsi = -torch.einsum("edbf,bg->egdf", T["ME"][s], phi[:, :, 0])
    Phi = torch.cat([phi[:, :, 0].T[None, :, None].expand(ne, -1, 1, -1), dphi], 2)
    D = torch.einsum("eigjdk,egda->ejika", Y, Phi)               # rows (j, i), cols (k, a)
    F = torch.einsum("eigjdk,egdf->ejifk", Y[:, :, :, :, 1:], dpsi)                # cols (f2, k)
    # faces
    wf = torch.einsum("ecfm,mq->efqc", w[:, :, perm], psi[:, :, 0])
    uhq = torch.einsum("efmc,mq->efqc", uhe.reshape(ne, nfe, npf, ncu), psi[:, :, 0])
    z = torch.cat([wf, uhq], -1)
    fh, dfh = _jacobian(lambda y: _fhat(p, y, nl, nd), z)
    rows = [(fh, dfh)]
    if p.bcm is not None:
        fb, dfb = fh.clone(), dfh.clone()
        bf = torch.as_tensor(p.mesh.bf[e0:e1], device=w.device)
        for ib, kind in enumerate(p.bcm):
            on = bf == -(ib + 1)
            if on.any():
                ui = torch.as_tensor(p.bcs[ib], dtype=F64, device=w.device)
                fb[on], dfb[on] = _jacobian(lambda y: _fbou(p, y, nl[on], nd, int(kind), ui), z[on])
        rows.append((fb, dfb))
    sel = torch.zeros(nfe, npf, npv, dtype=F64, device=w.device)
    for fc in range(nfe):
        sel[fc, torch.arange(npf), perm[fc]] = 1.0
    phin = torch.einsum("fma,mq->fqa", sel, psi[:, :, 0])                           # element basis on face points
    dphif = torch.einsum("edba,fqb->efqda", T["MC"][s], phin)
    dpsif = -torch.einsum("edbg,fqb->efqdg", T["ME"][s], phin)
    own = torch.zeros(nfe, psi.shape[1], ndf, dtype=F64, device=w.device)
    for fc in range(nfe):
        own[fc, :, fc * npf:(fc + 1) * npf] = psi[:, :, 0].T
    PhiF = torch.cat([phin[None, :, :, None].expand(ne, -1, -1, 1, -1), dphif], 3)
    out = []
    for val, der in rows:
        val, der = val * jf[..., None], der * jf[..., None, None]
        A = der[..., :nc].reshape(ne, nfe, -1, ncu, nd1, ncu)
        Rh = -torch.einsum("mq,efqj->efmj", psig[:, :, 0], val)
        K = torch.einsum("mq,efqjdk,efqda->efmjka", psig[:, :, 0], A, PhiF)
        H = torch.einsum("mq,efqjdk,efqdg->efmjgk", psig[:, :, 0], A[:, :, :, :, 1:], dpsif) \
            + torch.einsum("mq,efqjk,fqg->efmjgk", psig[:, :, 0], der[..., nc:], own)
        out.append((Rh.reshape(ne, ndf, ncu), K.reshape(ne, ndf, ncu, ncu, npv), H.reshape(ne, ndf, ncu, ndf, ncu)))
    lift = sel.reshape(ndf, npv)                                                   # trace dof -> element node
    Rh, K, H = out[0]
    Ru = Ru + torch.einsum("fi,efj->eji", lift, Rh)
    D = D + torch.einsum("fi,efjka->ejika", lift, K)
    F = F + torch.einsum("fi,efjgk->ejigk", lift, H)
    Rh, K, H = out[-1]
    n, nb = npv * ncu, ndf * ncu
    return (D.reshape(ne, n, n), F.reshape(ne, n, nb), K.reshape(ne, nb, n), H.reshape(ne, nb, nb), Ru.reshape(ne, n),
            Rh.reshape(ne, nb))


def _system(p, udg, uh, sh, condense=True):
    """The condensed system of one problem, laid out as the context's buffers."""
    dev = udg.device
    T = _tables(p, dev)
    me, m = p.mesh, p.master
    ncu, nb, bsz = m.nd + 2, p.n_trace, p.bsz
    t2f = torch.as_tensor(me.t2f.astype(np.int64), device=dev)
    rs, ci = (torch.as_tensor(a.astype(np.int64), device=dev) for a in (me.rowstart, me.colidx))
    key = torch.repeat_interleave(torch.arange(me.nf, device=dev), rs[1:] - rs[:-1]) * me.nf + ci
    skey, order = key.sort()
    out = dict(DinvF=[], DinvRu=[])
    Hg = torch.zeros(ci.numel(), bsz, bsz, dtype=F64, device=dev)                   # block k: [column, row]
    Rg, Rr = (torch.zeros(me.nf * bsz, dtype=F64, device=dev) for _ in range(2))
    ru2 = torch.zeros((), dtype=F64, device=dev)
    step = max(1, int(2e8) // (p.n_local * nb * 8))
    for e0 in range(0, me.ne, step):
        e1 = min(me.ne, e0 + step)
        D, F, K, H, Ru, Rh = _blocks(p, T, udg, uh, sh, e0, e1)
        dof = (T["elcon"][e0:e1, :, None] * ncu + torch.arange(ncu, device=dev)).reshape(e1 - e0, nb)
        ru2 += (Ru ** 2).sum()
        Rr.index_add_(0, dof.reshape(-1), Rh.reshape(-1))
        if not condense:
            continue
        sol = torch.linalg.solve(D, torch.cat([F, Ru[..., None]], -1))
        X, y = sol[..., :nb], sol[..., nb]
        H = H - K @ X
        Rg.index_add_(0, dof.reshape(-1), (Rh - (K @ y[..., None])[..., 0]).reshape(-1))
        out["DinvF"].append(X.transpose(1, 2).reshape(-1))
        out["DinvRu"].append(y.reshape(-1))
        loc = dof % bsz
        for a in range(m.nfe):
            for b in range(m.nfe):
                k = order[torch.searchsorted(skey, t2f[e0:e1, a] * me.nf + t2f[e0:e1, b])]
                r, c = loc[:, a * bsz:(a + 1) * bsz], loc[:, b * bsz:(b + 1) * bsz]
                blk = H[:, a * bsz:(a + 1) * bsz, b * bsz:(b + 1) * bsz].transpose(1, 2)
                flat = (k[:, None, None] * bsz + c[:, :, None]) * bsz + r[:, None, :]
                Hg.view(-1).index_add_(0, flat.reshape(-1), blk.reshape(-1))
    res = {k: torch.cat(v) for k, v in out.items() if v}
    return dict(res, Hg=Hg.reshape(-1), Rg=Rg, rnorm=float((ru2 + (Rr ** 2).sum()).sqrt()), T=T, key=key)


def _state(p, dev):
    return [torch.as_tensor(a, dtype=F64, device=dev) for a in (p.udg, p.uh, p.sh)]


def _newton_step(p, dev):
    """One full Newton step with a direct solve: the new state and the residual norms around it."""
    udg, uh, sh = _state(p, dev)
    T = _tables(p, dev)
    udg = _with_q(T, p, udg, uh, sh)
    S = _system(p, udg, uh, sh)
    me, bsz, ncu = p.mesh, p.bsz, p.nd + 2
    A = torch.zeros(me.nf, bsz, me.nf, bsz, dtype=F64, device=dev)
    A[S["key"] // me.nf, :, S["key"] % me.nf] = S["Hg"].view(-1, bsz, bsz).transpose(1, 2)
    x = torch.linalg.solve(A.view(me.nf * bsz, -1), S["Rg"]).view(-1, ncu)
    del A
    xe = x[T["elcon"]].reshape(me.ne, -1)
    du = S["DinvRu"].view(me.ne, -1) - torch.einsum("ecn,ec->en", S["DinvF"].view(me.ne, xe.shape[1], -1), xe)
    uh = uh + x
    udg[:, :ncu] += du.view(me.ne, ncu, -1)
    udg = _with_q(T, p, udg, uh, sh)
    return udg, uh, S["rnorm"], _system(p, udg, uh, sh, condense=False)["rnorm"]


DENSE = 38000       # most trace unknowns solved densely


def exact(case, seed):
    dev, probs = _device(), _problems(case, seed)
    kind = case["kind"]
    if kind == "dirk" or dev == "cpu" and sum(p.mesh.ne for p in probs) > 4000:
        return None
    if kind in ("newton", "batch"):
        if max(p.mesh.nf * p.bsz for p in probs) > DENSE or sum((p.mesh.nf * p.bsz) ** 3 for p in probs) > 1.5 * DENSE ** 3:
            return None
        got = [_newton_step(p, dev) for p in probs]
        norms = np.array([[g[2], g[3]] for g in got]).T
        return {"rnorms": norms[:, 0] if kind == "newton" else norms,
                "udg": torch.cat([g[0].reshape(-1) for g in got]), "uh": torch.cat([g[1].reshape(-1) for g in got])}
    systems = []
    for p in probs:
        udg, uh, sh = _state(p, dev)
        systems.append(_system(p, _with_q(_tables(p, dev), p, udg, uh, sh), uh, sh))
    if kind == "assemble":
        return {"rnorm": systems[0]["rnorm"], **{k: systems[0][k] for k in SYSTEM}}
    order = sorted({p.master.porder for p in probs})
    return {"rnorm": np.array([s["rnorm"] for s in systems]),
            "systems": [{k: torch.cat([s[k] for s, p in zip(systems, probs) if p.master.porder == o]) for k in SYSTEM}
                        for o in order]}
