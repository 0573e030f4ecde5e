"""What this engine is timed on, through its public entry points.

A case names a mesh family, a size, a scheme, a precision form and what is
asked of the engine:

``march``     the state in, CFL time steps and SSP-RK3 steps, the state out
``residual``  one residual of a new state
``gradient``  a new state, its residual's VJP (with the free-stream
              gradient) and JVP
``adjoint``   a checkpointed adjoint run of a scalar output
``implicit``  pseudo-time steps toward a steady state

The meshes are the seeded synthetic ones of ``ucns3d_b200.cases``.  A mesh and
its tables are made once per process and kept, as a program keeps its mesh;
the engine (its uploads and buffers) is made anew by every ``prepare``, and
the state, directions and cotangents come from the seed.

``exact`` evaluates the same outputs in FP64 torch operations from the mesh's
arrays (geometry, stencils, pseudo-inverses, smoothness matrices), which are
inputs of the engine too; gradients come from torch's automatic
differentiation.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch
import torch.utils.checkpoint

from ucns3d_b200 import _native as N
from ucns3d_b200.config import EULER, NAVIER_STOKES, make_config
from ucns3d_b200.engine import Engine
from ucns3d_b200.mesh import IC_TGV, IC_UNIFORM, IC_VORTEX, SCHEME_MUSCL, SCHEME_WENO, Mesh

GAMMA = 1.4
MACH_TGV = 0.1


def _case(name, work, mesh, n, order, steps=1, viscous=False, mixed=False, characteristic=False):
    c = {"work": work, "mesh": mesh, "n": n, "order": order, "steps": steps, "viscous": viscous, "mixed": mixed,
         "characteristic": characteristic}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a unit-test sized box: launches and latency are all there is
        _case("march_muscl_ns_hex8", "march", "hex", 8, 2, steps=20, viscous=True),
        # the 32^3 viscous Taylor-Green run in FP64
        _case("march_muscl_ns_hex32", "march", "hex", 32, 2, steps=20, viscous=True),
        # the bump channel (walls, inflow, outflow), mixed form
        _case("march_muscl_bump240", "march", "bump", 240, 2, steps=20, mixed=True),
        # jittered tetrahedra (every cell has its own matrices), WENO3, FP64
        _case("march_weno3_tet24", "march", "tet", 24, 3, steps=5),
        # the highest order on cells that all have their own matrices
        _case("march_weno5_tet14", "march", "tet", 14, 5, steps=2, mixed=True),
        # the isentropic vortex on 64^3 hexahedra, WENO5, mixed form
        _case("march_weno5_hex64", "march", "hex", 64, 5, steps=2, mixed=True),
        # the same scheme in characteristic variables, FP64, on a box whose
        # size fills no power of two
        _case("residual_weno5_char_hex30", "residual", "hex", 30, 5, characteristic=True),
        # hexahedra, pyramids, tetrahedra and prisms, viscous CWENO4, mixed form
        _case("march_cweno4_ns_mixed48", "march", "mixed", 48, 4, steps=2, viscous=True, mixed=True),
        # the adjoint workload's channel, viscous: one VJP and one JVP
        _case("gradient_muscl_ns_bump240", "gradient", "bump", 240, 2, viscous=True),
        # WENO5 VJP and JVP
        _case("gradient_weno5_hex24", "gradient", "hex", 24, 5),
        # dJ/dU0 and dJ/dp of the wall force through checkpointed RK3 steps
        _case("adjoint_muscl_bump120", "adjoint", "bump", 120, 2, steps=10),
        # implicit steps on the channel
        _case("implicit_muscl_bump120", "implicit", "bump", 120, 2, steps=5),
    ]


def _size(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["muscl_hex", "muscl_bump", "weno3_tet", "weno5_tet", "weno5_hex", "cweno4_mixed", "weno_bump",
                       "characteristic", "gradient_muscl", "gradient_weno", "adjoint", "implicit"])
    mixed, viscous = rng.random() < 0.5, rng.random() < 0.5
    if kind == "muscl_hex":
        return _case(None, "march", "hex", _size(rng, 6, 64), 2, rng.randint(3, 20), viscous, mixed)
    if kind == "muscl_bump":
        return _case(None, "march", "bump", _size(rng, 18, 240), 2, rng.randint(3, 20), viscous, mixed)
    if kind == "weno3_tet":
        return _case(None, rng.choice(["march", "residual"]), "tet", _size(rng, 5, 24), 3, rng.randint(1, 5), viscous,
                     mixed)
    if kind == "weno5_tet":
        return _case(None, "march", "tet", _size(rng, 6, 13), 5, rng.randint(1, 2), False, mixed)
    if kind == "weno5_hex":
        return _case(None, rng.choice(["march", "residual"]), "hex", _size(rng, 12, 56), 5, rng.randint(1, 2),
                     rng.random() < 0.25, mixed)
    if kind == "cweno4_mixed":
        return _case(None, "march", "mixed", 2 * _size(rng, 4, 22), 4, rng.randint(1, 2), viscous, mixed)
    if kind == "weno_bump":
        return _case(None, "march", "bump", _size(rng, 16, 32), rng.choice([3, 4]), rng.randint(1, 4), viscous, mixed)
    if kind == "characteristic":
        mesh, lo, hi, order = rng.choice([("hex", 12, 32, 5), ("tet", 5, 16, 3), ("mixed", 8, 20, 4)])
        n = _size(rng, lo, hi)
        return _case(None, "residual", mesh, n + n % 2 if mesh == "mixed" else n, order, 1, False, mixed, True)
    if kind == "gradient_muscl":
        return _case(None, "gradient", "bump", _size(rng, 18, 240), 2, 1, viscous)
    if kind == "gradient_weno":
        mesh, lo, hi, order = rng.choice([("hex", 12, 22, 5), ("tet", 5, 14, 3), ("mixed", 8, 20, 4)])
        n = _size(rng, lo, hi)
        return _case(None, "gradient", mesh, n + n % 2 if mesh == "mixed" else n, order, 1, viscous)
    if kind == "adjoint":
        return _case(None, "adjoint", "bump", _size(rng, 18, 120), 2, rng.randint(4, 10))
    return _case(None, "implicit", "bump", _size(rng, 18, 160), 2, rng.randint(1, 5), viscous)


# ---------------------------------------------------------------- inputs
ADJOINT_EVERY = 5  # checkpoint stride of the adjoint runs
CFL_EXPLICIT, CFL_IMPLICIT = 0.5, 20.0


@functools.lru_cache(maxsize=2)
def _mesh(mesh, n, order):
    """The prepared mesh, its cell centres and its base state."""
    if mesh == "hex":
        m = Mesh.box_hex(n, n, n, L=(10.0,) * 3 if order == 5 else (2 * np.pi,) * 3)
    elif mesh == "tet":
        m = Mesh.box_tet(n, n, n, jitter=0.15, seed=1234)
    elif mesh == "mixed":
        m = Mesh.mixed_box(n, seed=1234)
    elif order == 2:
        m = Mesh.bump_channel(n, max(6, n // 3), 4, seed=1234)
    else:  # the wide stencils need a thicker channel
        m = Mesh.bump_channel(n, max(8, n // 2), max(8, n // 2), seed=1234)
    scheme = SCHEME_MUSCL if order == 2 else SCHEME_WENO
    m.prepare(scheme, order - 1, ees=5 if order == 4 else 0)
    if mesh == "bump":
        u = 0.675 * math.sqrt(GAMMA)
        base = m.initial_condition(IC_UNIFORM, [GAMMA, 1.0, u, 0.0, 0.0, 1.0])
    elif mesh == "hex" and order == 5:
        u = 0.5 * math.sqrt(GAMMA) / math.sqrt(2.0)
        base = m.initial_condition(IC_VORTEX, [GAMMA, 5.0, u, u, 0.0, 5.0, 5.0, 5.0, 0.0, 10.0, 10.0, 10.0])
    else:
        base = m.initial_condition(IC_TGV, [GAMMA, 1.0 / (GAMMA * MACH_TGV ** 2), 1.0])
    return m, m.centres(), base


def _key(case):
    return case["mesh"], case["n"], case["order"]


def _config(case, m):
    bump = case["mesh"] == "bump"
    vortex = case["mesh"] == "hex" and case["order"] == 5
    return make_config(m, governing=NAVIER_STOKES if case["viscous"] else EULER,
                       precision=N.UCG_MIXED if case["mixed"] else N.UCG_FP64, prandtl=0.71,
                       reynolds=200.0 if bump else 1600.0,
                       pres=1.0 if bump or vortex else 1.0 / (GAMMA * MACH_TGV ** 2),
                       bc_state=(1.0, 0.675 * math.sqrt(GAMMA), 0.0, 0.0, 1.0),
                       wenwrt=2 if case["characteristic"] else 1)


def _inputs(case, seed):
    """The base state with a seeded smooth disturbance of about 1 % (so that
    limiters and weights see data without symmetries), the direction and the
    cotangent of the gradient cases, and the fixed step of the adjoint run."""
    m, x, base = _mesh(*_key(case))
    rng = np.random.default_rng(seed)
    span = x.max(0) - x.min(0)
    wave = np.zeros((len(x), 5))
    for _ in range(3):
        k = 2 * np.pi * rng.integers(1, 4, 3) / np.maximum(span, 1e-30)
        wave += rng.uniform(0.2, 0.4, 5) * np.sin((x @ k)[:, None] + rng.uniform(0, 2 * np.pi, 5))
    scale = np.abs(base).max(0)
    if case["mesh"] in ("tet", "mixed") or case["order"] == 2 and case["mesh"] == "hex":
        scale[[0, 4]] *= 0.02  # Mach 0.1: a weaker disturbance of density and energy
    U = base + 0.01 * wave * np.maximum(scale, 0.1 * scale.max() if case["mesh"] == "bump" else 0.05)
    out = {"U": U}
    if case["work"] == "gradient":
        out["du"] = rng.standard_normal(U.shape) * 1e-2 * np.maximum(np.abs(U).max(0), 0.1)
        out["dp"] = rng.standard_normal(5) * 1e-2
        out["lam"] = rng.standard_normal(U.shape)
    if case["work"] == "adjoint":
        g = m.geometry_struct()
        me = np.ctypeslib.as_array(g.minedge, shape=(m.ncells,))
        r, u = U[:, 0], np.abs(U[:, 1:4] / U[:, :1])
        p = (GAMMA - 1.0) * (U[:, 4] - 0.5 * r * (u * u).sum(1))
        out["dt"] = float(CFL_EXPLICIT / 3.0 * (me / (u.max(1) + np.sqrt(GAMMA * p / r))).min())
    return out


def _host(a):
    """A host array as a driver keeps it: page-locked."""
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t.numpy()


def prepare(case, seed):
    m, _, _ = _mesh(*_key(case))
    ins = _inputs(case, seed)
    state = {k: _host(v) if isinstance(v, np.ndarray) else v for k, v in ins.items()}
    state["case"] = case
    state["engine"] = Engine(m, _config(case, m))
    state["out"] = _host(ins["U"])
    return state


def run(state):
    case, e = state["case"], state["engine"]
    e.set_state(state["U"])
    if case["work"] == "march":
        e.time_marching(case["steps"], CFL_EXPLICIT)
        return {"U": e.get_state(state["out"]), "dt": e.last_dt()}
    if case["work"] == "residual":
        return {"rhs": e.residual()}
    if case["work"] == "gradient":
        mu, pbar = e.residual_vjp(state["lam"])
        return {"mu": mu, "pbar": pbar, "drhs": e.residual_jvp(state["du"], state["dp"])}
    if case["work"] == "adjoint":
        J, gU, gp = e.adjoint_run(case["steps"], state["dt"], ADJOINT_EVERY)
        return {"J": J, "dJdU": gU, "dJdp": gp}
    e.implicit_step(CFL_IMPLICIT, case["steps"])
    return {"U": e.get_state(state["out"])}


# ------------------------------------------------------- work and tolerance
def work(case):
    """Bytes and operations of one pass.  Per residual: the state in and the
    residual out, the geometry and the stencil indices of every cell, and the
    matrices of every distinct matrix set (once per pass if the sets fit in
    the 126 MB of L2, else once per residual, since nothing on the chip keeps
    them)."""
    m, _, _ = _mesh(*_key(case))
    s, n = m.sizes, m.ncells
    t = 4 if case["mixed"] else 8
    A, D, K, D2, K2 = s["admis_max"], s["ideg"], s["imax"], s["ideg2"], s["imax2"]
    F, Q = {"hex": 6, "tet": 4}.get(case["mesh"], 5), max(s["nq_quad"], s["nq_tri"])
    members = K + (A - 1) * (K2 if D2 else K)
    lsq = D * K + (A - 1) * (D2 * K2 if D2 else D * K)
    tri = 0 if case["order"] == 2 else D * (D + 1) // 2 + D2 * (D2 + 1) // 2
    tables = m.ntables * t * (lsq + tri)
    cell = 2 * 40 + 4 * members + t * F * Q * 3 + F * 50 + 24 + (9 * 8 if case["viscous"] else 0)
    forms = 0 if case["order"] == 2 else 2 * 5 * (D * D + (A - 1) * (D2 * D2 if D2 else D * D))
    point = 10 * D + 150 / 2 + (24 * D + 75 if case["viscous"] else 0)
    flop = 10 * lsq + forms + F * Q * point + (8 * D * K if case["viscous"] else 0)
    residuals = {"march": 3 * case["steps"], "residual": 1, "gradient": 5, "adjoint": 10 * case["steps"],
                 "implicit": case["steps"]}[case["work"]]
    extra = n * case["steps"] * (F * 200 + 10 * (F * 200 + 120)) if case["work"] == "implicit" else 0
    return {"bytes": residuals * n * cell + tables * (residuals if tables > 126e6 else 1) + extra,
            "flops": residuals * n * flop}


def tolerance(case):
    """Rounding only, a few times what the engine was seen to be off `exact`:
    the state by 3e-16 in FP64 and, since the mixed form carries FP32
    differences from the cell mean, by 1.3e-9 there; a residual (the small
    sum of large face fluxes) by 7e-14 and 1.1e-6; gradients by 8e-15."""
    if case["work"] == "residual":
        return {"rel": 8e-6, "max": 1e-3} if case["mixed"] else {"rel": 4e-13, "max": 1e-10}
    if case["work"] == "gradient":
        return {"rel": 2e-13, "max": 1e-9}
    if case["work"] == "adjoint":
        return {"rel": 5e-14, "max": 1e-9}
    if case["work"] == "implicit":
        return {"rel": 1e-14, "max": 1e-11}
    return {"rel": 6e-9, "max": 1e-6} if case["mixed"] else {"rel": 3e-15, "max": 1e-12}


# ------------------------------------------------------------------ exact
def _exponents(P):
    return [(n - c - b, b, c) for n in range(1, P + 1) for c in range(n + 1) for b in range(n - c + 1)]


def _monomials(x, P, derivative=None):
    """Monomials of degree 1..P of x [..., 3] (or one of their derivatives)."""
    powers = [[torch.ones_like(x[..., 0])] for _ in range(3)]
    for k in range(3):
        for _ in range(P):
            powers[k].append(powers[k][-1] * x[..., k])
    out = []
    for e in _exponents(P):
        e, f = list(e), 1.0
        if derivative is not None:
            f = float(e[derivative])
            e[derivative] = max(0, e[derivative] - 1)
        out.append(f * powers[0][e[0]] * powers[1][e[1]] * powers[2][e[2]])
    return torch.stack(out, -1)


def _prim(u):
    v = u[..., 1:4] / u[..., :1]
    p = (GAMMA - 1.0) * (u[..., 4] - 0.5 * u[..., 0] * (v * v).sum(-1))
    return u[..., 0], v, p


def _cons(r, v, p):
    e = p / (GAMMA - 1.0) + 0.5 * r * (v * v).sum(-1)
    return torch.cat([r[..., None], r[..., None] * v, e[..., None]], -1)


class _Exact:
    """The engine's scheme from the mesh's arrays, in FP64."""

    def __init__(self, case):
        self.case = case
        self.m, _, _ = _mesh(*_key(case))
        self.cfg = _config(case, self.m)
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        g, r, s = self.m.geometry(), self.m.recon(), self.m.sizes
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)  # noqa: E731
        self.n, self.P, self.Q = self.m.ncells, self.cfg.iorder, max(s["nq_quad"], s["nq_tri"])
        self.D, self.D2, self.K, self.K2, self.A = s["ideg"], s["ideg2"], s["imax"], s["imax2"], s["admis_max"]
        self.weno, self.cweno = self.cfg.scheme == SCHEME_WENO, bool(s["ideg2"])
        self.live = torch.arange(6, device=self.dev)[None] < t(g["nfaces"])[:, None]
        me = torch.arange(self.n, device=self.dev)[:, None].expand(-1, 6)
        neigh = t(g["neigh"]).long()
        self.inner = self.live & (neigh >= 0)
        self.neigh, self.nface = torch.where(self.inner, neigh, me), t(g["neigh_face"]).long().clamp(min=0)
        self.nface = torch.where(self.inner, self.nface, 0)
        self.bc = torch.where(self.live & ~self.inner, t(g["bc"]).long(), 0)
        self.qperm = t(g["qperm"][:, :, :self.Q]).long()
        ang = t(g["face_angle"])
        c1, s1, c2, s2 = (f(ang[..., k]) for k in (0, 1) for f in (torch.cos, torch.sin))
        self.rot = torch.stack([c1, s1, c2, s2], -1)
        self.normal = torch.stack([c1 * s2, s1 * s2, c2], -1)
        self.area = torch.where(self.live, t(g["face_area"]), 0.0)
        self.dih = torch.where(self.live, t(g["dih"]), 1.0)
        quad, tri = (np.pad(np.array(s[k][:s[q]]), (0, self.Q - s[q])) for k, q in
                     (("quad_w", "nq_quad"), ("tri_w", "nq_tri")))
        isquad = t(g["face_type"] == 5)
        self.weight = torch.where(isquad[..., None], t(quad), t(tri)) * self.live[..., None]
        self.points = torch.where((self.weight > 0)[..., None], t(g["qpoints"][:, :, :self.Q]), 0.0)
        self.vol, self.minedge = t(g["volume"]), t(g["minedge"])
        self.jinv, self.bmean = t(g["invccjac"]), t(g["basis_mean"])
        self.admis, self.full = t(g["admis"]).long(), t(g["full"]).bool()
        self.others = (self.admis - 1).clamp(min=1).double()
        self.sten = t(r["stencil"]).long()
        self.tid = t(r["table_id"]).long() if r["table_id"] is not None else torch.arange(self.n, device=self.dev)
        self.ntab = int(r["ntables"])
        self.host = r
        self.t = t
        self.bc_state = torch.tensor(list(self.cfg.bc_state), dtype=torch.float64, device=self.dev)

    # products with per-cell matrices, a block of cells (or one shared set) at a time
    def _per_cell(self, host, form):
        order = torch.argsort(self.tid, stable=True)
        parts = []
        if self.ntab * 8 <= self.n:
            counts = torch.bincount(self.tid, minlength=self.ntab).tolist()
            at = 0
            for k, c in enumerate(counts):
                if c:
                    parts.append(form(self.t(host[k])[None], order[at:at + c]))
                at += c
        else:
            step = max(1, int(1e9 // (host[0].size * 8)))
            for at in range(0, self.n, step):
                cells = order[at:at + step]
                parts.append(form(self.t(host[self.tid[cells].cpu().numpy()]), cells))
        back = torch.empty_like(order)
        back[order] = torch.arange(self.n, device=self.dev)
        return torch.cat(parts)[back]

    def _fit(self, W, ll):
        """Least-squares coefficients [n][D][vars] of stencil ll on cell values W."""
        low = self.cweno and ll > 0
        k, d = (self.K2, self.D2) if low else (self.K, self.D)
        host = self.host["invmat2" if low else "invmat"][:, ll]
        ok = self.admis > ll
        idx = torch.where(ok[:, None], self.sten[:, ll, 1:k + 1], torch.arange(self.n, device=self.dev)[:, None])

        def form(M, cells):
            dW = W[idx[cells]] - W[cells][:, None]
            return torch.einsum("ckd,ckv->cdv", M[:, :k, :d].expand(len(cells), -1, -1), dW) if M.shape[0] > 1 else \
                torch.einsum("kd,ckv->cdv", M[0, :k, :d], dW)

        g = self._per_cell(host, form) * ok[:, None, None]
        return torch.cat([g, g.new_zeros(self.n, self.D - d, g.shape[2])], 1) if d < self.D else g

    def _forms(self, G, ll):
        """G^T S G [n][vars][vars] of one stencil polynomial."""
        low = self.cweno and ll > 0
        d = self.D2 if low else self.D
        host = self.host["indicator2" if low else "indicator"]

        def form(S, cells):
            g = G[cells][:, :d]
            return torch.einsum("cdu,cdw->cuw", g, torch.einsum("cde,cew->cdw", S, g) if S.shape[0] > 1 else
                                torch.einsum("de,cew->cdw", S[0], g))

        return self._per_cell(host, form)

    def _basis(self, f):
        return _monomials(self.points[:, f], self.P) - self.bmean[:, None]

    def _weights(self, IS):
        """Nonlinear weights from the indicators IS [n][A][vars]."""
        on = (torch.arange(self.A, device=self.dev)[None] < self.admis[:, None])[..., None]
        lam = torch.ones(self.n, self.A, 1, dtype=torch.float64, device=self.dev)
        if self.cweno:
            lc1 = 1.0 - 1.0 / self.cfg.lwci
            lam = lam * ((1.0 - lc1) / self.others)[:, None, None]
            lam[:, 0] = lc1
        else:
            lam[:, 0] = self.cfg.lwci
        w = torch.where(on, lam / (self.cfg.weno_eps + IS) ** 4, 0.0)
        return w / w.sum(1, keepdim=True)

    def _ghost(self, f, cl):
        """Ghost states [n][Q][5] of the physical faces in slot f (others unused)."""
        n = self.normal[:, f, None]
        r, v, p = _prim(cl)
        code = self.bc[:, f, None]
        out = cl
        if (code == 4).any() or (code == 3).any():
            mirror = _cons(r, v - 2.0 * (v * n).sum(-1, keepdim=True) * n, p)
            noslip = torch.cat([cl[..., :1], -cl[..., 1:4], cl[..., 4:]], -1)
            wall = noslip if self.case["viscous"] else mirror
            out = torch.where((code == 3)[..., None], mirror, torch.where((code == 4)[..., None], wall, out))
        if (code == 1).any() or (code == 2).any():  # subsonic characteristic states
            r1, v1, p1 = self.bc_state[0], self.bc_state[1:4], self.bc_state[4]
            a = torch.sqrt(GAMMA * p / r)
            sup = (v * v).sum(-1).clamp(min=1e-300).sqrt() / a > 1.0
            p3 = 0.5 * (p1 + p - r * a * (n * (v1 - v)).sum(-1))
            sub_in = _cons(r1 + (p3 - p1) / a ** 2, v1 - n * ((p1 - p3) / (a * r))[..., None], p3)
            pb = p1.expand_as(p)
            sub_out = _cons(r + (pb - p) / a ** 2, v + n * ((p - pb) / (a * r))[..., None], pb)
            free = _cons(r1.expand_as(r), v1.expand_as(v), pb)
            sup = sup[..., None]
            out = torch.where((code == 1)[..., None], torch.where(sup, free, sub_in), out)
            out = torch.where((code == 2)[..., None], torch.where(sup, cl, sub_out), out)
        return out

    def _limited(self, U, G):
        """Venkatakrishnan-limited face differences of the polynomial G, per face."""
        nb = torch.where(self.inner[..., None], U[self.neigh], U[:, None])
        lo, hi = (torch.cat([U[:, None], nb], 1).amin(1) - U)[:, None], (torch.cat([U[:, None], nb], 1).amax(1) - U)[:, None]
        eps2 = (self.cfg.kappa_ven * self.minedge[:, None, None]) ** 3
        dd = [torch.einsum("cqd,cdv->cqv", self._basis(f), G) for f in range(6)]
        phi = []
        for f in range(6):
            d = dd[f]
            used = (self.weight[:, f] > 0)[..., None] & (d != 0)
            x = torch.where(used, d + 1e-13 * d.sign(), 1.0)
            y = torch.where(d > 0, hi, lo)
            num = (y * y + eps2) * x + 2.0 * x * x * y
            phi.append(torch.where(used, num / (x * (y * y + 2.0 * x * x + x * y + eps2)), 1e13))
        slope = torch.stack(phi, 1).amin((1, 2))
        slope = torch.where(slope > 1e12, 1.0, slope)[:, None]
        return [d * slope for d in dd]

    def faces(self, U):
        """Face values minus the cell mean, six tensors [n][Q][5]."""
        G0 = self._fit(U, 0)
        if not self.weno:
            return self._limited(U, G0)
        G = [G0] + [self._fit(U, ll) for ll in range(1, self.A)]
        if self.cweno:
            lc1 = 1.0 - 1.0 / self.cfg.lwci
            lk = ((1.0 - lc1) / self.others)[:, None, None]
            G[0] = (G[0] - lk * sum(G[1:])) / lc1
        forms = [self._forms(g, ll) for ll, g in enumerate(G)]
        if self.case["characteristic"]:
            out = [self._char_face(U, G, forms, f) for f in range(6)]
        else:
            w = self._weights(torch.stack([torch.diagonal(q, dim1=1, dim2=2) for q in forms], 1))
            poly = sum(w[:, ll, None] * G[ll] for ll in range(self.A))
            out = [torch.einsum("cqd,cdv->cqv", self._basis(f), poly) for f in range(6)]
        if not bool(self.full.all()):  # cells without all their stencils: limited central polynomial
            lim = self._limited(U, G0)
            out = [torch.where(self.full[:, None, None], out[f], lim[f]) for f in range(6)]
        return out

    def _char_face(self, U, G, forms, f):
        gm, (c1, s1, c2, s2) = GAMMA - 1.0, self.rot[:, f].unbind(-1)
        z = torch.zeros_like(c1)
        R3 = torch.stack([torch.stack([c1 * s2, s1 * s2, c2], -1), torch.stack([c1 * c2, s1 * c2, -s2], -1),
                          torch.stack([-s1, c1, z], -1)], 1)
        nb = torch.where(self.inner[:, f, None], U[self.neigh[:, f]], self._ghost(f, U[:, None])[:, 0])
        a, b = (torch.cat([u[:, :1], torch.einsum("cij,cj->ci", R3, u[:, 1:4]), u[:, 4:]], 1) for u in (U, nb))
        r = 0.5 * (a[:, 0] + b[:, 0])
        u, v, w = (0.5 * (a[:, 1:4] / a[:, :1] + b[:, 1:4] / b[:, :1])).unbind(-1)
        q2 = u * u + v * v + w * w
        p = gm * (0.5 * (a[:, 4] + b[:, 4]) - 0.5 * r * q2)
        s = torch.sqrt(GAMMA * p / r)
        h = 0.5 * q2 + s * s / gm
        o = torch.ones_like(u)
        ER = torch.stack([torch.stack(x, -1) for x in
                          ([o, o, z, z, o], [u - s, u, z, z, u + s], [v, v, o, z, v], [w, w, z, o, w],
                           [h - u * s, 0.5 * q2, v, w, h + u * s])], 1)
        EL = torch.linalg.inv(ER)
        wt = self._weights(torch.stack([torch.einsum("cku,cuw,ckw->ck", EL, q, EL) for q in forms], 1))
        poly, mean = 0.0, 0.0
        for ll in range(self.A):
            M = torch.einsum("cvk,ck,cku->cvu", ER, wt[:, ll], EL)
            poly = poly + torch.einsum("cdu,cvu->cdv", G[ll], M)
            mean = mean + torch.einsum("cvu,cu->cv", M, U)
        return torch.einsum("cqd,cdv->cqv", self._basis(f), poly) + (mean - U)[:, None]

    def _hllc(self, f, L, R):
        """Flux of the two states through the faces in slot f, along their normals."""
        n = self.normal[:, f, None]
        rl, vl, pl = _prim(L)
        rr, vr, pr = _prim(R)
        ul, ur = (vl * n).sum(-1), (vr * n).sum(-1)
        al, ar = torch.sqrt(GAMMA * pl / rl), torch.sqrt(GAMMA * pr / rr)
        ql, qr = torch.sqrt(rl), torch.sqrt(rr)
        am = torch.sqrt((al * al * ql + ar * ar * qr) / (ql + qr) + 0.5 * ql * qr / (ql + qr) ** 2 * (ur - ul) ** 2)
        um = (ul * ql + ur * qr) / (ql + qr)
        sl = torch.minimum(ul - al, um - am).clamp(max=0.0)
        sr = torch.maximum(ur + ar, um + am).clamp(min=0.0)
        sm = (pr - pl + rl * ul * (sl - ul) - rr * ur * (sr - ur)) / (rl * (sl - ul) - rr * (sr - ur))
        sides = []
        for u, r, v, p, un, s in ((L, rl, vl, pl, ul, sl), (R, rr, vr, pr, ur, sr)):
            F = un[..., None] * u
            F = F + p[..., None] * torch.cat([torch.zeros_like(F[..., :1]), n.expand_as(v), un[..., None]], -1)
            m = r * (s - un) / (s - sm)
            es = u[..., 4] / r + (sm - un) * (sm + p / (r * (s - un)))
            star = torch.cat([m[..., None], m[..., None] * (v + (sm - un)[..., None] * n), (m * es)[..., None]], -1)
            sides.append(F + s[..., None] * (star - u))
        return torch.where((sm >= 0)[..., None], *sides)

    def _sutherland(self, r, p):
        c = self.cfg
        t0, t1 = c.pres / (c.rres * c.r_gas), p / (r * c.r_gas)
        x = t1 / t0
        mu = c.visc * x * torch.sqrt(x) * (t0 + 0.412158681 * t0) / (t1 + 0.412158681 * t0)
        return mu, mu * c.r_gas * GAMMA / (c.prandtl * (GAMMA - 1.0))

    def _viscous(self, f, L, R, grad):
        """Viscous flux from the mean face gradients grad [n][Q][4][3] of T, u, v, w."""
        c, n = self.cfg, self.normal[:, f, None]
        rl, vl, pl = _prim(L)
        rr, vr, pr = _prim(R)
        (ml, ll), (mr, lr) = self._sutherland(rl, pl), self._sutherland(rr, pr)
        mu, lam = 0.5 * (ml + mr), 0.5 * (ll + lr)
        jump = torch.cat([(pr / (rr * c.r_gas) - pl / (rl * c.r_gas))[..., None], vr - vl], -1)
        damp = c.lamx * ((self.bc[:, f] < 1) | (self.bc[:, f] > 4)).double()
        g = grad + (damp * (4.0 / 3.0) / self.dih[:, f].abs())[:, None, None, None] * jump[..., None] * n[:, :, None]
        dv = g[..., 1:, :]
        div = dv.diagonal(dim1=-2, dim2=-1).sum(-1)
        tau = mu[..., None, None] * (dv + dv.transpose(-1, -2)
                                     - (2.0 / 3.0) * div[..., None, None] * torch.eye(3, device=self.dev, dtype=mu.dtype))
        vm = (L[..., 1:4] + R[..., 1:4]) / (L[..., :1] + R[..., :1])
        tn = torch.einsum("cqij,cqj->cqi", tau, n.expand_as(vm))
        heat = lam * (g[..., 0, :] * n).sum(-1)
        return torch.cat([torch.zeros_like(heat)[..., None], tn, (heat + (vm * tn).sum(-1))[..., None]], -1)

    def _gradients(self, U):
        """Face-point gradients of T, u, v, w, six tensors [n][Q][4][3]."""
        r, v, p = _prim(U)
        W = torch.cat([(p / (r * self.cfg.r_gas))[:, None], v], 1)
        C = self._fit(W, 0)
        out = []
        for f in range(6):
            d = torch.stack([_monomials(self.points[:, f], self.P, k) for k in range(3)], -1)
            out.append(torch.einsum("cqdj,cdv,cjk->cqvk", d, C, self.jinv))
        return out

    def _other(self, x, f):
        """The neighbours' values of per-face data x at the points of the faces in slot f."""
        return torch.stack(x, 1)[self.neigh[:, f, None], self.nface[:, f, None], self.qperm[:, f]]

    def residual(self, U):
        d = self.faces(U)
        grads = self._gradients(U) if self.case["viscous"] else None
        total = torch.zeros_like(U)
        for f in range(6):
            L = U[:, None] + d[f]
            inner = self.inner[:, f, None, None]
            R = torch.where(inner, U[self.neigh[:, f]][:, None] + self._other(d, f), self._ghost(f, L))
            flux = self._hllc(f, L, R)
            if grads is not None:
                other = torch.where(inner[..., None], self._other(grads, f), grads[f])
                flux = flux - self._viscous(f, L, R, 0.5 * (grads[f] + other))
            total = total + ((self.weight[:, f] * self.area[:, f, None])[..., None] * flux).sum(1)
        return total

    def local_dt(self, U, cfl):
        r, v, p = _prim(U)
        speed = v.abs().amax(1) + torch.sqrt(GAMMA * p / r)
        if not self.case["viscous"]:
            return cfl / 3.0 * self.minedge / speed
        mu, lam = self._sutherland(r, p)
        return cfl / 3.0 / (speed / self.minedge + 0.5 * (lam + mu) / self.minedge ** 2)

    def rk3(self, U, dt):
        V = self.vol[:, None]
        A = U - dt * self.residual(U) / V
        B = 0.75 * U + 0.25 * A - 0.25 * dt * self.residual(A) / V
        return U / 3.0 + 2.0 / 3.0 * B - 2.0 / 3.0 * dt * self.residual(B) / V

    def force(self, U):
        d = self.faces(U)
        J = 0.0
        for f in range(6):
            p = _prim(U[:, None] + d[f])[2]
            on = (self.bc[:, f] == 4) * self.area[:, f] * self.normal[:, f, 0]
            J = J + (on * ((self.weight[:, f] * p).sum(1) - self.cfg.pres)).sum()
        return J

    def implicit(self, U, cfl, sweeps=10):
        """One step: first-order Jacobian from the cell means, `sweeps` Jacobi sweeps."""
        rhs, dtl = self.residual(U), self.local_dt(U, cfl)
        diag, blocks = self.vol / dtl, []
        for f in range(6):
            n = self.normal[:, f]
            nb = torch.where(self.inner[:, f, None], U[self.neigh[:, f]], self._ghost(f, U[:, None])[:, 0])
            (rl, vl, pl), (rr, vr, pr) = _prim(U), _prim(nb)
            vpp = torch.maximum(torch.sqrt(GAMMA * pl / rl) + (vl * n).sum(1).abs(),
                                torch.sqrt(GAMMA * pr / rr) + (vr * n).sum(1).abs())
            area = self.area[:, f]
            if self.case["viscous"]:
                mu = 0.5 * (self._sutherland(rl, pl)[0] + self._sutherland(rr, pr)[0])
                rh = 0.5 * (U[:, 0] + nb[:, 0])
                vpp = vpp + mu * area / (rh * self.dih[:, f]) * max(4.0 / 3.0, GAMMA / self.cfg.prandtl)
            diag = diag + 0.5 * vpp * area
            blocks.append((0.5 * self._jacobian(nb, n) - 0.5 * vpp[:, None, None]
                           * torch.eye(5, device=self.dev, dtype=U.dtype)) * area[:, None, None])
        du = torch.zeros_like(U)
        for _ in range(sweeps):
            b = -rhs
            for f in range(6):
                n, code = self.normal[:, f], self.bc[:, f, None]
                mirror = torch.cat([du[:, :1], du[:, 1:4] - 2.0 * (du[:, 1:4] * n).sum(1, keepdim=True) * n, du[:, 4:]], 1)
                noslip = torch.cat([du[:, :1], -du[:, 1:4], du[:, 4:]], 1)
                edge = torch.where(code == 1, 0.0, torch.where(code == 3, mirror, torch.where(
                    code == 4, noslip if self.case["viscous"] else mirror, du)))
                d1 = torch.where(self.inner[:, f, None], du[self.neigh[:, f]], edge)
                b = b - torch.einsum("cij,cj->ci", blocks[f], d1)
            du = b / diag[:, None]
        return U + du

    def _jacobian(self, q, n):
        """Flux Jacobian along n; entry (5, 3) carries gamma - 2 as in the
        scheme's definition (COMPUTE_JACOBIANSE, src/flow_operations.f90:4004)."""
        a2, a3 = GAMMA - 1.0, GAMMA - 2.0
        r, v, _ = _prim(q)
        phi, vn = 0.5 * a2 * (v * v).sum(1), (v * n).sum(1)
        a1 = GAMMA * q[:, 4] / r - phi
        J = torch.zeros(len(q), 5, 5, dtype=q.dtype, device=self.dev)
        J[:, 0, 1:4] = n
        J[:, 1:4, 0] = n * phi[:, None] - v * vn[:, None]
        J[:, 1:4, 1:4] = v[:, :, None] * n[:, None] - a2 * n[:, :, None] * v[:, None]
        J[:, 1:4, 1:4] += vn[:, None, None] * torch.eye(3, device=self.dev, dtype=q.dtype)
        J[:, 1:4, 4] = a2 * n
        J[:, 4, 0] = vn * (phi - a1)
        J[:, 4, 1:4] = n * a1[:, None] - torch.tensor([a2, a3, a2], dtype=q.dtype, device=self.dev) * v * vn[:, None]
        J[:, 4, 4] = GAMMA * vn
        return J


def exact(case, seed):
    ins = _inputs(case, seed)
    e = _Exact(case)
    U = e.t(ins["U"])
    if case["work"] == "gradient":
        bc = e.bc_state.clone().requires_grad_(True)
        e.bc_state, U = bc, U.requires_grad_(True)
        seed_lam = e.t(ins["lam"]).requires_grad_(True)
        R = e.residual(U)
        mu, pbar = torch.autograd.grad(R, (U, bc), seed_lam, create_graph=True, allow_unused=True)
        # the tangent by the transpose of the (linear) cotangent map
        dot = (mu * e.t(ins["du"])).sum() + ((pbar * e.t(ins["dp"])).sum() if pbar is not None else 0.0)
        (drhs,) = torch.autograd.grad(dot, seed_lam)
        pbar = torch.zeros(5, dtype=torch.float64) if pbar is None else pbar
        return {"mu": mu.detach().cpu(), "pbar": pbar.detach().cpu(), "drhs": drhs.cpu()}
    if case["work"] == "adjoint":
        e.bc_state.requires_grad_(True)
        U0 = U.requires_grad_(True)
        U = U0
        for _ in range(case["steps"]):
            U = torch.utils.checkpoint.checkpoint(e.rk3, U, ins["dt"], use_reentrant=False)
        J = e.force(U)
        gU, gp = torch.autograd.grad(J, (U0, e.bc_state))
        return {"J": float(J), "dJdU": gU.cpu(), "dJdp": gp.cpu()}
    with torch.no_grad():
        if case["work"] == "residual":
            return {"rhs": e.residual(U).cpu()}
        dt = None
        for _ in range(case["steps"]):
            if case["work"] == "implicit":
                U = e.implicit(U, CFL_IMPLICIT)
            else:
                dt = float(e.local_dt(U, CFL_EXPLICIT).min())
                U = e.rk3(U, dt)
        return {"U": U.cpu()} if dt is None else {"U": U.cpu(), "dt": dt}
