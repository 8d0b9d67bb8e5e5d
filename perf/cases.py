"""Performance cases of up3d_b200: what a full-potential solve has the library do.

Every case is one call (or one step of a solver's loop) through the public
entry points, on the synthetic bump channel of the repository's own
configurations: Kuhn-split boxes from 10 x 4 x 3 (720 tets, the fixtures'
mesh) over 40 x 10 x 10, 100 x 30 x 25 and 200 x 60 x 50 to 320 x 96 x 80
(14.7 M tets).  Meshes are fixed by the case; the potential, the Mach number
or the right-hand side come from the seed, as in a solve, which evaluates
many states on one mesh.  ``exact`` restates each result in plain 64-bit
torch.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from up3d_b200.mesh.kuhn import bump_channel, choking_mach

GAMMA, M_CAP, M_CRIT, UPWIND_C, FLOOR = 1.4, 3.0, 0.95, 1.5, 0.05
DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest call: one residual + Jacobian of the fixtures' mesh; launches and host work
        dict(name="eval_10x4x3", kind="eval", nx=10, ny=4, nz=3, amplitude=0.05, mach=0.85,
             state="seeded", jacobian=True, frozen=False, merged=False),
        # the largest mesh: residual + Jacobian of a seeded subsonic state
        dict(name="eval_320x96x80", kind="eval", nx=320, ny=96, nz=80, amplitude=0.05, mach=0.75,
             state="seeded", jacobian=True, frozen=False, merged=False),
        # a line-search trial of the frozen finish: residual only, ragged mid-size mesh
        dict(name="residual_frozen_101x31x23", kind="eval", nx=101, ny=31, nz=23, amplitude=0.05, mach=0.8,
             state="pocket", jacobian=False, frozen=True, merged=False),
        # a transonic Newton assembly: supersonic pocket over the bump, Term 3, the merged matrix
        dict(name="pocket_200x60x50", kind="eval", nx=200, ny=60, nz=50, amplitude=0.08, mach=0.8,
             state="pocket", jacobian=True, frozen=False, merged=True),
        # the drop-in operators one by one, as a driver written for the reference calls them
        dict(name="operators_40x10x10", kind="operators", nx=40, ny=10, nz=10, amplitude=0.05, mach=0.8,
             state="mixed"),
        # one outer iteration of the density Picard: matrix, AMG with the new values, CG
        dict(name="picard_200x60x50", kind="picard", nx=200, ny=60, nz=50, amplitude=0.08, mach=0.65,
             state="seeded"),
        # one Newton step's linear solve in FP64: Jacobian, AMG with the new values, GMRES
        dict(name="gmres_100x30x25", kind="gmres", nx=100, ny=30, nz=25, amplitude=0.05, mach=0.75,
             state="seeded", mixed=False),
        # the same in mixed precision at the full channel's size
        dict(name="gmres_mixed_200x60x50", kind="gmres", nx=200, ny=60, nz=50, amplitude=0.08, mach=0.65,
             state="seeded", mixed=True),
        # a whole small solve: Picard seed and Newton from the freestream
        dict(name="newton_40x10x10", kind="newton", nx=40, ny=10, nz=10, amplitude=0.05, mach=0.5),
        # forward and backward of the residual (shape and Mach gradients)
        dict(name="adjoint_100x30x25", kind="adjoint", nx=100, ny=30, nz=25, amplitude=0.05, mach=0.8,
             state="pocket"),
        # many cases of uneven size in one evaluation
        dict(name="batched_12", kind="batched", cases=12, nx=100, ny=30, nz=25, shrink=5.0, layout=0),
        # the weighted upwind density of a Picard sweep
        dict(name="weighted_200x60x50", kind="weighted", nx=200, ny=60, nz=50, amplitude=0.08, mach=0.8,
             state="pocket", mode="kernel"),
    ]


def _shape(rng, lo, hi):
    """nx log-uniform in [lo, hi], the channel's proportions give or take a fifth."""
    nx = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    ny = max(2, int(round(nx * 0.30 * rng.uniform(0.8, 1.2))))
    nz = max(2, int(round(nx * 0.25 * rng.uniform(0.8, 1.2))))
    return dict(nx=nx, ny=ny, nz=nz, amplitude=round(rng.uniform(0.02, 0.08), 3))


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval", "operators", "picard", "gmres", "newton", "adjoint", "batched",
                       "weighted"])
    if kind == "eval":
        c = _shape(rng, 10, 260)
        jac = rng.random() < 0.7
        return dict(kind=kind, **c, mach=round(rng.uniform(0.5, 0.85), 3),
                    state=rng.choice(["seeded", "pocket", "mixed"]), jacobian=jac, frozen=rng.random() < 0.4,
                    merged=jac and rng.random() < 0.5)
    if kind == "operators":
        return dict(kind=kind, **_shape(rng, 10, 120), mach=round(rng.uniform(0.5, 0.85), 3),
                    state=rng.choice(["pocket", "mixed"]))
    if kind == "newton":
        c = _shape(rng, 20, 48)
        return dict(kind=kind, **c, mach=round(rng.uniform(0.3, 0.5), 3))
    if kind == "batched":
        c = _shape(rng, 30, 100)
        return dict(kind=kind, cases=rng.randint(3, 16), nx=c["nx"], ny=c["ny"], nz=c["nz"],
                    shrink=round(rng.uniform(1.5, 5.0), 2), layout=rng.randrange(1000))
    if kind == "weighted":
        return dict(kind=kind, **_shape(rng, 20, 190), mach=round(rng.uniform(0.7, 0.85), 3), state="pocket",
                    mode=rng.choice(["kernel", "kernel", "blend"]))
    if kind == "adjoint":
        return dict(kind=kind, **_shape(rng, 20, 180), mach=round(rng.uniform(0.5, 0.85), 3),
                    state=rng.choice(["seeded", "pocket"]))
    # the linear solves: subsonic states, where every size converges
    c = _shape(rng, 20, 170)
    c = dict(kind=kind, **c, mach=round(rng.uniform(0.4, 0.65), 3), state="seeded")
    if kind == "gmres":
        c["mixed"] = rng.random() < 0.5
    return c


# --------------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=3)
def _mesh(nx, ny, nz, amplitude, seed=0):
    return bump_channel(nx, ny, nz, amplitude=amplitude, seed=seed)


def _mesh_of(c):
    return _mesh(c["nx"], c["ny"], c["nz"], c["amplitude"])


def _potential(mesh, state, seed):
    """A nodal potential of the given family (unit freestream along x, channel length 4)."""
    rng = np.random.default_rng(seed)
    lx, ly, lz = mesh.lengths
    X = torch.from_numpy(mesh.nodes).to(DEV)
    x, y, z = X[:, 0], X[:, 1], X[:, 2]
    f = torch.zeros_like(x)
    for _ in range(4):      # low modes that vanish on the inflow and outflow planes
        kx, ky, kz = (int(v) for v in rng.integers(1, 4, size=3))
        py, pz = rng.uniform(0.0, 2.0 * np.pi, size=2)
        f += (rng.standard_normal() * torch.sin(np.pi * kx * x / lx) * torch.cos(np.pi * ky * y / ly + py)
              * torch.cos(np.pi * kz * z / lz + pz))
    phi = x + 0.01 * f / f.abs().max()
    if state == "pocket":   # an accelerated region over the bump, supersonic above M about 0.75
        a, w, h = rng.uniform(0.28, 0.34), 0.55, 0.5
        phi = phi + a * w * 0.5 * math.sqrt(math.pi) * torch.erf((x - 2.0) / w) * torch.exp(-(z / h) ** 2)
    elif state == "mixed":  # sub- and supersonic stretches along the channel, nodal noise
        s = x / lx
        noise = torch.from_numpy(rng.standard_normal(len(mesh.nodes))).to(DEV)
        phi = lx * (1.25 * s + 0.12 * torch.sin(2.0 * np.pi * s)) + 0.04 * lx / mesh.shape[0] * noise
    return phi.contiguous()


def _nearby(mesh, phi, seed):
    """A later iterate near phi (the selection frozen at phi is used there)."""
    rng = np.random.default_rng(seed + 77777)
    x, z = (torch.from_numpy(np.ascontiguousarray(mesh.nodes[:, k])).to(DEV) for k in (0, 2))
    a, k = rng.uniform(0.5, 1.5) * 1e-4, int(rng.integers(1, 4))
    return phi + a * torch.sin(np.pi * k * x / mesh.lengths[0]) * torch.cos(np.pi * z)


def _batch_of(c):
    """(meshes, Mach caps) of a batched case: sizes log-uniform between the largest box and 1/shrink of it."""
    rng = np.random.default_rng(c["layout"])
    meshes, caps = [], []
    for k in range(c["cases"]):
        f = 1.0 if k == 0 else math.exp(-rng.uniform(0.0, math.log(c["shrink"])))
        sh = [max(2, int(round(c[d] * f))) for d in ("nx", "ny", "nz")]
        amp = float(rng.uniform(0.02, 0.08))
        meshes.append(bump_channel(*sh, amplitude=amp, seed=k))
        caps.append(choking_mach(amp) - 0.02)
    return meshes, caps


def _batch_state(c, meshes, caps, seed):
    rng = np.random.default_rng(seed)
    machs = [float(min(rng.uniform(0.5, 0.75), cap)) for cap in caps]
    return machs, torch.cat([_potential(m, "pocket" if k % 2 else "seeded", seed + 31 * k)
                             for k, m in enumerate(meshes)])


def _newton_mach(c, seed):
    return c["mach"] + 0.1 * np.random.default_rng(seed).random()


def prepare(case, seed):
    from up3d_b200.adjoint import AdjointContext
    from up3d_b200.kernels.jacobian import PicardOperator
    from up3d_b200.kernels.upwind import UpwindOperator
    from up3d_b200.solve.batched import BatchedChannels
    from up3d_b200.solve.fused import FlowParams
    from up3d_b200.solve.newton import ChannelWorkspace
    c, kind = case, case["kind"]
    s = {"case": c}
    if kind == "batched":
        meshes, caps = _batch_of(c)
        s["machs"], s["phi"] = _batch_state(c, meshes, caps, seed)
        s["batch"] = BatchedChannels(meshes)
        return s
    mesh = _mesh_of(c)
    if kind in ("operators", "weighted"):
        nodes, elements = torch.from_numpy(mesh.nodes), torch.from_numpy(mesh.elements)
        s["phi"] = _potential(mesh, c["state"], seed)
        if kind == "operators":
            s["op"], s["upw"] = PicardOperator(nodes, elements), UpwindOperator(nodes, elements)
            return s
        s["upw"] = UpwindOperator(nodes, elements, weighted=True, mode=c["mode"])
        g = _Plain(mesh)
        grad, q2 = g.velocities(s.pop("phi"))
        s["grad"], s["q2"] = grad.contiguous(), g.limited(q2, c["mach"]).contiguous()
        s["rho"] = g.density(s["q2"], c["mach"]).contiguous()
        return s
    s["ws"] = ws = ChannelWorkspace(mesh.nodes, mesh.elements, mesh.dirichlet_nodes)
    if kind == "newton":
        s["flow"] = FlowParams(m_inf=_newton_mach(c, seed))
        return s
    s["flow"] = FlowParams(m_inf=c["mach"])
    phi = _potential(mesh, c["state"], seed)
    if kind == "eval" and c["frozen"]:
        s["frozen"] = _Plain(mesh).select(phi, c["mach"])
        phi = _nearby(mesh, phi, seed)
    s["phi"] = phi
    if kind == "picard":
        g = _Plain(mesh)
        s["rho"] = g.density(g.velocities(phi)[1], c["mach"]).contiguous()
        s["amg"] = None
    elif kind == "gmres":
        s["amg"] = None
    elif kind == "adjoint":
        s["ctx"] = AdjointContext(ws, phi, s["flow"])
        s["ctx"].JT
        s["X"] = torch.from_numpy(mesh.nodes).to(DEV)
        s["M"] = torch.tensor(c["mach"], dtype=F64, device=DEV)
        s["g"] = _cotangent(mesh, seed)
    return s


def _cotangent(mesh, seed):
    return torch.from_numpy(np.random.default_rng(seed + 5).standard_normal(len(mesh.nodes))).to(DEV)


# ------------------------------------------------------------------- one pass

def run(s):
    c = s["case"]
    return _RUN[c["kind"]](s, c)


def _run_eval(s, c):
    ev = s["ws"].ev
    R = ev.evaluate(s["phi"], s["flow"], jacobian=c["jacobian"], frozen=s.get("frozen"))
    out = {"R": R, "rho_tilde": ev.rho_tilde, "upstream": ev.upstream}
    if c["jacobian"]:
        out["data"] = ev.data
    if c["merged"]:
        out["indptr"], out["Jv"] = _merged(ev.jacobian(), s["phi"])
    return out


def _merged(J, v):
    """Row pointer of the merged Jacobian and its first product in the linear solve (how many entries it
    holds depends on the state)."""
    return J.indptr, J.matvec(v)


def _run_operators(s, c):
    from up3d_b200.physics.isentropic import density_field, limit_q2_field
    op, upw, phi, m = s["op"], s["upw"], s["phi"], c["mach"]
    grad, q2 = op.velocities(phi)
    q2l = limit_q2_field(q2, m, M_CAP)
    rho = density_field(q2l, m)
    rt = upw.rho_tilde(grad, q2l, rho, m, UPWIND_C, M_CRIT)
    se, su, up = upw.rho_tilde_sensitivities(grad, q2l, rho, m, UPWIND_C, M_CRIT)
    lim = q2l == q2
    A = op.assemble_matrix(rt)
    R = op.assemble_residual(phi, rt)
    J = op.assemble_newton_jacobian(phi, rt, se, su, up, lim_mask=lim)
    indptr, Jv = _merged(J, phi)
    return {"R": R, "rho_tilde": rt, "s_e": se, "s_u": su, "upstream": up, "A": A.data, "indptr": indptr,
            "Jv": Jv}


def _run_picard(s, c):
    from up3d_b200.solve.linear import amg_for, solve_cg, with_dirichlet
    ws = s["ws"]
    A = ws.op.assemble_matrix(s["rho"])
    rhs = -A.matvec(ws.phi_dir)
    rhs[ws.dn] = 0.0
    Af = with_dirichlet(A, ws.mask)
    s["amg"] = amg_for(Af, s["amg"])
    x, _, info = solve_cg(Af, rhs, M=s["amg"], rtol=1e-12, maxiter=3000)
    return {"A": A.data, "phi": torch.where(ws.free, x, ws.phi_dir)}


def _run_gmres(s, c):
    from up3d_b200.solve.linear import amg_for, solve_gmres, solve_gmres_mixed, with_dirichlet
    ws = s["ws"]
    R, _ = ws.residual(s["phi"], s["flow"], jacobian=True)
    rhs = -ws.r_free(R)
    Jf = with_dirichlet(ws.ev.jacobian(), ws.mask)
    s["amg"] = amg_for(ws.picard_matrix(), s["amg"], fp32="both" if c["mixed"] else False)
    if c["mixed"]:
        dphi = solve_gmres_mixed(Jf, rhs, M=s["amg"], rtol=1e-10, restart=60, maxiter=10, inner_rtol=1e-5)[0]
    else:
        dphi = solve_gmres(Jf, rhs, M=s["amg"], rtol=1e-10, restart=60, maxiter=10, on_fail="return")[0]
    return {"R": R, "data": ws.ev.data, "dphi": dphi.masked_fill(ws.mask.bool(), 0.0)}


def _run_newton(s, c):
    from up3d_b200.solve.newton import solve_newton
    phi = solve_newton(s["ws"], s["flow"])["phi"]
    return {"phi": phi, "rho_tilde": s["ws"].ev.rho_tilde}


def _run_adjoint(s, c):
    from up3d_b200.adjoint import ResidualFunction
    phi, X, M = (s[k].detach().requires_grad_(True) for k in ("phi", "X", "M"))
    R = ResidualFunction.apply(s["ctx"], phi, X, M)
    gphi, gX, gM = torch.autograd.grad(R, (phi, X, M), s["g"])
    return {"R": R, "gphi": gphi, "gX": gX, "gM": gM}


def _run_batched(s, c):
    b = s["batch"]
    R = b.evaluate(s["phi"], s["machs"], jacobian=True)
    ev = b.ws.ev
    return {"R": R, "data": ev.data, "rho_tilde": ev.rho_tilde, "upstream": ev.upstream}


def _run_weighted(s, c):
    rt = s["upw"].rho_tilde(s["grad"], s["q2"], s["rho"], c["mach"], UPWIND_C, M_CRIT)
    return {"rho_tilde": rt, "nu": s["upw"].nu}


_RUN = {"eval": _run_eval, "operators": _run_operators, "picard": _run_picard, "gmres": _run_gmres,
        "newton": _run_newton, "adjoint": _run_adjoint, "batched": _run_batched, "weighted": _run_weighted}


# ----------------------------------------------------------------------- work

def _counts(nx, ny, nz):
    """Nodes, tets and P1 non-zeros of a Kuhn-split box."""
    N = (nx + 1) * (ny + 1) * (nz + 1)
    E = 6 * nx * ny * nz
    edges = (nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
             + nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz + nx * ny * nz)
    return N, E, N + 2 * edges


def work(case):
    """Inputs read once, outputs written once.  Of a solve: the mesh, the state and the solution, and the
    matrix once more; how often an iteration has to read the matrix is the method's."""
    c, kind = case, case["kind"]
    if kind == "batched":
        shapes = [m.shape for m in _batch_of(c)[0]]
        N, E, Z = (sum(v) for v in zip(*(_counts(*sh) for sh in shapes)))
    else:
        N, E, Z = _counts(c["nx"], c["ny"], c["nz"])
    state = 32 * E + 32 * N             # connectivity, face neighbours, coordinates, potential
    matrix = 12 * Z
    if kind in ("eval", "batched"):
        jac = c.get("jacobian", True)
        by = state + 8 * N + 12 * E + (matrix if jac else 0) + (9 * E if c.get("frozen") else 0)
        by += 24 * Z + 16 * N if c.get("merged") else 0
        return {"bytes": by, "flops": E * (700 if jac else 400)}
    if kind == "operators":
        return {"bytes": state + 8 * N + 32 * E + 2 * matrix + 12 * Z, "flops": 900 * E}
    if kind == "picard":
        return {"bytes": 24 * E + 48 * N + 2 * matrix, "flops": 100 * E + 60 * Z}
    if kind == "gmres":
        return {"bytes": state + 24 * N + 3 * matrix, "flops": 800 * E + 200 * Z}
    if kind == "newton":
        return {"bytes": 10 * (state + 3 * matrix), "flops": 8000 * E + 2000 * Z}
    if kind == "adjoint":
        return {"bytes": state + 88 * N + 12 * E + matrix, "flops": 1200 * E}
    nb = 35 if c["mode"] == "kernel" else 4
    return {"bytes": E * (16 + 40 + 16 + 24 + 4 * nb) + 24 * N, "flops": E * nb * 60}


# ---------------------------------------------- the same in plain 64-bit torch

class _Plain:
    """The discrete equations on one mesh, element arrays at a time."""

    def __init__(self, mesh, X=None):
        self.X = torch.from_numpy(mesh.nodes).to(DEV) if X is None else X
        self.c = torch.from_numpy(np.ascontiguousarray(mesh.elements)).to(DEV).long()
        self.E, self.N = len(self.c), len(mesh.nodes)
        x0, x1, x2, x3 = (self.X[self.c[:, k]] for k in range(4))
        v1, v2, v3 = x1 - x0, x2 - x0, x3 - x0
        c23 = torch.linalg.cross(v2, v3)
        det = (v1 * c23).sum(1)
        inv = (1.0 / det)[:, None]
        b1, b2, b3 = c23 * inv, torch.linalg.cross(v3, v1) * inv, torch.linalg.cross(v1, v2) * inv
        self.B = torch.stack([-(b1 + b2 + b3), b1, b2, b3], 1)
        self.V = det.abs() / 6.0

    # adjacency --------------------------------------------------------------
    @functools.cached_property
    def fnbr(self):
        """Element across the face opposite local node k, -1 at the boundary."""
        faces = torch.cat([self.c[:, [j for j in range(4) if j != k]] for k in range(4)]).sort(1).values
        key = faces[:, 0] * self.N + faces[:, 1]
        owner = torch.arange(self.E, device=DEV).repeat(4)
        o1 = torch.argsort(faces[:, 2], stable=True)
        o = o1[torch.argsort(key[o1], stable=True)]
        same = (key[o][1:] == key[o][:-1]) & (faces[o, 2][1:] == faces[o, 2][:-1])
        out = torch.full((4 * self.E,), -1, dtype=torch.long, device=DEV)
        a, b = o[:-1][same], o[1:][same]
        out[a], out[b] = owner[b], owner[a]
        return out.view(4, self.E).T.contiguous()

    @functools.cached_property
    def cen(self):
        x = self.X
        return (((x[self.c[:, 0]] + x[self.c[:, 1]]) + x[self.c[:, 2]]) + x[self.c[:, 3]]) * 0.25

    @functools.cached_property
    def keys(self):
        """Sorted (row, col) keys of the P1 pattern."""
        k = torch.cat([self.c[:, i] * self.N + self.c[:, j] for i in range(4) for j in range(i, 4)])
        k = torch.unique(k)
        return torch.unique(torch.cat([k, (k % self.N) * self.N + k // self.N]))

    # physics ----------------------------------------------------------------
    def velocities(self, phi):
        p = phi[self.c]
        g = ((p[:, 0, None] * self.B[:, 0] + p[:, 1, None] * self.B[:, 1]) + p[:, 2, None] * self.B[:, 2]
             ) + p[:, 3, None] * self.B[:, 3]
        return g, (g * g).sum(1)

    @staticmethod
    def _base(q2, m):
        return 1.0 + 0.2 * m * m * (1.0 - q2)

    def limited(self, q2, m):
        cap = M_CAP ** 2 * (1.0 + 0.2 * m * m) / (m * m * (1.0 + 0.2 * M_CAP ** 2))
        cap = cap if torch.is_tensor(cap) else torch.tensor(cap, dtype=F64, device=DEV)
        return torch.minimum(q2, cap)

    def density(self, q2, m):
        return self._base(q2, m).clamp(min=1e-10) ** 2.5

    def switch(self, q2, m):
        m2 = q2 * m * m / self._base(q2, m)
        return UPWIND_C * (1.0 - M_CRIT ** 2 / m2.clamp(min=M_CRIT ** 2)).clamp(min=0.0)

    @torch.no_grad()
    def walk(self, g):
        cur = torch.arange(self.E, device=DEV)
        pr = (self.X[self.c] * g[:, None, :]).sum(2)
        target = 0.8 * (pr.max(1).values - pr.min(1).values)
        del pr
        reach = torch.zeros_like(target)
        live = reach < target
        for _ in range(4):
            e = torch.nonzero(live).flatten()
            if not len(e):
                break
            here = cur[e]
            nb = self.fnbr[here]
            d = ((self.cen[nb.clamp(min=0)] - self.cen[here][:, None, :]) * g[e][:, None, :]).sum(2)
            d = torch.where(nb >= 0, d, torch.zeros_like(d))
            best, k = d.min(1)
            go = best < 0.0
            cur[e[go]] = nb[go, k[go]]
            reach[e[go]] -= best[go]
            live[e[~go]] = False
            live &= reach < target
        return cur

    @torch.no_grad()
    def select(self, phi, m):
        """The (upstream, branch) selection at phi."""
        g, q2 = self.velocities(phi)
        q2 = self.limited(q2, m)
        rho, nu = self.density(q2, m), self.switch(q2, m)
        up = self.walk(g)
        nuu = nu[up]
        rt = rho - torch.maximum(nu, nuu) * (rho - rho[up])
        br = torch.where(torch.maximum(nu, nuu) == 0.0, 0, torch.where(nu >= nuu, 1, 2))
        own = up == torch.arange(self.E, device=DEV)
        br = torch.where(own, 0, br)
        br = torch.where(torch.where(own, rho, rt) <= FLOOR, 3, br)
        return up, br.to(torch.int8)

    def flux(self, phi, m, frozen=None, up=None):
        """grad, limited q2, rho~, the upstream element and q2 itself."""
        g, q2 = self.velocities(phi)
        q2l = self.limited(q2, m)
        rho = self.density(q2l, m)
        nu = self.switch(q2l, m)
        if frozen is not None:
            up, br = frozen
            br = br.long()
            nu = torch.where(br == 1, nu, torch.where(br == 2, nu[up], torch.zeros_like(nu)))
            rt = torch.where(br == 3, torch.full_like(rho, FLOOR), rho - nu * (rho - rho[up]))
        else:
            up = self.walk(g.detach()) if up is None else up
            nu = torch.maximum(nu, nu[up])
            rt = (rho - nu * (rho - rho[up])).clamp(min=FLOOR)
        return g, q2, q2l, rt, up

    def residual(self, phi, m, **kw):
        g, _, _, rt, up = self.flux(phi, m, **kw)
        r = (rt * self.V)[:, None] * (self.B * g[:, None, :]).sum(2)
        return self.nodal(r), rt, up

    def nodal(self, r):
        return torch.zeros(self.N, dtype=F64, device=DEV).index_add(0, self.c.reshape(-1), r.reshape(-1))

    def sensitivities(self, phi, m, frozen=None):
        """d rho~ / d q2 of the element and of its upstream element, by autograd; zero where the limiter acts."""
        with torch.no_grad():
            _, q2, _, _, up = self.flux(phi, m, frozen=frozen)
        own = up == torch.arange(self.E, device=DEV)
        qe, qu = q2.clone().requires_grad_(True), q2[up].requires_grad_(True)
        le, lu = self.limited(qe, m), self.limited(qu, m)
        re, ru = self.density(le, m), self.density(lu, m)
        ne, nu = self.switch(le, m), self.switch(lu, m)
        if frozen is not None:
            br = frozen[1].long()
            n = torch.where(br == 1, ne, torch.where(br == 2, nu, torch.zeros_like(ne)))
            rt = torch.where(br == 3, torch.zeros_like(re), re - n * (re - ru))
        else:
            rt = re - torch.where(ne >= nu, ne, nu) * (re - ru)
            rt = torch.where(own, re, rt)
            rt = torch.where(rt <= FLOOR, torch.zeros_like(rt), rt)
        a, b = torch.autograd.grad(rt.sum(), (qe, qu))
        return a, b, up

    def slots(self, row, col):
        return torch.searchsorted(self.keys, row * self.N + col)

    def stiffness(self, w):
        """P1 data of sum_e w_e (B_i . B_j)."""
        data = torch.zeros(len(self.keys), dtype=F64, device=DEV)
        for i in range(4):
            for j in range(4):
                data.index_add_(0, self.slots(self.c[:, i], self.c[:, j]), w * (self.B[:, i] * self.B[:, j]).sum(1))
        return data

    def jacobian(self, phi, m, frozen=None):
        """(P1 data with Term 3 folded in, the entries outside the pattern as (keys, values))."""
        with torch.no_grad():
            g, _, _, rt, _ = self.flux(phi, m, frozen=frozen)
        se, su, up = self.sensitivities(phi, m, frozen)
        gB = (self.B * g[:, None, :]).sum(2)
        data = self.stiffness(rt * self.V)
        w2 = 2.0 * se * self.V
        for i in range(4):
            for j in range(4):
                data.index_add_(0, self.slots(self.c[:, i], self.c[:, j]), w2 * gB[:, i] * gB[:, j])
        act = torch.nonzero(su != 0.0).flatten()
        a, u = (2.0 * su * self.V)[act, None] * gB[act], up[act]
        b = (self.B[u] * g[u][:, None, :]).sum(2)
        k = torch.stack([self.c[act, i] * self.N + self.c[u, j] for i in range(4) for j in range(4)], 1).reshape(-1)
        v = torch.stack([a[:, i] * b[:, j] for i in range(4) for j in range(4)], 1).reshape(-1)
        z = torch.searchsorted(self.keys, k).clamp(max=len(self.keys) - 1)
        inside = self.keys[z] == k
        data.index_add_(0, z[inside], v[inside])
        xk, inv = torch.unique(k[~inside], return_inverse=True)
        xv = torch.zeros(len(xk), dtype=F64, device=DEV).index_add_(0, inv, v[~inside])
        return data, xk, xv

    def csr(self, data, xk=None, xv=None, keep=None):
        """Sparse matrix; keep: a mask of the unknowns, the others become identity rows."""
        k, v = (self.keys, data) if xk is None else (torch.cat([self.keys, xk]), torch.cat([data, xv]))
        r, c = k // self.N, k % self.N
        if keep is not None:
            ok = keep[r] & keep[c]
            d = torch.nonzero(~keep).flatten()
            r, c, v = torch.cat([r[ok], d]), torch.cat([c[ok], d]), torch.cat([v[ok], torch.ones(len(d), dtype=F64, device=DEV)])
        return torch.sparse_coo_tensor(torch.stack([r, c]), v, (self.N, self.N)).coalesce().to_sparse_csr()


def _diag(A):
    ip, ix = A.crow_indices(), A.col_indices()
    r = torch.repeat_interleave(torch.arange(A.shape[0], device=DEV), ip[1:] - ip[:-1])
    d = torch.ones(A.shape[0], dtype=F64, device=DEV)
    on = r == ix
    d[r[on]] = A.values()[on]
    return d


def _cg(A, b, tol=1e-15, most=6000):
    dinv = 1.0 / _diag(A)
    x = torch.zeros_like(b)
    r = b.clone()
    z = dinv * r
    p, rz, end = z.clone(), r @ z, tol * float(b.norm())
    for k in range(most):
        q = A @ p
        a = rz / (p @ q)
        x, r = x + a * p, r - a * q
        if k % 20 == 0 and float(r.norm()) < end:
            break
        z = dinv * r
        new = r @ z
        p, rz = z + (new / rz) * p, new
    return x


def _bicgstab(A, b, tol=1e-14, rounds=4, most=3000):
    """Jacobi-preconditioned BiCGStab with restarts from the true residual."""
    dinv = 1.0 / _diag(A)
    x = torch.zeros_like(b)
    end = tol * float(b.norm())
    for _ in range(rounds):
        r = b - A @ x
        if float(r.norm()) < end:
            break
        r0, p = r.clone(), r.clone()
        rho = r0 @ r
        for k in range(most):
            y = dinv * p
            v = A @ y
            al = rho / (r0 @ v)
            s = r - al * v
            z = dinv * s
            t = A @ z
            om = (t @ s) / (t @ t)
            x = x + al * y + om * z
            r = s - om * t
            if k % 20 == 0 and (not math.isfinite(float(om)) or float(r.norm()) < end):
                break
            new = r0 @ r
            p = r + (new / rho) * (al / om) * (p - om * v)
            rho = new
    return x


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "batched":
        return _exact_batched(c, seed)
    mesh = _mesh_of(c)
    g, m = _Plain(mesh), c["mach"]
    if kind == "newton":
        return _exact_newton(c, mesh, g, seed)
    phi = _potential(mesh, c["state"], seed)
    if kind == "eval":
        frozen = g.select(phi, m) if c["frozen"] else None
        if frozen is not None:
            phi = _nearby(mesh, phi, seed)
        R, rt, up = g.residual(phi, m, frozen=frozen)
        out = {"R": R, "rho_tilde": rt, "upstream": up.to(torch.int32)}
        if c["jacobian"]:
            J = g.jacobian(phi, m, frozen)
            out["data"] = J[0]
            if c["merged"]:     # the row pointer leaves out entries that cancel exactly
                out["indptr"], out["Jv"] = None, g.csr(*J) @ phi
        return out
    if kind == "operators":
        R, rt, up = g.residual(phi, m)
        se, su, _ = g.sensitivities(phi, m)
        return {"R": R, "rho_tilde": rt, "s_e": se, "s_u": su, "upstream": up, "A": g.stiffness(rt * g.V),
                "indptr": None, "Jv": g.csr(*g.jacobian(phi, m)) @ phi}
    if kind == "weighted":
        return _exact_weighted(c, g, phi)
    if kind == "adjoint":
        return _exact_adjoint(c, mesh, phi, seed)
    keep = torch.ones(g.N, dtype=torch.bool, device=DEV)
    keep[torch.from_numpy(mesh.dirichlet_nodes).to(DEV)] = False
    if kind == "picard":
        data = g.stiffness(g.density(g.velocities(phi)[1], m) * g.V)
        phi_dir = torch.where(keep, torch.zeros_like(phi), g.X[:, 0])
        rhs = torch.where(keep, -(g.csr(data) @ phi_dir), torch.zeros_like(phi))
        x = _cg(g.csr(data, keep=keep), rhs)
        return {"A": data, "phi": torch.where(keep, x, phi_dir)}
    R = g.residual(phi, m)[0]
    data, xk, xv = g.jacobian(phi, m)
    x = _bicgstab(g.csr(data, xk, xv, keep=keep), torch.where(keep, -R, torch.zeros_like(R)))
    return {"R": R, "data": data, "dphi": x}


def _exact_newton(c, mesh, g, seed):
    """Dense Newton to rounding level."""
    if g.N > 12000:
        return None
    m = _newton_mach(c, seed)
    keep = torch.ones(g.N, dtype=torch.bool, device=DEV)
    keep[torch.from_numpy(mesh.dirichlet_nodes).to(DEV)] = False
    phi = g.X[:, 0].clone()
    for _ in range(12):
        R = torch.where(keep, g.residual(phi, m)[0], torch.zeros_like(phi))
        if float(R.abs().max()) < 1e-15:
            break
        step = torch.linalg.solve(g.csr(*g.jacobian(phi, m), keep=keep).to_dense(), -R)
        phi = phi + step
        if float(step.abs().max()) < 1e-13:
            break
    return {"phi": phi, "rho_tilde": g.flux(phi, m)[3]}


def _exact_batched(c, seed):
    meshes, caps = _batch_of(c)
    machs, phi = _batch_state(c, meshes, caps, seed)
    out, n, e = {"R": [], "data": [], "rho_tilde": [], "upstream": []}, 0, 0
    for mesh, m in zip(meshes, machs):
        g = _Plain(mesh)
        p = phi[n:n + g.N]
        R, rt, up = g.residual(p, m)
        for k, v in zip(out, (R, g.jacobian(p, m)[0], rt, (up + e).to(torch.int32))):
            out[k].append(v)
        n, e = n + g.N, e + g.E
    return {k: torch.cat(v) for k, v in out.items()}


def _exact_adjoint(c, mesh, phi, seed):
    phi = phi.detach().requires_grad_(True)
    X = torch.from_numpy(mesh.nodes).to(DEV).requires_grad_(True)
    M = torch.tensor(c["mach"], dtype=F64, device=DEV, requires_grad=True)
    with torch.no_grad():
        p = _Plain(mesh)
        up = p.walk(p.velocities(phi)[0])
        del p
    R = _Plain(mesh, X).residual(phi, M, up=up)[0]
    gphi, gX, gM = torch.autograd.grad(R, (phi, X, M), _cotangent(mesh, seed))
    return {"R": R.detach(), "gphi": gphi, "gX": gX, "gM": gM}


def _exact_weighted(c, g, phi):
    """The streamline-Gaussian sample over three face hops, or the blend over the four faces."""
    m = c["mach"]
    grad, q2 = g.velocities(phi)
    q2 = g.limited(q2, m)
    rho, m2 = g.density(q2, m), q2 * m * m / g._base(q2, m)
    nu_out, rt_out = torch.empty_like(rho), torch.empty_like(rho)
    for a in range(0, g.E, 400_000):
        e = torch.arange(a, min(g.E, a + 400_000), device=DEV)
        v = grad[e] / grad[e].norm(dim=1, keepdim=True)
        pr = (g.X[g.c[e]] * v[:, None, :]).sum(2)
        ext = pr.max(1).values - pr.min(1).values
        nb = g.fnbr[e]
        if c["mode"] == "kernel":
            ring = nb
            for _ in range(2):
                ring = torch.where(ring[:, :, None] >= 0, g.fnbr[ring.clamp(min=0)], -1).reshape(len(e), -1)
                nb = torch.cat([nb, ring], 1)
            nb = nb.sort(1).values
            ok = (nb >= 0) & (nb != e[:, None])
            ok[:, 1:] &= nb[:, 1:] != nb[:, :-1]
        else:
            ok = nb >= 0
        nb = nb.clamp(min=0)
        d = g.cen[nb] - g.cen[e][:, None, :]
        upd = -(d * v[:, None, :]).sum(2)
        ok &= upd > 0.0
        if c["mode"] == "kernel":
            sg = (2.0 * (0.35 * ext) ** 2)[:, None]
            perp = ((d * d).sum(2) - upd * upd).clamp(min=0.0)
            w = torch.exp(-((upd - ext[:, None]) ** 2 / sg + perp / sg))
        else:
            w = (upd / d.norm(dim=2)).clamp(min=0.0) ** 3.0
        w = torch.where(ok, w, torch.zeros_like(w))
        ws = w.sum(1)
        has = ws > 0.0
        safe = torch.where(has, ws, torch.ones_like(ws))
        ru, m2u = (w * rho[nb]).sum(1) / safe, (w * m2[nb]).sum(1) / safe
        nu_e = g.switch(q2[e], m)
        nu_u = UPWIND_C * (1.0 - M_CRIT ** 2 / m2u.clamp(min=M_CRIT ** 2)).clamp(min=0.0)
        nu = torch.where(has, torch.maximum(nu_e, nu_u), nu_e)
        gain = 1.0
        if c["mode"] != "kernel":
            gain = (ext / ((w * upd).sum(1) / safe).clamp(min=1e-30)).clamp(min=1.0, max=4.0)
        rt = (rho[e] - nu * gain * (rho[e] - ru)).clamp(min=FLOOR)
        nu_out[e], rt_out[e] = nu, torch.where(has & (nu > 0.0), rt, rho[e])
    return {"rho_tilde": rt_out, "nu": nu_out}
