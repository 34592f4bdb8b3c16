"""The workloads whose speed is measured: calls a flow solver makes through ``semo_mesh_gb300.Context``.

A case is a dict of plain values:

``call``
    ``outer``     one outer iteration (momentum, then pressure correction)
    ``step``      a volume-fraction sub-iteration, then one outer iteration
    ``pressure``  one pressure correction alone
    ``momentum``  one momentum predictor alone
    ``vof``       one volume-fraction sub-iteration alone
    ``coupled``   one compressible coupled 5x5 pass (tetrahedra)
    ``adjoint``   forward pressure solve and the gradient of an objective
    ``coo_p``     a caller-supplied symmetric system (SEMO's COO triple)
    ``coo_m``     a caller-supplied non-symmetric system, three right-hand sides
``n``
    the box has n^3 hexahedra (6 n^3 tetrahedra for ``coupled``); the COO
    systems live on an n x (n + 3) x (n - 1) lattice
``fluid``
    ``box`` one fluid on the plain lattice, ``vof`` a water drop in air with
    gravity on a jittered mesh, ``drop`` the same with surface tension
``precision``
    of the pressure (or coupled) solver: ``mixed`` or ``fp64``
``rebuild``
    the pressure hierarchy is built in every pass (a pass of a new time step,
    whose densities are new) instead of being kept while the matrix stays the
    same (a further outer iteration inside a time step)

Every pass goes the way a host program does: the fields go in from its own
(pinned) arrays, the call is made, the updated fields come back.  Old
velocities and old volume fractions belong to the time step and are set with
the case.  Everything is seeded; the mesh topology is kept between cases of
one size, the vertex positions and all fields come from the seed.
"""
from __future__ import annotations

import functools
import math
from dataclasses import replace

import numpy as np
import torch

import semo_mesh_gb300 as semo
from semo_mesh_gb300 import cases as cs
from semo_mesh_gb300.meshgen import hex_box, tet_box


def listed():
    return [
        # the headline run: a time step's first outer iteration at the size the bench reports
        dict(name="outer_vof_128", call="outer", n=128, fluid="vof", precision="mixed", rebuild=True),
        # the same in all-FP64, on a box whose side fills no tile
        dict(name="outer_vof_61_fp64", call="outer", n=61, fluid="vof", precision="fp64", rebuild=True),
        # the small plain case: latency and launches count
        dict(name="outer_box_32", call="outer", n=32, fluid="box", precision="mixed", rebuild=True),
        # the smallest call a test or a tuning loop makes
        dict(name="pressure_box_14", call="pressure", n=14, fluid="box", precision="mixed", rebuild=True),
        # a further pressure correction inside a time step: the matrix is the last one's
        dict(name="pressure_vof_96_kept", call="pressure", n=96, fluid="vof", precision="mixed", rebuild=False),
        # the momentum predictor alone (three right-hand sides)
        dict(name="momentum_vof_75", call="momentum", n=75, fluid="vof", precision="mixed", rebuild=True),
        # a whole time step: volume fraction, then momentum and pressure
        dict(name="step_vof_80", call="step", n=80, fluid="vof", precision="mixed", rebuild=True),
        # the same with surface tension, odd size
        dict(name="step_drop_47", call="step", n=47, fluid="drop", precision="mixed", rebuild=True),
        # compressible coupled system on tetrahedra (131,712 cells)
        dict(name="coupled_tet_28", call="coupled", n=28, fluid="gas", precision="fp64", rebuild=True),
        # gradient of an objective through the pressure solve, on the jittered 64^3 mesh
        dict(name="adjoint_vof_64", call="adjoint", n=64, fluid="vof", precision="mixed", rebuild=True),
        # systems assembled by the caller
        dict(name="coo_pressure_48", call="coo_p", n=48, fluid="vof", precision="mixed", rebuild=True),
        dict(name="coo_momentum_40", call="coo_m", n=40, fluid="vof", precision="mixed", rebuild=True),
    ]


# call: smallest and largest n that it is drawn with
RANGES = {"outer": (14, 120), "step": (16, 104), "pressure": (12, 120), "momentum": (12, 120), "vof": (12, 110),
          "coupled": (6, 26), "adjoint": (16, 80), "coo_p": (12, 60), "coo_m": (12, 60)}
BOX_DT = 5e-3   # time step of the plain box: Courant numbers of 0.1 to 0.6


def draw(rng):
    call = rng.choice(list(RANGES))
    lo, hi = RANGES[call]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    fluid = "gas" if call == "coupled" else "vof"
    if call in ("outer", "pressure", "momentum"):
        fluid = rng.choice(("vof", "vof", "box", "drop"))
    elif call in ("step", "vof"):
        fluid = rng.choice(("vof", "drop"))
    elif call == "adjoint":
        fluid = rng.choice(("vof", "box"))
    return dict(call=call, n=n, fluid=fluid, precision=rng.choice(("mixed", "mixed", "fp64")),
                rebuild=rng.random() < 0.75)


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=24)
def _topology(n, tets):
    return tet_box(n) if tets else hex_box(n)


def _jittered(mesh, n, rng, amount=0.2):
    """The mesh with every interior vertex moved by uniform[-amount, amount] of the spacing."""
    pts = mesh.points.reshape(n + 1, n + 1, n + 1, 3).copy()
    pts[1:-1, 1:-1, 1:-1] += rng.uniform(-amount / n, amount / n, size=(n - 1, n - 1, n - 1, 3))
    return replace(mesh, points=pts.reshape(-1, 3))


def _centres(mesh, n):
    p = mesh.points.reshape(n + 1, n + 1, n + 1, 3)
    s = sum(p[i:n + i, j:n + j, k:n + k] for i in (0, 1) for j in (0, 1) for k in (0, 1))
    return (s / 8.0).reshape(-1, 3)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    out = t.numpy()
    out[...] = a
    return out


def _hex_case(case, seed):
    """A ``cases.Case`` of this seed, with its BDF2 history."""
    n, rng = case["n"], np.random.default_rng(seed)
    mesh = _topology(n, False)
    plain = case["fluid"] == "box"
    mesh = replace(mesh) if plain else _jittered(mesh, n, rng)
    nc = mesh.n_cells
    bc_type = np.zeros((len(mesh.patch_names), 3), dtype=np.int32)
    bc_value = np.zeros((len(mesh.patch_names), 5))
    bc_type[mesh.patch_names.index("zmax"), 0] = cs.BC_FIXED_VALUE
    u = rng.uniform(-1.0, 1.0, size=(3, nc))
    c = cs.Case(name=case["fluid"], mesh=mesh, P=rng.uniform(-1.0, 1.0, size=nc), U=u[0], V=u[1], W=u[2],
                VF=np.ones(nc), bc_type=bc_type, bc_value=bc_value, dt=BOX_DT)
    if not plain:
        r = np.linalg.norm(_centres(mesh, n) - 0.5 - rng.uniform(-0.05, 0.05, size=3), axis=1)
        c.VF = 0.5 * (1.0 - np.tanh((r - 0.25) / 0.01))
        c.dt, c.rho, c.mu = 1e-4, (1000.0, 1.2), (1e-3, 1.8e-5)
        c.gravity, c.use_gravity = (0.0, 0.0, -9.81), True
        c.sigma = 0.072 if case["fluid"] == "drop" else 0.0
        c.old_vf = np.clip(c.VF + 0.05 * rng.uniform(-1.0, 1.0, size=nc), 0.0, 1.0)
        c.old2_vf = np.clip(c.VF + 0.05 * rng.uniform(-1.0, 1.0, size=nc), 0.0, 1.0)
    c.old = tuple(x + 0.1 * rng.uniform(-1.0, 1.0, size=nc) for x in (c.U, c.V, c.W))
    c.old2 = tuple(x + 0.1 * rng.uniform(-1.0, 1.0, size=nc) for x in (c.U, c.V, c.W))
    return c


def _gas_case(case, seed):
    """Ideal gas on tetrahedra: a smooth pressure noise, uniform temperature and velocity noise, walls."""
    n, rng = case["n"], np.random.default_rng(seed)
    mesh = _jittered(_topology(n, True), n, rng)
    nc = mesh.n_cells
    noise = rng.standard_normal((n, n, n))
    for ax in (0, 1, 2):
        e = np.pad(noise, [(1, 1) if a == ax else (0, 0) for a in range(3)], mode="edge")
        noise = (np.take(e, range(n), ax) + noise + np.take(e, range(2, n + 2), ax)) / 3.0
    P = 1e5 + 1e3 * np.repeat(noise.reshape(-1), 6)
    u = rng.uniform(-50.0, 50.0, size=(3, nc))
    cur = np.stack([P, u[0], u[1], u[2], 300.0 + rng.uniform(-5.0, 5.0, size=nc)])
    old, old2 = (cur * (1.0 + 1e-3 * rng.uniform(-1.0, 1.0, size=cur.shape)) for _ in range(2))
    bc_type = np.zeros((len(mesh.patch_names), 3), dtype=np.int32)
    bc_type[:, 1] = cs.BC_NO_SLIP
    return cs.CoupledCase(name="gas", mesh=mesh, P=cur[0], U=cur[1], V=cur[2], W=cur[3], T=cur[4], old=old,
                          old2=old2, bc_type=bc_type, bc_value=np.zeros((len(mesh.patch_names), 5)))


def _coo(case, seed):
    """SEMO's COO triple of a lattice system (diagonals first, then two entries a face) and its right-hand sides."""
    n, rng = case["n"], np.random.default_rng(seed)
    shape = (n, n + 3, max(n - 1, 2))
    N = shape[0] * shape[1] * shape[2]
    idx = np.arange(N).reshape(shape)
    o, q, ax = [], [], []
    for a in range(3):
        lo, hi = np.take(idx, range(shape[a] - 1), a).reshape(-1), np.take(idx, range(1, shape[a]), a).reshape(-1)
        o.append(lo); q.append(hi); ax.append(np.full(lo.size, a))
    o, q, ax = np.concatenate(o), np.concatenate(q), np.concatenate(ax)
    order = np.lexsort((q, o))
    o, q, ax = o[order], q[order], ax[order]
    if case["call"] == "coo_p":
        # dt/rho between the two fluids, one face of the lattice at a fixed pressure
        pos = np.stack(np.unravel_index(np.arange(N), shape), 1) / np.array(shape) - 0.5 - rng.uniform(-0.05, 0.05, 3)
        r = np.linalg.norm(pos, axis=1)
        vf = 0.5 * (1.0 - np.tanh((r - 0.25) / 0.02))
        irho = 1.0 / (1000.0 * vf + 1.2 * (1.0 - vf))
        c = 0.5 * (irho[o] + irho[q]) * rng.uniform(0.8, 1.25, o.size)
        diag = np.bincount(o, c, N) + np.bincount(q, c, N)
        top = idx[:, :, -1].reshape(-1)
        diag[top] += 2.0 * irho[top]
        lr = rl = -c
        b = rng.uniform(-1.0, 1.0, size=(1, N))
    else:
        # an implicit time term, upwind convection and diffusion
        flux, visc = rng.uniform(-1.0, 1.0, o.size), 0.1 * rng.uniform(0.5, 1.5, o.size)
        lr, rl = np.minimum(flux, 0.0) - visc, -np.maximum(flux, 0.0) - visc
        diag = np.full(N, 4.0) + rng.uniform(0.0, 1.0, N)
        diag += np.bincount(o, np.maximum(flux, 0.0) + visc, N) + np.bincount(q, -np.minimum(flux, 0.0) + visc, N)
        b = rng.uniform(-1.0, 1.0, size=(3, N))
    i = np.arange(N)
    rows = np.concatenate([i, np.stack([o, q], 1).reshape(-1)]).astype(np.int32)
    cols = np.concatenate([i, np.stack([q, o], 1).reshape(-1)]).astype(np.int32)
    vals = np.concatenate([diag, np.stack([lr, rl], 1).reshape(-1)])
    return rows, cols, vals, b


def prepare(case, seed):
    ctx = semo.Context(precision=case["precision"], reuse_hierarchy=not case["rebuild"])
    call = case["call"]
    if call in ("coo_p", "coo_m"):
        return dict(case=case, ctx=ctx, system=_coo(case, seed))
    if call == "coupled":
        c = _gas_case(case, seed)
        ctx.set_coupled_case(c)
        old, old2 = c.history()
        return dict(case=case, ctx=ctx, fields=[_pinned(a) for a in (c.P, c.U, c.V, c.W, c.T)], old=_pinned(old),
                    old2=_pinned(old2))
    c = _hex_case(case, seed)
    ctx.set_case(c)
    nc = c.mesh.n_cells
    s = dict(case=case, ctx=ctx, fields=[_pinned(a) for a in (c.P, c.U, c.V, c.W, c.VF)],
             out={k: _pinned(np.zeros(nc)) for k in ("P", "U", "V", "W")})
    if call == "adjoint":
        # d/dx of the sum of squares of a target's misfit on the top cells
        dJ = np.zeros(nc)
        top = c.mesh.patch_cells("zmax")
        dJ[top] = np.random.default_rng(seed + 1).uniform(-1.0, 1.0, size=top.size)
        s["dJ"] = dJ
    return s


# -------------------------------------------------------------------- a pass
def run(state):
    ctx, call = state["ctx"], state["case"]["call"]
    if call == "coo_p":
        rows, cols, vals, b = state["system"]
        return {"x0": ctx.solve_amgcl("pressure", 1, rows, cols, vals, b[0]).x}
    if call == "coo_m":
        rows, cols, vals, b = state["system"]
        return {"x%d" % j: r.x for j, r in enumerate(ctx.solve_amgcl("momentum", 1, rows, cols, vals, *b))}
    if call == "coupled":
        ctx.set_coupled_fields(*state["fields"], state["old"], state["old2"])
        norm, _ = ctx.calc_comp_coupled_eq()
        return dict(ctx.coupled_fields(), norm=norm)
    ctx.set_fields(*state["fields"])
    if call == "adjoint":
        ctx.assemble()
        x = ctx.solve().x
        lam, grad, _ = ctx.vjp_fields(state["dJ"])
        return dict(grad, x=x, adjoint=lam)
    out = {}
    if call in ("step", "vof"):
        out["norm_vf"], _ = ctx.calc_volfrac_eq()
    if call in ("outer", "step"):
        (out["norm_m"], out["norm_p"]), _ = ctx.outer_iteration()
    elif call == "pressure":
        out["norm_p"], _ = ctx.calc_pressure_eq()
    elif call == "momentum":
        out["norm_m"], _ = ctx.calc_momentum_eqs()
    elif call == "vof":
        return dict(out, VF=ctx.get_array("VF", ctx.n_cells))
    return dict(out, **ctx.fields(state["out"]))


# ------------------------------------------------------- what a pass must move
def work(case):
    """Mesh geometry, fields and systems read once, results written once; the gradients' arithmetic."""
    n, call = case["n"], case["call"]
    if call in ("coo_p", "coo_m"):
        N = n * (n + 3) * max(n - 1, 2)
        return {"bytes": 16.0 * 7 * N + (16.0 if call == "coo_p" else 48.0) * N, "flops": 14.0 * N}
    if call == "coupled":
        N, F = 6 * n ** 3, 12 * n ** 3
        return {"bytes": 120.0 * F + 8.0 * (20 + 10) * N, "flops": 2.0 * 25 * (N + 2 * F) + 2.0 * 15 * 60 * N}
    N, F = n ** 3, 3 * n ** 2 * (n + 1)
    fields = {"outer": 5 + 6 + 4, "step": 5 + 6 + 2 + 5, "pressure": 5 + 4, "momentum": 5 + 6 + 4, "vof": 5 + 2 + 1,
              "adjoint": 5 + 1 + 6}[call]
    passes = {"outer": 2, "step": 3, "adjoint": 2}.get(call, 1)
    # a face: two cells, normal, area, weight, distance, alpha, direction, skewness; a cell: volume, LSQ inverse, stencil
    return {"bytes": 112.0 * F + (8.0 * (1 + 6 + fields) + 4.0 * 26) * N, "flops": passes * 2.0 * 15 * 26 * N}


# ----------------------------------------------------------- 64-bit references
def _solve_coo(case, seed):
    """The COO system in torch FP64: conjugate gradients or Jacobi iteration, to rounding."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rows, cols, vals, b = _coo(case, seed)
    N = b.shape[1]
    r, c, v = (torch.as_tensor(a, device=dev) for a in (rows.astype(np.int64), cols.astype(np.int64), vals))
    A = torch.sparse_coo_tensor(torch.stack([r, c]), v, (N, N)).coalesce().to_sparse_csr()
    d, B = v[:N, None], torch.as_tensor(b.T.copy(), device=dev)
    x = torch.zeros_like(B)
    if case["call"] == "coo_m":   # strictly diagonally dominant
        for _ in range(400):
            res = B - A @ x
            if float(res.norm() / B.norm()) < 1e-15:
                break
            x += res / d
        return {"x%d" % j: x[:, j].cpu().numpy() for j in range(3)}
    for _ in range(3):   # restarted from the true residual
        res = B - A @ x
        z = res / d
        p, rz, first = z.clone(), (res * z).sum(), float(res.norm())
        for it in range(6000):
            q = A @ p
            alpha = rz / (p * q).sum()
            x += alpha * p
            res -= alpha * q
            if it % 50 == 0 and float(res.norm()) < 1e-12 * max(first, 1e-3 * float(B.norm())):
                break
            z = res / d
            new = (res * z).sum()
            p = z + (new / rz) * p
            rz = new
    return {"x0": x[:, 0].cpu().numpy()}


class _Lattice:
    """SEMO's discretisation on the plain n^3 box of one fluid (rho = 1, mu = 1e-3), where every face is
    orthogonal: cells as (z, y, x) arrays, pressure 0 on zmax, zero gradient elsewhere."""

    dt, mu, urf = BOX_DT, 1e-3, 0.3

    def __init__(self, n):
        self.n, self.h = n, 1.0 / n

    def shift(self, f, ax, by, ghost):
        """f of the neighbour along ax (by = +-1), ghost on the boundary plane."""
        g = np.empty_like(f)
        src, dst, end = [slice(None)] * 3, [slice(None)] * 3, [slice(None)] * 3
        src[ax], dst[ax], end[ax] = ((slice(1, None), slice(None, -1), -1) if by > 0
                                     else (slice(None, -1), slice(1, None), 0))
        g[tuple(dst)] = f[tuple(src)]
        g[tuple(end)] = ghost[tuple(end)] if isinstance(ghost, np.ndarray) else ghost
        return g

    def gradient(self, f, top=None):
        """Least squares over the vertex neighbours and the boundary faces (weight 1/d^2); top: the value on zmax."""
        n, h = self.n, self.h
        pad, live = np.zeros((n + 2,) * 3), np.zeros((n + 2,) * 3)
        pad[1:-1, 1:-1, 1:-1], live[1:-1, 1:-1, 1:-1] = f, 1.0
        M, r = np.zeros((3, 3, n, n, n)), np.zeros((3, n, n, n))
        for off in np.ndindex(3, 3, 3):
            d = (np.array(off) - 1) * h   # (z, y, x)
            if not d.any():
                continue
            at = tuple(slice(o, o + n) for o in off)
            w = live[at] / (d @ d)
            for a in range(3):
                r[a] += w * d[a] * (pad[at] - f)
                for b in range(3):
                    M[a, b] += w * d[a] * d[b]
        for a in range(3):
            for end, sign in ((0, -1.0), (n - 1, 1.0)):
                at = [slice(None)] * 3
                at[a] = end
                at = tuple(at)
                M[a, a][at] += 1.0
                if top is not None and a == 0 and sign > 0:
                    r[a][at] += 2.0 / h * (top - f[at])
        return np.moveaxis(np.linalg.solve(np.moveaxis(M, (0, 1), (3, 4)), np.moveaxis(r, 0, 3)[..., None])[..., 0],
                           3, 0)

    def face_velocity(self, P, u, gP, ax):
        """Normal velocity of the faces between a cell and its upper neighbour along ax (last plane unused)."""
        up = lambda f: self.shift(f, ax, 1, 0.0)  # noqa: E731
        return (0.5 * (u[ax] + up(u[ax])) - self.dt * (up(P) - P) / self.h + 0.5 * self.dt * (gP[ax] + up(gP[ax])))

    def boundary_velocity(self, P, u, gP, ax, sign):
        at = self.plane(ax, sign)
        un = sign * u[ax][at]
        if ax == 0 and sign > 0:
            un = un + self.dt * P[at] / (0.5 * self.h) + self.dt * gP[0][at]
        return un

    def plane(self, ax, sign):
        at = [slice(None)] * 3
        at[ax] = self.n - 1 if sign > 0 else 0
        return tuple(at)

    def momentum(self, P, u, old, old2):
        n, h, mu = self.n, self.h, self.mu
        A, V = h * h, h ** 3
        gP, gu = self.gradient(P, 0.0), [self.gradient(f) for f in u]
        diag = np.full((n,) * 3, 1.5 * V / self.dt)
        b = [-(1.5 * u[c] - 2.0 * old[c] + 0.5 * old2[c]) * V / self.dt for c in range(3)]
        off = {}
        inner = lambda ax: tuple(slice(None, -1) if a == ax else slice(None) for a in range(3))  # noqa: E731
        outer = lambda ax: tuple(slice(1, None) if a == ax else slice(None) for a in range(3))  # noqa: E731
        ad = mu * A / h
        for ax in range(3):
            lo, hi = inner(ax), outer(ax)
            mf = self.face_velocity(P, u, gP, ax)[lo] * A
            pos, neg = np.maximum(mf, 0.0), np.minimum(mf, 0.0)
            diag[lo] += pos + ad
            diag[hi] -= neg - ad
            off[ax] = (neg - ad, -pos - ad)
            mx, mn = self.limits(P)
            PF = 0.5 * (P[lo] + P[hi])
            PF = np.maximum(mn[lo], np.minimum(mx[lo], PF))
            PF = np.maximum(mn[hi], np.minimum(mx[hi], PF))
            for c in range(3):
                uf = np.where(mf > 0.0, u[c][lo], u[c][hi])
                base = mf * uf - ad * (u[c][hi] - u[c][lo]) + (PF * A if c == ax else 0.0)
                b[c][lo] -= base - mu * A * gu[c][ax][lo]
                b[c][hi] += base - mu * A * gu[c][ax][hi]
            for sign in (-1.0, 1.0):
                at = self.plane(ax, sign)
                un = self.boundary_velocity(P, u, gP, ax, sign)
                pb = 0.0 if (ax == 0 and sign > 0) else P[at]
                diag[at] += un * A
                for c in range(3):
                    extra = sign * gu[c][ax][at]   # the grad.n terms of the boundary face
                    b[c][at] -= u[c][at] * un * A + (sign * pb * A if c == ax else 0.0) - mu * A * extra
        def mv(x):
            y = diag * x
            for ax in range(3):
                lo, hi = inner(ax), outer(ax)
                y[lo] += off[ax][0] * x[hi]
                y[hi] += off[ax][1] * x[lo]
            return y
        new = []
        for c in range(3):   # the time term dominates the diagonal: Jacobi iteration to rounding
            x, best = np.zeros_like(diag), math.inf
            while True:
                r = b[c] - mv(x)
                if not np.linalg.norm(r) < 0.95 * best:
                    break
                best = np.linalg.norm(r)
                x += r / diag
            new.append(u[c] + self.urf * x)
        den = math.sqrt(sum(float((f ** 2).sum()) for f in new))
        num = math.sqrt(sum(float(((f - g) ** 2).sum()) for f, g in zip(new, u))) / self.urf
        return new, num / den

    def limits(self, f):
        e = np.pad(f, 1, mode="edge")
        n = self.n
        win = [e[tuple(slice(o, o + n) for o in off)] for off in np.ndindex(3, 3, 3)]
        return np.max(win, axis=0), np.min(win, axis=0)

    def pressure(self, P, u):
        n, h, dt = self.n, self.h, self.dt
        A, V = h * h, h ** 3
        gP = self.gradient(P, 0.0)
        b = np.zeros((n,) * 3)
        for ax in range(3):
            lo = tuple(slice(None, -1) if a == ax else slice(None) for a in range(3))
            hi = tuple(slice(1, None) if a == ax else slice(None) for a in range(3))
            flux = self.face_velocity(P, u, gP, ax)[lo] * A
            b[lo] -= flux
            b[hi] += flux
            for sign in (-1.0, 1.0):
                at = self.plane(ax, sign)
                b[at] -= self.boundary_velocity(P, u, gP, ax, sign) * A
        # the Laplacian is separable: eigenvectors of the 1-D operators (Neumann in x and y, fixed value on zmax)
        def one(fixed):
            T = 2.0 * np.eye(n) - np.eye(n, k=1) - np.eye(n, k=-1)
            T[0, 0], T[-1, -1] = 1.0, 3.0 if fixed else 1.0
            return np.linalg.eigh(T)
        (lz, Qz), (ly, Qy) = one(True), one(False)
        k = dt / h * A
        y = np.einsum("zyx,za,yb,xc->abc", b, Qz, Qy, Qy, optimize=True)
        y /= k * (lz[:, None, None] + ly[None, :, None] + ly[None, None, :])
        x = np.einsum("abc,za,yb,xc->zyx", y, Qz, Qy, Qy, optimize=True)
        g = []
        for ax in range(3):
            upf = 0.5 * (x + self.shift(x, ax, 1, x))
            dnf = 0.5 * (x + self.shift(x, ax, -1, x))
            if ax == 0:
                upf[self.plane(0, 1.0)] = 0.0
            g.append((upf - dnf) * A / V)
        Pn = P + self.urf * x
        un = [f - self.urf * dt * d for f, d in zip(u, g)]
        num = (x ** 2).sum() + sum(((self.urf * dt * d) ** 2).sum() for d in g)
        den = (Pn ** 2).sum() + sum((f ** 2).sum() for f in un)
        return Pn, un, math.sqrt(float(num)) / math.sqrt(float(den))


def exact(case, seed):
    """What run() returns, in 64 bits without this package: the caller-supplied systems, and the calls on the plain
    box, whose discretisation is short enough to be written down again."""
    call, n = case["call"], case["n"]
    if call in ("coo_p", "coo_m"):
        return _solve_coo(case, seed)
    if case["fluid"] != "box" or call not in ("outer", "pressure", "momentum") or n > 40:
        return None
    c = _hex_case(case, seed)
    grid = lambda f: f.reshape(n, n, n)  # noqa: E731
    L, P = _Lattice(n), grid(c.P)
    u = [grid(f) for f in (c.W, c.V, c.U)]   # (z, y, x) as the axes
    out = {}
    if call in ("outer", "momentum"):
        u, out["norm_m"] = L.momentum(P, u, [grid(f) for f in c.old[::-1]], [grid(f) for f in c.old2[::-1]])
    if call in ("outer", "pressure"):
        P, u, out["norm_p"] = L.pressure(P, u)
    return dict(out, P=P.reshape(-1), U=u[2].reshape(-1), V=u[1].reshape(-1), W=u[0].reshape(-1))
