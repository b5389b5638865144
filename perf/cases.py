"""The work a user of this framework has it do, as cases that can be timed and compared.

A case is a call sequence through the public entry points (``dpgsolver_gb300.solver`` and the C ABI of
``include/dgpu.h`` behind it) at one size: explicit residuals, SSP-RK3 time stepping with the state on the device or in
the caller's pinned host memory, uniform QUAD/HEX meshes, meshes of mixed order and mixed element type, Navier-Stokes,
and the two linearisations (adjoint of a time march, directional derivative). The meshes are the ones of the
framework's own tests and benchmark. Everything is FP64, the only type the framework has.

``exact`` evaluates the same discretisation with dense operators in plain torch, in 64 bits, from the arrays a caller
hands to the library (operators, geometric factors, connectivity, state).
"""
import ctypes
import functools
import math

import numpy as np
import torch

from dpgsolver_gb300 import _lib, solver
from dpgsolver_gb300.host import mixed, mixed_types, problem

_ROE, _LF = problem.NUM_FLUX_ROE_PIKE, problem.NUM_FLUX_LAX_FRIEDRICHS


# ---- the cases ------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one residual of the linear advection test mesh, where launches and latency are everything
        {"name": "advection_quad16_p2_rhs", "kind": "rhs", "mesh": "advection", "d": 2, "n": 16, "p": 2,
         "flux": "upwind"},
        # the 2D isentropic vortex march (the framework's 2D benchmark mesh), many short steps
        {"name": "vortex_quad64_p3_steps", "kind": "steps", "mesh": "vortex", "d": 2, "n": 64, "p": 3, "flux": "roe",
         "steps": 20},
        # the headline mesh: a resolved 3D Euler march with the state resident on the device; the largest case
        {"name": "vortex_hex32_p3_steps", "kind": "steps", "mesh": "vortex", "d": 3, "n": 32, "p": 3, "flux": "lf",
         "steps": 5},
        # one time step of a host code that keeps its state in its own pinned memory
        {"name": "vortex_hex32_p3_host_step", "kind": "host_step", "mesh": "vortex", "d": 3, "n": 32, "p": 3,
         "flux": "lf"},
        # a bounded domain (supersonic in- and outflow, slip walls, characteristic sides) with an odd number of volumes
        {"name": "duct_hex21_p2_steps", "kind": "steps", "mesh": "duct", "d": 3, "n": 21, "p": 2, "flux": "roe",
         "steps": 5},
        # the residual alone (an outer solver's function evaluation) at the highest order
        {"name": "vortex_hex15_p4_rhs", "kind": "rhs", "mesh": "vortex", "d": 3, "n": 15, "p": 4, "flux": "roe"},
        # viscous march: Taylor-Green vortex
        {"name": "taylor_green_hex24_p3_steps", "kind": "steps", "mesh": "taylor_green", "d": 3, "n": 24, "p": 3,
         "flux": "roe", "steps": 3},
        # a p-adapted HEX mesh
        {"name": "mixed_order_hex20_steps", "kind": "batch_steps", "mesh": "mixed_order", "d": 3, "n": 20, "p": 4,
         "flux": "roe", "steps": 4},
        # an unstructured-style 3D mesh: HEX, TET, WEDGE and PYR volumes of several orders
        {"name": "mixed_types_18_steps", "kind": "batch_steps", "mesh": "mixed_types", "d": 3, "n": 18, "p": 4,
         "flux": "roe", "steps": 4},
        # a 2D mesh of QUADs and TRIs of several orders
        {"name": "tri_quad_96_steps", "kind": "batch_steps", "mesh": "tri_quad", "d": 2, "n": 96, "p": 4,
         "flux": "roe", "steps": 4},
        # sensitivity of an output after a short march (checkpointed discrete adjoint)
        {"name": "adjoint_hex12_p3", "kind": "adjoint", "mesh": "vortex", "d": 3, "n": 12, "p": 3, "flux": "lf",
         "steps": 4},
        # the matrix-free product of an implicit solver
        {"name": "jvp_hex17_p2", "kind": "jvp", "mesh": "vortex", "d": 3, "n": 17, "p": 2, "flux": "roe"},
    ]


_MAX_WORK = 32 ** 3 * 4 ** 3 * 5 * 15   # state values times residuals of the largest listed case


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, every order, both fluxes."""
    kind, mesh, d = rng.choice([
        ("rhs", "advection", 2), ("rhs", "vortex", 2), ("rhs", "vortex", 3), ("steps", "vortex", 2),
        ("steps", "vortex", 3), ("steps", "vortex", 3), ("host_step", "vortex", 3), ("host_step", "vortex", 2),
        ("steps", "duct", 3), ("steps", "taylor_green", 3), ("rhs", "taylor_green", 3),
        ("batch_steps", "mixed_order", 2), ("batch_steps", "mixed_order", 3), ("batch_steps", "mixed_types", 3),
        ("batch_steps", "tri_quad", 2), ("batch_steps", "mixed_ns", 3), ("adjoint", "vortex", 3),
        ("jvp", "vortex", 2), ("jvp", "vortex", 3), ("jvp", "taylor_green", 3)])
    p = rng.randint(2, 4) if kind == "batch_steps" else rng.randint(1, 4)
    lo, hi = {("batch_steps", 2): (12, 120), ("batch_steps", 3): (6, 18), ("adjoint", 3): (6, 12)}.get(
        (kind, d), (8, 128) if d == 2 else (5, 32))
    if mesh in ("taylor_green", "mixed_ns"):
        hi = 16
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if mesh == "mixed_types":
        n += n % 2   # this mesh's blocks need an even count
    c = {"kind": kind, "mesh": mesh, "d": d, "n": n, "p": p,
         "flux": "upwind" if mesh == "advection" else rng.choice(["roe", "lf"])}
    if kind in ("steps", "batch_steps", "adjoint"):
        c["steps"] = rng.randint(2, 4) if kind == "adjoint" else rng.randint(2, 8)
    weight = {"taylor_green": 4, "mixed_ns": 4}.get(mesh, 1)   # gradients, liftings and viscous fluxes on top
    while c["n"] ** d * (p + 1) ** d * (d + 2) * weight * 3 * c.get("steps", 1) > _MAX_WORK and c["n"] > 6:
        c["n"] -= 2
    return c


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _key(case):
    return tuple(case[k] for k in ("mesh", "d", "n", "p", "flux"))


@functools.lru_cache(maxsize=2)
def _problem(mesh, d, n, p, flux):
    """Mesh, operators, geometry and base state (what a caller reads from its own files; the seed does not enter)."""
    fx = _LF if flux == "lf" else _ROE
    if mesh == "advection":
        return problem.advection_2d(n, p)
    if mesh == "vortex":
        return problem.euler_vortex_2d(n, p, num_flux=fx) if d == 2 else \
            problem.euler_hex_3d(n, p, num_flux=fx, perturb=0.0)
    if mesh == "duct":
        return problem.euler_duct_3d(n, p, num_flux=fx)
    if mesh == "taylor_green":
        return problem.ns_taylor_green(n, p, num_flux=fx)
    orders = tuple(range(1, p + 1))
    if mesh == "mixed_order":
        return mixed.mixed_euler(d, n, p_set=orders, num_flux=fx)
    if mesh == "mixed_ns":
        return mixed.mixed_ns(d, n, p_set=orders, num_flux=fx)
    if mesh == "mixed_types":
        return mixed_types.mixed_types_euler(n, p_set=orders, num_flux=fx)
    return mixed_types.mixed_tri_quad_euler(n, p_set=orders, num_flux=fx, perturb=0.05)


def _noise(b, d, rng):
    """Seeded noise on blocks (volumes, variables, basis): 1e-3 relative on the density (or the advected scalar), 1e-3
    absolute on the momentum, so that no velocity component is exactly zero."""
    b[:, 0] *= 1.0 + 1e-3 * rng.uniform(-1.0, 1.0, size=b[:, 0].shape)
    if b.shape[1] > 1:
        b[:, 1:1 + d] += 1e-3 * rng.uniform(-1.0, 1.0, size=b[:, 1:1 + d].shape)
    return b


def _state(prob, seed):
    rng = np.random.default_rng(seed)
    sol = prob.sol.copy()
    if sol.ndim == 3:
        return _noise(sol, prob.d, rng)
    for g in range(len(prob.groups)):
        if len(prob.group_vols[g]):
            prob.set_group(sol, g, _noise(prob.group_view(sol, g), prob.d, rng))
    return sol


def _direction(prob, seed):
    return np.random.default_rng(seed + 1).uniform(-1.0, 1.0, size=prob.sol.shape)


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64))
    return t.pin_memory() if torch.cuda.is_available() else t


def _ptr(t):
    return ctypes.cast(t.data_ptr(), _lib.c_double_p)


def prepare(case, seed):
    prob = _problem(*_key(case))
    sol = _state(prob, seed)
    sim = solver.BatchSimulation(prob) if case["kind"] == "batch_steps" else solver.Simulation(prob)
    s = {"case": case, "sim": sim, "dt": prob.dt, "out": _pinned(np.zeros_like(sol))}
    if case["kind"] in ("host_step", "jvp", "adjoint"):
        s["sol"] = _pinned(sol)
    else:
        sim.upload_state(sol)
    if case["kind"] == "jvp":
        s["dir"] = _pinned(_direction(prob, seed))
        s["rhs"] = _pinned(np.zeros_like(sol))
    if case["kind"] == "adjoint":
        sim.set_objective_faces(prob.faces_on_plane(2))
        s["budget"] = 64 * 8 * int(sol.size)
    return s


def run(state):
    case, sim, out = state["case"], state["sim"], state["out"]
    lib, h, kind = _lib.load(), sim._h, case["kind"]
    if kind == "rhs":
        mx = solver.compute_rhs_dg(sim)
        _lib.check(lib.dgpu_download_rhs(h, _ptr(out)), h)
        return {"rhs": out, "max_rhs": mx}
    if kind == "steps":
        mx = solver.solve_explicit(sim, case["steps"], state["dt"])
        _lib.check(lib.dgpu_download_state(h, _ptr(out)), h)
        return {"sol": out, "max_rhs": mx}
    if kind == "batch_steps":
        mx = sim.ssp_rk3_steps(state["dt"], case["steps"])
        _lib.check(lib.dgpu_batch_download_state(h, _ptr(out)), h, batch=True)
        return {"sol": out, "max_rhs": mx}
    if kind == "host_step":
        mx = ctypes.c_double()
        _lib.check(lib.dgpu_ssp_rk3_step_host(h, state["dt"], _ptr(state["sol"]), _ptr(out), ctypes.byref(mx)), h)
        return {"sol": out, "max_rhs": mx.value}
    if kind == "jvp":
        _lib.check(lib.dgpu_jvp(h, _ptr(state["sol"]), _ptr(state["dir"]), _ptr(state["rhs"]), _ptr(out)), h)
        return {"rhs": state["rhs"], "jv": out}
    J = ctypes.c_double()
    _lib.check(lib.dgpu_adjoint_ssp_rk3(h, state["dt"], case["steps"], state["budget"], _ptr(state["sol"]),
                                        ctypes.byref(J), _ptr(out), None), h)
    return {"J": J.value, "gradient": out}


def work(case):
    """The state, the geometric factors and the outputs once each; the sum-factorised passes and the pointwise fluxes
    of every residual (a backward or tangent evaluation counted as twice its residual)."""
    prob = _problem(*_key(case))
    d, nv, kind = prob.d, prob.n_var, case["kind"]
    groups = prob.groups if hasattr(prob, "groups") else [prob.ops]
    count = [len(v) for v in prob.group_vols] if hasattr(prob, "groups") else [prob.n_volumes]
    nodes = sum(c * int(g.n_vc) for c, g in zip(count, groups))
    face_nodes = int(prob.face_off[-1]) if hasattr(prob, "face_off") else prob.mesh.n_faces * prob.ops.n_fc
    per_eval = face_nodes * (2.0 if nv == 1 else 200.0)
    for c, g in zip(count, groups):
        if getattr(g, "dense", False):   # dense operators: V, D_k^T, M^-1 and the faces
            per_eval += c * (2.0 * nv * g.n_vs * (g.n_vc * (1 + d) + g.n_vs) + g.n_vc * 60.0)
        else:                            # 1D passes: volume term, traces and lifting of the 2d faces
            per_eval += c * g.n_vc * (2.0 * nv * (d * g.q + 4 * d) + (6.0 if nv == 1 else 90.0))
    ns = prob.ns if getattr(prob, "ns", None) is not None else None
    if ns is not None:                   # gradients of every variable, their liftings and traces, the viscous flux
        per_eval *= 1.0 + d / 2.0
    evals = {"rhs": 1, "jvp": 3, "host_step": 3, "adjoint": 3 * 3 * case.get("steps", 1)}.get(
        kind, 3 * case.get("steps", 1))
    state = 8.0 * int(np.size(prob.sol))
    io = {"jvp": 4}.get(kind, 2)
    return {"bytes": io * state + 8.0 * (nodes * (d * d + 1) + face_nodes * (d + 1)), "flops": evals * per_eval}


# ---- the same discretisation with dense operators ------------------------------------------------------------------------
_GAMMA, _GM1 = 1.4, 0.4


def _lagrange(xn, x):
    L = np.ones((len(x), len(xn)))
    for j in range(len(xn)):
        for m in range(len(xn)):
            if m != j:
                L[:, j] *= (x - xn[m]) / (xn[j] - xn[m])
    return L


def _kron(ops):
    """Tensor product with the first direction fastest."""
    out = ops[0]
    for o in ops[1:]:
        out = np.kron(o, out)
    return out


class _Dense:
    """The caller's arrays regrouped for batched products."""

    def __init__(self, prob):
        self.dev = dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        fl = problem.flat_arrays(prob)
        self.d, self.nv, self.pde = prob.d, int(prob.n_var), prob.pde
        self.flux, self.ns, self.b = prob.num_flux, getattr(prob, "ns", None), prob.b_adv
        d, nv, mesh = self.d, self.nv, prob.mesh

        def T(a):
            return torch.tensor(a, device=dev)
        vg = np.asarray(fl["vol_group"])
        n_vs = np.array([int(g.n_vs) for g in fl["groups"]])[vg]
        n_vc = np.array([int(g.n_vc) for g in fl["groups"]])[vg]
        off = np.concatenate([[0], np.cumsum(nv * n_vs)])
        voff = np.concatenate([[0], np.cumsum(n_vc)])
        pos = np.zeros(len(vg), dtype=np.int64)
        self.G = []
        for g, ops in enumerate(fl["groups"]):
            v = np.nonzero(vg == g)[0]
            pos[v] = np.arange(len(v))
            nq, ns_ = int(ops.n_vc), int(ops.n_vs)
            idx = off[v][:, None] + np.arange(nv * ns_)
            midx = (d * d * voff[v])[:, None] + np.arange(d * d * nq)
            m = np.asarray(fl["metrics_vc"])[midx].reshape(len(v), d, d, nq)     # [j][i][node]
            J = np.asarray(fl["jacobian_det_vc"])[voff[v][:, None] + np.arange(nq)]
            V = np.asarray(ops.cv0_vs_vc())
            G = {"idx": T(idx), "shape": (len(v), nv, ns_), "m": T(m), "V": T(V),
                 "D": T(np.stack([np.asarray(ops.cv1_vs_vc(k)) for k in range(d)])), "w": T(np.asarray(ops.w_vc))}
            if nq == ns_ and not getattr(ops, "dense", False):
                G["Vinv"], G["iwJ"] = T(np.linalg.inv(V)), T(1.0 / (np.asarray(ops.w_vc) * J))
            else:
                G["M"] = torch.einsum("na,vn,nb->vab", T(V), T(np.asarray(ops.w_vc) * J), T(V))
            self.G.append(G)
        nf = mesh.n_faces
        foff = np.asarray(prob.face_off) if hasattr(prob, "face_off") else np.arange(nf + 1) * prob.ops.n_fc
        n_fc = np.diff(foff)
        self.rows = int(foff[-1])
        self.n = T(np.asarray(fl["normals_fc"]).reshape(-1, d))
        self.jf = T(np.asarray(fl["jacobian_det_fc"]))
        inner = np.repeat(mesh.face_vol[:, 1] >= 0, n_fc)
        perm = np.repeat(foff[:-1], n_fc) + np.asarray(fl["nc_fc"])
        self.perm = T(np.where(inner, perm, np.arange(self.rows)))
        fo = fl.get("face_ord")
        fo = np.zeros((nf, 2), dtype=np.int64) if fo is None else np.asarray(fo)
        self.sides = [[], []]
        for s in (0, 1):
            sel = np.nonzero(mesh.face_vol[:, s] >= 0)[0]
            keys = np.stack([vg[mesh.face_vol[sel, s]], mesh.face_lf[sel, s], fo[sel, s],
                             np.asarray(fl["face_q"])[sel]], axis=1)
            uniq, inv = np.unique(keys, axis=0, return_inverse=True)
            for u, (g, lf, o, qf) in enumerate(uniq):
                f = sel[np.ravel(inv) == u]
                E, w = self._face_op(fl["groups"][g], int(lf), int(o), int(qf))
                rows = foff[f][:, None] + np.arange(len(w))
                self.sides[s].append((int(g), T(pos[mesh.face_vol[f, s]]), T(rows.ravel()), T(E), T(w)))
        if fl.get("bc_fc") is not None:
            self.bc = T(np.repeat(np.where(mesh.face_vol[:, 1] < 0, np.asarray(fl["bc_fc"]) % 10000, 0), n_fc))
            self.ext = T(np.asarray(fl["bc_state_fc"]).reshape(-1, nv))
        else:
            self.bc = None

    def _face_op(self, ops, lf, o, qf):
        if getattr(ops, "dense", False):
            return np.asarray(ops.cv0_vs_fc(lf, o, qf)), np.asarray(ops.w_fc(lf, qf))
        x, w = np.polynomial.legendre.leggauss(qf)
        xn, end = np.asarray(ops.x_vs), np.array([1.0 if lf % 2 else -1.0])
        E = _kron([_lagrange(xn, end if k == lf // 2 else x) for k in range(self.d)])
        return E, _kron([w] * (self.d - 1))

    # -- pieces of the residual
    def _minv(self, G, r):
        if "Vinv" in G:
            return ((r @ G["Vinv"]) * G["iwJ"][:, None, :]) @ G["Vinv"].T
        return torch.linalg.solve(G["M"], r.transpose(1, 2)).transpose(1, 2)

    def _traces(self, coef, s):
        """Side s's coefficients (list of (volumes, k, n_vs)) at every face node, (face nodes, k)."""
        k = coef[0].shape[1]
        out = torch.zeros((self.rows, k), dtype=torch.float64, device=self.dev)
        for g, v, rows, E, _ in self.sides[s]:
            out = out.index_copy(0, rows, (coef[g][v] @ E.T).transpose(1, 2).reshape(-1, k))
        return out

    def _lift(self, acc, face, s):
        """acc[g] += E^T w face over side s's faces."""
        for g, v, rows, E, w in self.sides[s]:
            b = face[rows].reshape(len(v), len(w), -1).transpose(1, 2)
            acc[g] = acc[g].index_add(0, v, (b * w) @ E)
        return acc

    def _unperm(self, face):
        return torch.zeros_like(face).index_copy(0, self.perm, face)

    def _pressure(self, W):
        m = W[1:-1]
        return _GM1 * (W[-1] - 0.5 * (m * m).sum(0) / W[0])

    def _flux(self, W):
        """Physical flux [direction][equation] of W (equation, ...)."""
        if self.nv == 1:
            return [[float(self.b[i]) * W[0]] for i in range(self.d)]
        u, p = W[1:-1] / W[0], self._pressure(W)
        return [[W[1 + i]] + [W[1 + k] * u[i] + (p if k == i else 0.0) for k in range(self.d)] + [(W[-1] + p) * u[i]]
                for i in range(self.d)]

    def _viscous(self, W, g):
        """Viscous flux [direction][equation] (equation 0 zero) of W and its gradient g[direction] (equation, ...)."""
        d, mu, Pr = self.d, self.ns["mu"], self.ns["Pr"]
        rho, E, u = W[0], W[-1], W[1:-1] / W[0]
        du = [[(g[x][1 + s] - g[x][0] * u[s]) / rho for x in range(d)] for s in range(d)]
        div = sum(du[k][k] for k in range(d))
        tau = [[mu * (du[a][b] + du[b][a] - (2.0 / 3.0 * div if a == b else 0.0)) for b in range(d)] for a in range(d)]
        out = []
        for x in range(d):
            dT = (g[x][-1] * rho - E * g[x][0]) / (rho * rho) - sum(u[k] * du[k][x] for k in range(d))
            out.append([torch.zeros_like(rho)] + [tau[k][x] for k in range(d)] +
                       [_GAMMA / Pr * mu * dT + sum(u[k] * tau[x][k] for k in range(d))])
        return out

    def _numerical(self, L, R, n):
        """Normal numerical flux of traces L, R (equation, node) and normals n (direction, node)."""
        d = self.d
        if self.nv == 1:
            bn = sum(float(self.b[i]) * n[i] for i in range(d))
            return torch.where(bn > 1e-15, bn * L[0], bn * R[0])[None]
        FL, FR = self._flux(L), self._flux(R)
        F = torch.stack([sum(n[i] * (FL[i][k] + FR[i][k]) for i in range(d)) for k in range(d + 2)])
        uL, uR, pL, pR = L[1:-1] / L[0], R[1:-1] / R[0], self._pressure(L), self._pressure(R)
        if self.flux == _LF:
            lam = [torch.sqrt((u * u).sum(0)) + torch.sqrt(_GAMMA * p / W[0])
                   for u, p, W in ((uL, pL, L), (uR, pR, R))]
            return 0.5 * (F + torch.where(lam[0] > lam[1], lam[0], lam[1]) * (L - R))
        VL, VR = (n * uL).sum(0), (n * uR).sum(0)
        r = torch.sqrt(R[0] / L[0])
        u, rho = (r * uR + uL) / (r + 1.0), r * L[0]
        H = (r * (R[-1] + pR) / R[0] + (L[-1] + pL) / L[0]) / (r + 1.0)
        Vn = (n * u).sum(0)
        c = torch.sqrt(_GM1 * (H - 0.5 * (u * u).sum(0)))
        a, b = VL - c, Vn - c
        l1 = torch.where(a.abs() < b.abs(), a, b).abs()
        a, b = VR + c, Vn + c
        l5, l = torch.where(a.abs() > b.abs(), a, b).abs(), torch.where(Vn > 0.0, Vn, -Vn)
        dp, dV = pR - pL, VR - VL
        x1, x2 = 0.5 * (l5 + l1) - l, 0.5 * (l5 - l1)
        D1 = x1 * dp / (c * c) + x2 * rho * dV / c
        D2 = x1 * rho * dV + x2 * dp / c
        dis = l * (R - L) + torch.cat([D1[None], D1 * u + D2 * n, (D1 * H + D2 * Vn)[None]])
        return 0.5 * (F - dis)

    def _outside(self, L, R, n):
        """R with the boundary values on the boundary faces' nodes (slip wall, characteristic, supersonic)."""
        if self.bc is None:
            return R
        e, bc = self.ext.T, self.bc
        wall = torch.cat([L[:1], L[1:-1] - 2.0 * (n * L[1:-1]).sum(0) * n, L[-1:]])
        e1 = torch.where(bc == 101, e, L)   # other nodes: any admissible state
        uL, uR, pL, pR = L[1:-1] / L[0], e1[1:-1] / e1[0], self._pressure(L), self._pressure(e1)
        VL, VR = (n * uL).sum(0), (n * uR).sum(0)
        cL, cR = torch.sqrt(_GAMMA * pL / L[0]), torch.sqrt(_GAMMA * pR / e1[0])
        a, b = VL + 2.0 / _GM1 * cL, VR - 2.0 / _GM1 * cR
        V, c = 0.5 * (a + b), 0.25 * _GM1 * (a - b)
        c2 = c * c / _GAMMA
        inflow, sup = V < 0.0, V.abs() >= c.abs()
        s = torch.where(inflow, pR / e1[0] ** _GAMMA, pL / L[0] ** _GAMMA)
        rho = torch.where(sup, torch.where(inflow, e1[0], L[0]), (c2 / s) ** (1.0 / _GM1))
        p = torch.where(sup, torch.where(inflow, pR, pL), c2 * rho)
        ut = torch.where(inflow, uR - VR * n, uL - VL * n)
        uu = torch.where(sup, torch.where(inflow, uR, uL), V * n + ut)
        far = torch.cat([rho[None], rho * uu, (p / _GM1 + 0.5 * rho * (uu * uu).sum(0))[None]])
        for code, val in ((101, far), (102, wall), (105, e), (106, L)):
            R = torch.where(bc == code, val, R)
        return R

    def residual(self, sol):
        d = self.d
        c = [sol[G["idx"]].reshape(G["shape"]) for G in self.G]
        n = self.n.T
        L = self._traces(c, 0).T
        R = self._outside(L, self._traces(c, 1)[self.perm].T, n)
        if self.ns is not None:   # BR2: volume gradient, liftings of the jump, gradients at the faces
            gv, gt, gL, gR = [], [], [], []
            for x in range(d):
                a = [self._minv(G, ((sum(G["m"][:, k, x][:, None] * (c_ @ G["D"][k].T) for k in range(d)))
                                    * G["w"]) @ G["V"]) for G, c_ in zip(self.G, c)]
                X = (self.jf * n[x] * 0.5 * (R - L)).T
                lift = [self._lift([torch.zeros_like(b) for b in c], X, 0),
                        self._lift([torch.zeros_like(b) for b in c], self._unperm(X), 1)]
                gv.append(a)
                gt.append([b + self._minv(G, l0 + l1) for G, b, l0, l1 in zip(self.G, a, *lift)])
                own = [X, self._unperm(X)]
                face = []
                for s in (0, 1):   # the face's own lifting only, scaled by 1.01 * 2 d
                    t = self._traces(a, s)
                    for g, v, rows, E, w in self.sides[s]:
                        G = self.G[g]
                        b = (own[s][rows].reshape(len(v), len(w), -1).transpose(1, 2) * w) @ E
                        sub = {k: (G[k][v] if k in ("iwJ", "M") else G[k]) for k in G if k in ("Vinv", "iwJ", "M")}
                        b = self._minv(sub, b) @ E.T
                        t = t.index_add(0, rows, 1.01 * 2 * d * b.transpose(1, 2).reshape(len(rows), -1))
                    face.append(t)
                gL.append(face[0].T)
                gR.append(face[1][self.perm].T)
        rhs = []
        for g, (G, c_) in enumerate(zip(self.G, c)):
            W = (c_ @ G["V"].T).transpose(0, 1)                                   # (equation, volume, node)
            F = self._flux(W)
            if self.ns is not None:
                Q = self._viscous(W, [(gt[x][g] @ G["V"].T).transpose(0, 1) for x in range(d)])
                F = [[F[x][k] - Q[x][k] for k in range(d + 2)] for x in range(d)]
            F = [torch.stack(f) for f in F]
            rhs.append(sum(((sum(G["m"][:, j, i] * F[i] for i in range(d)) * G["w"]).transpose(0, 1)) @ G["D"][j]
                           for j in range(d)))
        nF = self._numerical(L, R, n)
        if self.ns is not None:
            QL, QR = self._viscous(L, gL), self._viscous(R, gR)
            nF = nF - torch.stack([sum(0.5 * n[x] * (QL[x][k] + QR[x][k]) for x in range(d)) for k in range(d + 2)])
        nF = (nF * self.jf).T
        rhs = self._lift(rhs, -nF, 0)
        rhs = self._lift(rhs, self._unperm(nF), 1)
        out = torch.zeros_like(sol)
        for G, r in zip(self.G, rhs):
            out = out.index_copy(0, G["idx"].ravel(), self._minv(G, r).reshape(-1))
        return out

    def march(self, sol, dt, steps):
        """SSP-RK3 steps; the new state and the last stage's residual."""
        r = None
        for _ in range(steps):
            u = sol + dt * self.residual(sol)
            u = 0.25 * (3.0 * sol + u + dt * self.residual(u))
            r = self.residual(u)
            sol = (sol + 2.0 * u + 2.0 * dt * r) / 3.0
        return sol, r


def exact(case, seed):
    prob = _problem(*_key(case))
    kind = case["kind"]
    D = _Dense(prob)
    state = _state(prob, seed)
    sol = torch.as_tensor(state.ravel(), device=D.dev)

    def host(t):
        return t.detach().reshape(state.shape).cpu()
    if kind == "rhs":
        r = D.residual(sol)
        return {"rhs": host(r), "max_rhs": float(r.abs().max())}
    if kind in ("steps", "host_step", "batch_steps"):
        u, r = D.march(sol, prob.dt, case.get("steps", 1))
        return {"sol": host(u), "max_rhs": float(r.abs().max())}
    if kind == "jvp":
        v = torch.as_tensor(_direction(prob, seed).ravel(), device=D.dev)
        r, jv = torch.func.jvp(D.residual, (sol,), (v,))
        return {"rhs": host(r), "jv": host(jv)}
    # pressure over side 0 of the objective faces, after the march
    faces = prob.faces_on_plane(2)
    rows = torch.as_tensor((np.asarray(faces)[:, None] * prob.ops.n_fc + np.arange(prob.ops.n_fc)).ravel(),
                           device=D.dev)
    w = torch.as_tensor(np.tile(_kron([np.asarray(prob.ops.w_vc_1d)] * (prob.d - 1)), len(faces)), device=D.dev)
    u0 = sol.clone().requires_grad_(True)
    u, _ = D.march(u0, prob.dt, case["steps"])
    W = D._traces([u[D.G[0]["idx"]].reshape(D.G[0]["shape"])], 0)[rows].T
    J = (w * D.jf[rows] * D._pressure(W)).sum()
    J.backward()
    return {"J": float(J.detach()), "gradient": host(u0.grad)}
