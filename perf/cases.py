"""The work a flow solver has this library do, as cases that can be timed and
checked: residuals of the explicit and implicit paths, pseudo-time steps,
Newton steps, exact linearisations and sensitivity solves, all through the
public classes of ``aerof_dev_b200`` on the jittered Kuhn tet meshes of the
benchmark configurations.

A case is a dict of plain values; ``prepare`` makes its state from a seed,
``run`` is one pass, ``exact`` the same result in plain 64-bit torch.  A mesh
and its context are kept between states, as a solver keeps them between
calls; every state has its own flow field.
"""
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import aerof_dev_b200 as A
from aerof_dev_b200 import workloads as W

GAMMA, BETA = 1.4, 1.0 / 3.0
VISC = {"reynolds_mu": 2000.0, "prandtl": 0.72, "sutherland_alpha": 1.3, "sutherland_Ts": 0.35}
NU_REF = 1e-3
RECS = {"constant": A.REC_CONSTANT, "vanalbada": A.REC_VANALBADA, "linear": A.REC_LINEAR}


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the first-order far-field run of a small mesh: ten explicit steps,
        # where launches and waits are most of the time
        {"name": "rk2_21", "kind": "rk2", "n": 21, "codes": "farfield", "rec": "constant", "mach": 0.5, "steps": 10},
        # the piece of a decomposed mesh: an odd size of ordinary extent,
        # unlimited reconstruction
        {"name": "residual_47", "kind": "residual", "n": 47, "codes": "channel", "rec": "linear", "mach": 0.8,
         "host": False},
        # the second-order residual of the benchmark configuration
        {"name": "residual_101", "kind": "residual", "n": 101, "codes": "channel", "rec": "vanalbada", "mach": 0.8,
         "host": False},
        # the same from page-locked host arrays, as a host solver that owns
        # the state calls it
        {"name": "residual_host_101", "kind": "residual", "n": 101, "codes": "channel", "rec": "vanalbada",
         "mach": 0.8, "host": True},
        # nodal gradients of a primitive field for the caller's own terms
        {"name": "gradients_61", "kind": "gradients", "n": 61, "codes": "channel", "rec": "vanalbada", "mach": 0.8},
        # laminar flow: the residual with the viscous Galerkin term
        {"name": "laminar_61", "kind": "galerkin", "n": 61, "codes": "channel", "rec": "vanalbada", "mach": 0.8,
         "model": "laminar"},
        # turbulent flow: six variables, Spalart-Allmaras source and diffusion
        {"name": "turbulent_81", "kind": "galerkin", "n": 81, "codes": "channel", "rec": "vanalbada", "mach": 0.8,
         "model": "sa"},
        # a caller's own pseudo-time step: residual, local time step, H1
        # operator, block-Jacobi, twenty GMRES iterations
        {"name": "pseudo_step_81", "kind": "pseudo_step", "n": 81, "codes": "channel", "rec": "vanalbada",
         "mach": 0.8, "precision": 32, "cfl": 1e3, "its": 20},
        # the library's own Newton driver, mixed precision
        {"name": "newton_61", "kind": "newton", "n": 61, "codes": "channel", "rec": "vanalbada", "mach": 0.8,
         "precision": 32, "pc": "jacobi", "steps": 5},
        # both products of the adjoint gradient from one reverse sweep
        {"name": "adjoint_101", "kind": "adjoint", "n": 101, "codes": "channel", "rec": "vanalbada", "mach": 0.8},
        # forward products: J v and the right-hand side (dR/dX) Xdot of one
        # shape mode
        {"name": "forward_61", "kind": "forward", "n": 61, "codes": "channel", "rec": "vanalbada", "mach": 0.8,
         "stored": False},
        # direct sensitivities of several shape modes in one batched solve
        {"name": "sensitivities_41", "kind": "sensitivities", "n": 41, "codes": "channel", "rec": "vanalbada",
         "mach": 0.8, "pc": "ilu", "modes": 4},
    ]


# kind -> (weight, smallest lattice, largest lattice)
_RANGE = {"rk2": (2, 7, 41), "residual": (4, 9, 101), "gradients": (1, 9, 81), "galerkin": (2, 11, 81),
          "pseudo_step": (2, 13, 81), "newton": (2, 13, 61), "adjoint": (2, 11, 101), "forward": (2, 11, 71),
          "sensitivities": (1, 13, 41)}


def draw(rng):
    kind = rng.choices(list(_RANGE), [r[0] for r in _RANGE.values()])[0]
    lo, hi = _RANGE[kind][1:]
    c = {"kind": kind, "n": int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))),
         "codes": rng.choice(["channel", "channel", "farfield"]), "rec": "vanalbada",
         "mach": round(rng.uniform(0.4, 0.85), 3)}
    if kind == "rk2":
        c["rec"] = rng.choice(["constant", "vanalbada", "linear"])
        c["steps"] = rng.randint(2, 10)
    elif kind == "residual":
        c["rec"] = rng.choice(["constant", "vanalbada", "vanalbada", "linear"])
        c["host"] = rng.random() < 0.25
    elif kind == "galerkin":
        c["rec"] = rng.choice(["vanalbada", "linear"])
        c["model"] = rng.choice(["laminar", "sa"])
    elif kind == "pseudo_step":
        c["precision"] = rng.choice([32, 32, 64])
        c["cfl"] = round(10.0 ** rng.uniform(1.0, 4.0), 2)
        c["its"] = rng.randint(8, 30)
    elif kind == "newton":
        c["precision"] = rng.choice([32, 32, 64])
        c["pc"] = rng.choice(["jacobi", "jacobi", "ilu"])
        c["steps"] = rng.randint(2, 5)
    elif kind == "adjoint":
        c["rec"] = rng.choice(["constant", "vanalbada", "vanalbada", "linear"])
    elif kind == "forward":
        c["rec"] = rng.choice(["vanalbada", "vanalbada", "linear"])
        c["stored"] = rng.random() < 0.5
    elif kind == "sensitivities":
        c["pc"] = rng.choice(["jacobi", "ilu"])
        c["modes"] = rng.randint(2, 4)
    return c


# ------------------------------------------------------------------ states
_MESHES, _CONTEXTS = {}, {}


def _mesh(case):
    key = (case["n"], case["codes"])
    if key not in _MESHES:
        if len(_MESHES) >= 12:
            _MESHES.pop(next(iter(_MESHES)))
        _MESHES[key] = W.make_lattice_mesh(case["n"], jitter=0.2, codes=case["codes"])
    return _MESHES[key]


def _wall_distance(m):
    return np.abs(m["X"][:, 2]) + 0.02 * m["X"][:, 0]


def _freestream6(mach):
    return np.concatenate([W.freestream(mach), [NU_REF]])


def _context(case):
    """The solver's context: one per mesh, scheme and model."""
    key = (case["n"], case["codes"], case["rec"], case["mach"], case.get("model"), case.get("pc"))
    if key not in _CONTEXTS:
        if len(_CONTEXTS) >= 12:
            _CONTEXTS.pop(next(iter(_CONTEXTS))).close()
        m = _mesh(case)
        ctx = A.Context.from_mesh(m, W.freestream(case["mach"]), reconstruction=RECS[case["rec"]], gamma=GAMMA,
                                  beta=BETA)
        if case.get("model"):
            ctx.set_viscosity(model=2, **VISC)
        if case.get("model") == "sa":
            ctx.set_turbulence(_wall_distance(m), _freestream6(case["mach"]))
        if case.get("pc") == "ilu":
            ctx.set_preconditioner(A.PC_ILU0)
        _CONTEXTS[key] = ctx
    return _CONTEXTS[key]


def _flow(case, seed):
    """A flow field away from the free stream, [N][5] on the GPU: a smooth
    disturbance of seeded phase plus 0.2 % noise, in primitive variables, and
    the generator for the state's other arrays."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    X = torch.from_numpy(_mesh(case)["X"]).cuda()
    N = X.shape[0]
    ph = 2.0 * math.pi * torch.rand(5, 3, generator=g, device="cuda", dtype=torch.float64)
    s = torch.stack([torch.sin(math.pi * X[:, 0] + ph[k, 0]) * torch.sin(math.pi * X[:, 1] + ph[k, 1])
                     * torch.sin(math.pi * X[:, 2] + ph[k, 2]) for k in range(5)], dim=1)
    s = 0.02 * s + 0.002 * torch.randn(N, 5, generator=g, device="cuda", dtype=torch.float64)
    p0 = 1.0 / (GAMMA * case["mach"] ** 2)
    V = torch.stack([1.0 + s[:, 0], 1.0 + s[:, 1], s[:, 2], s[:, 3], p0 * (1.0 + s[:, 4])], dim=1)
    return V, g


def _cons(V):
    E = V[:, 4] / (GAMMA - 1.0) + 0.5 * V[:, 0] * (V[:, 1:4] ** 2).sum(1)
    return torch.cat([V[:, :1], V[:, :1] * V[:, 1:4], E[:, None]], dim=1).contiguous()


def _inputs(case, seed):
    """The arrays of a state, on the GPU."""
    V, g = _flow(case, seed)
    N, kind = V.shape[0], case["kind"]
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    s = {"U": _cons(V)}
    if kind == "gradients":
        s["V"] = V.contiguous()
    elif kind == "galerkin" and case["model"] == "sa":
        X = torch.from_numpy(_mesh(case)["X"]).cuda()
        bump = torch.exp(-((X - 0.5) ** 2).sum(1) / 0.05)
        nu = NU_REF * (1.0 + 4.0 * bump) * (1.0 + 0.1 * torch.rand(N, generator=g, device="cuda",
                                                                    dtype=torch.float64))
        s["U"] = torch.cat([s["U"], (V[:, 0] * nu)[:, None]], dim=1).contiguous()
    elif kind == "adjoint":
        s["lam"] = rand(N, 5)
    elif kind in ("forward", "sensitivities"):
        modes = W.shape_modes(_mesh(case)["X"], case.get("modes", 1), seed=int(seed) % (1 << 31))
        s["Xdot"] = torch.from_numpy(modes).cuda()
        if kind == "forward":
            s["v"], s["w"] = rand(N, 5), rand(N, 5)
    return s


def prepare(case, seed):
    s = {"case": case, "ctx": _context(case), **_inputs(case, seed)}
    if case.get("host"):
        s["U"] = s["U"].cpu().pin_memory().numpy()
        s["R"] = torch.empty(s["U"].shape, dtype=torch.float64, pin_memory=True).numpy()
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "rk2":
        return A.ExplicitRK2(ctx, 0.8).run(s["U"], case["steps"])
    if kind == "residual":
        return A.SpaceOperator(ctx).computeResidual(s["U"], s.get("R"))
    if kind == "gradients":
        return A.SpaceOperator(ctx).computeGradients(s["V"])
    if kind == "galerkin":
        sp = A.SpaceOperator(ctx)
        return sp.computeResidualSA(s["U"]) if case["model"] == "sa" else sp.computeResidual(s["U"])
    if kind == "pseudo_step":
        sp = A.SpaceOperator(ctx)
        R, bad = sp.computeResidual(s["U"])
        dt = sp.computeTimeStep(s["U"], case["cfl"])
        A.MatVecProdH1(ctx, case["precision"]).evaluate(s["U"], dt)
        A.JacobiPrec(ctx).setup()
        x, its, res = A.GmresSolver(ctx, 30, case["its"], 0.0).solve(-R)
        return {"R": R, "bad": bad, "dt": dt, "dU": x, "its": its, "res": res}
    if kind == "newton":
        U, info = A.ImplicitSteadySolver(ctx, precision=case["precision"], max_steps=case["steps"]).solve(s["U"])
        return {"U": U, "history": info["history"]}
    if kind == "adjoint":
        return A.Sensitivity(ctx).adjoint_products(s["U"], s["lam"])
    if kind == "forward":
        S = A.Sensitivity(ctx)
        if case["stored"]:
            S.h2_evaluate(s["U"])
            return S.h2_apply(s["v"]), S.h2_apply(s["w"], transpose=True)
        return S.jvp(s["U"], s["v"]), S.dRdX(s["U"], s["Xdot"][0])
    S = A.Sensitivity(ctx)
    B = torch.stack([S.dRdX(s["U"], x) for x in s["Xdot"]])
    # a bounded number of outer iterations: every mode takes them all
    X, its, res = S.solve_batch(s["U"], B, krylov=30, maxits=24, eps=1e-10, inner_its=10)
    return {"B": B, "X": X, "its": its, "res": res}


# ------------------------------------------------------------------ work
def work(case):
    """Bytes of the arrays a pass cannot do without (state, results, node and
    edge geometry, operator blocks, Krylov vectors: each once where the
    algorithm lets it be once) and floating-point operations."""
    z = W.lattice_sizes(case["n"])
    N, E, T, F = z["N"], z["E"], z["T"], z["F"]
    second = case["rec"] != "constant"
    grad_f = (90 * 2 * E if second else 0)
    res_b = 32 * E + (80 + 8 + 24 + (48 if second else 0)) * N + 40 * F
    res_f = (450 if second else 170) * E + grad_f + 30 * N
    dt_b, dt_f = 32 * E + (40 + 8 + 8) * N, 40 * E
    kind = case["kind"]
    if kind == "rk2":
        return {"bytes": case["steps"] * (2 * res_b + dt_b), "flops": case["steps"] * (2 * res_f + dt_f)}
    if kind == "residual":
        return {"bytes": res_b, "flops": res_f}
    if kind == "gradients":
        return {"bytes": 8 * E + (40 + 24 + 48 + 120) * N, "flops": grad_f}
    if kind == "galerkin":
        w = 6 if case["model"] == "sa" else 5
        return {"bytes": res_b * w / 5 + 16 * T, "flops": res_f * w / 5 + 350 * T}
    if kind in ("pseudo_step", "newton"):
        s = case["precision"] // 8
        its = case.get("its", 10)
        vec = 5 * N * s
        op_b = 8 * E + 25 * s * (N + 2 * E) + 2 * vec
        op_f = 50 * (N + 2 * E)
        b = res_b + dt_b + its * op_b + its * (its + 1) / 2 * vec
        f = res_f + dt_f + 400 * E + its * op_f + its * (its + 1) * 20 * N
        k = case.get("steps", 1)
        return {"bytes": k * b, "flops": k * f}
    if kind == "adjoint":
        return {"bytes": res_b + (40 + 24) * N + 16 * T, "flops": res_f + 1100 * E + 250 * T}
    if kind == "forward":
        if case["stored"]:
            return {"bytes": res_b + 3 * 560 * E + 240 * N, "flops": res_f + 3500 * E}
        return {"bytes": 2 * (res_b + 64 * N) + 16 * T, "flops": 2 * 3 * res_f + 250 * T}
    its = 24 * case["modes"]
    return {"bytes": its * (560 * E + 10 * (25 * 4 * (N + 2 * E))) / case["modes"], "flops": its * 10 * 50 * (N + 2 * E)}


# About four times what was measured.  64-bit results: 5e-14 to 7e-14 of
# exact() (the fluxes cancel to about 1e-2 of their size), 1e-16 to 5e-16
# without that cancellation, up to 1.6e-13 for the transposed products.  The
# solve of a step: 9e-8 to 1.6e-7 with the 32-bit operator, 2e-8 to 6e-8 with
# the 64-bit one (round-off in the forward differences of its far-field
# blocks).  With the 32-bit operator's blocks formed in 64 bits and rounded
# once, Newton's state differs by up to 7e-10 and its history by 1.1e-8, the
# sensitivities by 5e-9 and their residual norms by 2.6e-7.
def tolerance(case):
    kind = case["kind"]
    if kind == "pseudo_step":
        return {"rel": 6e-7 if case["precision"] == 32 else 3e-7}
    if kind == "newton":
        return {"rel": 5e-8}
    if kind == "sensitivities":
        return {"rel": 1e-6}
    return {"rel": 6e-13 if kind in ("adjoint", "forward") else 3e-13}


# ------------------------------------------------------------------ exact
# The same equations in plain 64-bit torch.  |A|, A+ and A- of the Euler flux
# are applied through f(A) q = f1 q + (s1 b/c^2 + s2 a/c) (1, u, H)
# + (s1 a + s2 b/c) (0, n, un), a = n.m - un rho, b = (gam - 1)(q2/2 rho -
# u.m + E), s1 = (f+ + f-)/2 - f1, s2 = (f+ - f-)/2.
CHUNK = 1 << 20


class _Topology:
    def __init__(self, m):
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).long().cuda()  # noqa: E731
        self.N = m["X"].shape[0]
        self.tets, self.faces = t(m["tets"]), t(m["faces"])
        self.wall = t(m["codes"]) == W.BC_SLIP_WALL_MOVING
        ends = torch.tensor([[0, 1], [0, 2], [0, 3], [1, 2], [1, 3], [2, 3]], device="cuda")
        e = self.tets[:, ends]
        self.sign = torch.where(e[..., 0] < e[..., 1], 1.0, -1.0).double()
        key, inv = torch.unique(e.amin(-1) * self.N + e.amax(-1), return_inverse=True)
        self.tet_edge = inv
        self.i, self.j = key // self.N, key % self.N

    def geometry(self, X):
        x = X[self.tets]
        c = torch.linalg.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0])
        v = ((x[:, 3] - x[:, 0]) * c).sum(1) / 24.0
        vol = torch.zeros(self.N, dtype=X.dtype, device=X.device)
        for k in range(4):
            vol = vol.index_add(0, self.tets[:, k], v)
        f = torch.stack([x[:, 0] + x[:, 1] + x[:, 2], x[:, 0] + x[:, 1] + x[:, 3], x[:, 0] + x[:, 2] + x[:, 3],
                         x[:, 1] + x[:, 2] + x[:, 3]], 1) / 3.0 - x.mean(1, keepdim=True)
        en = torch.zeros(self.i.numel(), 3, dtype=X.dtype, device=X.device)
        for k, (a, b) in enumerate([(0, 1), (2, 0), (1, 2), (0, 3), (3, 1), (2, 3)]):
            n = 1.5 * torch.linalg.cross(f[:, b], f[:, a]) * self.sign[:, k, None]
            en = en.index_add(0, self.tet_edge[:, k], n)
        y = X[self.faces]
        fn = 0.5 * torch.linalg.cross(y[:, 2] - y[:, 0], y[:, 1] - y[:, 0])
        return vol, en, fn

    def gradients(self, X, V):
        """Least-squares gradients [N][3][C]."""
        N, C = V.shape
        S = torch.zeros(N, 9, dtype=V.dtype, device=V.device)
        M = torch.zeros(N, 3 * C, dtype=V.dtype, device=V.device)
        for c in range(0, self.i.numel(), CHUNK):
            i, j = self.i[c:c + CHUNK], self.j[c:c + CHUNK]
            d, dv = X[j] - X[i], V[j] - V[i]
            dd = (d[:, :, None] * d[:, None, :]).reshape(-1, 9)
            m = (d[:, :, None] * dv[:, None, :]).reshape(-1, 3 * C)
            S = S.index_add(0, i, dd).index_add(0, j, dd)
            M = M.index_add(0, i, m).index_add(0, j, m)
        a = S.reshape(N, 3, 3)
        r = [torch.linalg.cross(a[:, 1], a[:, 2]), torch.linalg.cross(a[:, 2], a[:, 0]),
             torch.linalg.cross(a[:, 0], a[:, 1])]
        inv = torch.stack(r, 2) / (a[:, 0] * r[0]).sum(1)[:, None, None]
        return inv @ M.reshape(N, 3, C)


_TOPOLOGY = {}


def _topology(case):
    key = (case["n"], case["codes"])
    if key not in _TOPOLOGY:
        _TOPOLOGY.clear()
        _TOPOLOGY[key] = _Topology(_mesh(case))
    return _TOPOLOGY[key]


def _prim(U):
    u = U[:, 1:4] / U[:, :1]
    p = (GAMMA - 1.0) * (U[:, 4] - 0.5 * U[:, 0] * (u * u).sum(1))
    return torch.cat([U[:, :1], u, p[:, None], U[:, 5:] / U[:, :1]], dim=1)


def _limited(a, b):
    eps, ab = 1e-16, a * b
    num = torch.where(ab > 0, a * (b * b + eps) + b * (a * a + eps),
                      torch.where(ab == 0, 0.5 * eps * (a + b), torch.zeros_like(a)))
    return num / (a * a + b * b + 2 * eps)


def _reconstruct(rec, dx, Vi, Gi, Vj, Gj):
    if rec == "constant":
        return Vi, Vj
    di, dj, d = (dx[:, None] @ Gi)[:, 0], (dx[:, None] @ Gj)[:, 0], Vj - Vi
    if rec == "linear":
        return Vi + (0.5 - BETA) * d + BETA * di, Vj - (0.5 - BETA) * d - BETA * dj
    b2 = (1 - 2 * BETA) * d
    return Vi + 0.5 * _limited(b2 + 2 * BETA * di, d), Vj - 0.5 * _limited(b2 + 2 * BETA * dj, d)


def _cons5(V):
    return _cons(V[:, :5])


def _roe_average(Vi, Vj):
    wi, wj = Vi[:, 0].sqrt(), Vj[:, 0].sqrt()
    u = (wi[:, None] * Vi[:, 1:4] + wj[:, None] * Vj[:, 1:4]) / (wi + wj)[:, None]
    Hi, Hj = ((_cons5(V)[:, 4] + V[:, 4]) / V[:, 0] for V in (Vi, Vj))
    H = (wi * Hi + wj * Hj) / (wi + wj)
    return u, H, ((GAMMA - 1.0) * (H - 0.5 * (u * u).sum(1))).sqrt()


def _apply(f1, fp, fm, n, u, H, c, q):
    """f(A) q for the eigenvalue functions f1, f+, f- (unit normal n)."""
    un = (u * n).sum(-1)
    a = (n * q[..., 1:4]).sum(-1) - un * q[..., 0]
    b = (GAMMA - 1.0) * (0.5 * (u * u).sum(-1) * q[..., 0] - (u * q[..., 1:4]).sum(-1) + q[..., 4])
    s1, s2 = 0.5 * (fp + fm) - f1, 0.5 * (fp - fm)
    k1, k2 = s1 * b / (c * c) + s2 * a / c, s1 * a + s2 * b / c
    one, zero = torch.ones_like(un)[..., None], torch.zeros_like(un)[..., None]
    r1, r2 = torch.cat([one, u, H[..., None]], -1), torch.cat([zero, n, un[..., None]], -1)
    return f1[..., None] * q + k1[..., None] * r1 + k2[..., None] * r2


def _roe_flux(n, Vi, Vj):
    """Upwind selection of the physical flux plus the dissipation of the one
    acoustic wave that opposes it; a sixth variable is advected."""
    S = (n * n).sum(1).sqrt()
    e = n / S[:, None]
    u, H, c = _roe_average(Vi[:, :5], Vj[:, :5])
    un = (u * e).sum(1)
    left = un > 0
    Vs = torch.where(left[:, None], Vi, Vj)
    m = Vs[:, 0] * (Vs[:, 1:4] * e).sum(1)
    Us = _cons5(Vs)
    f = torch.cat([m[:, None], m[:, None] * Vs[:, 1:4] + Vs[:, 4:5] * e, (m / Vs[:, 0] * (Us[:, 4] + Vs[:, 4]))[:, None]], 1)
    q = _cons5(Vj) - _cons5(Vi)
    z = torch.zeros_like(un)
    lam = torch.clamp(torch.where(left, un - c, un + c), max=0.0) * left + torch.clamp(un + c, min=0.0) * (~left)
    # f = F_i + A- dq (left) or F_j - A+ dq (right), only the acoustic wave
    # that runs against un
    add = _apply(z, torch.where(left, z, lam), torch.where(left, lam, z), e, u, H, c, q)
    f = f + torch.where(left[:, None], add, -add)
    if Vi.shape[1] > 5:
        f = torch.cat([f, (f[:, 0] * torch.where(f[:, 0] >= 0, Vi[:, 5], Vj[:, 5]))[:, None]], 1)
    return f * S[:, None]


def _face_flux(wall, n, V, Ub):
    """Slip wall, or Steger-Warming A+(V) U(V) + A-(V) Ub."""
    S = (n * n).sum(1).sqrt()
    e = n / S[:, None]
    U5, u = _cons5(V), V[:, 1:4]
    c = (GAMMA * V[:, 4] / V[:, 0]).sqrt()
    H, un = (U5[:, 4] + V[:, 4]) / V[:, 0], (u * e).sum(1)
    pos = [torch.clamp(x, min=0.0) for x in (un, un + c, un - c)]
    neg = [torch.clamp(x, max=0.0) for x in (un, un + c, un - c)]
    far = _apply(*pos, e, u, H, c, U5) + _apply(*neg, e, u, H, c, Ub[:5].expand_as(U5))
    z = torch.zeros_like(un)[:, None]
    f = torch.where(wall[:, None], torch.cat([z, V[:, 4:5] * e, z], 1), far)
    if V.shape[1] > 5:
        adv = f[:, 0] * torch.where(f[:, 0] >= 0, V[:, 5], Ub[5] / Ub[0])
        f = torch.cat([f, torch.where(wall, torch.zeros_like(adv), adv)[:, None]], 1)
    return f * S[:, None]


def _edge_chunk(rec, i, j, X, V, G, en):
    Vi, Vj = _reconstruct(rec, X[j] - X[i], V[i], G[i] if G is not None else None, V[j],
                          G[j] if G is not None else None)
    return _roe_flux(en, Vi, Vj)


def _galerkin(case, t, X, V, d2w):
    """vol (r . grad N_k) of the laminar or Spalart-Allmaras Galerkin term,
    summed per node (component 0 is zero)."""
    sa = V.shape[1] > 5
    out = torch.zeros(t.N, V.shape[1], dtype=V.dtype, device=V.device)
    ore, cp = 1.0 / VISC["reynolds_mu"], GAMMA / (GAMMA - 1.0)
    for c in range(0, t.tets.shape[0], CHUNK):
        nd = t.tets[c:c + CHUNK]
        x, v = X[nd], V[nd]
        J = x[:, 1:] - x[:, :1]
        g = torch.linalg.inv(J)
        g = torch.cat([-g.sum(2, keepdim=True), g], 2).transpose(1, 2)
        vol = torch.linalg.det(J) / 6.0
        T = v[..., 4] / (v[..., 0] * (GAMMA - 1.0))
        du = torch.einsum("tkj,tka->taj", g, v[..., 1:4])
        dT = torch.einsum("tkj,tk->tj", g, T)
        Ta = VISC["sutherland_alpha"] * T.mean(1)
        mul = Ta ** 1.5 * (1.0 + VISC["sutherland_Ts"]) / (Ta + VISC["sutherland_Ts"])
        mu, lam, kap = mul, -2.0 / 3.0 * mul, cp * mul / VISC["prandtl"]
        if sa:
            mt = (v[..., 0] * v[..., 5]).mean(1)
            mut = mt * (mt / mul) ** 3 / ((mt / mul) ** 3 + 7.1 ** 3)
            mu, lam, kap = mu + mut, lam - 2.0 / 3.0 * mut, kap + cp * mut / 0.9
        tau = ore * (mu[:, None, None] * (du + du.transpose(1, 2))
                     + (lam * du.diagonal(dim1=1, dim2=2).sum(1))[:, None, None] * torch.eye(3, device=V.device))
        q = (tau @ v[..., 1:4].mean(1)[..., None])[..., 0] + ore * kap[:, None] * dT
        share = torch.cat([torch.zeros_like(T)[..., None], torch.einsum("tkj,taj->tka", g, tau),
                           torch.einsum("tkj,tj->tk", g, q)[..., None]], 2)
        if sa:
            dnu = torch.einsum("tkj,tk->tj", g, v[..., 5])
            chi = torch.clamp(mt / mul, min=0.001)
            fv1 = chi ** 3 / (chi ** 3 + 7.1 ** 3)
            d2, rho = d2w[nd].mean(1) ** 2, v[..., 0].mean(1)
            z = ore / 0.41 ** 2 * torch.clamp(mt, min=0.0) / rho / d2
            w = torch.stack([du[:, 0, 1] - du[:, 1, 0], du[:, 1, 2] - du[:, 2, 1], du[:, 2, 0] - du[:, 0, 2]], 1)
            St = torch.clamp((w * w).sum(1).sqrt() + z * (1.0 - chi / (1.0 + chi * fv1)), min=1e-12)
            r = torch.clamp(z / St, max=2.0)
            gg = r + 0.3 * (r ** 6 - r)
            fw = gg * ((1.0 + 2.0 ** 6) / (gg ** 6 + 2.0 ** 6)) ** (1.0 / 6.0)
            sg = 1.5 * ore
            cw1 = (0.1355 / 0.41 ** 2 + 1.622 * 1.5) * ore
            src = (sg * 0.622 * rho * (dnu * dnu).sum(1) + 0.1355 * St * mt.abs()
                   - cw1 * fw / rho * torch.clamp(mt, min=0.0) ** 2 / d2)
            dif = sg * (mul + mt.abs())
            share = torch.cat([share, (dif[:, None] * torch.einsum("tkj,tj->tk", g, dnu) - 0.25 * src[:, None])[..., None]], 2)
        share = share * vol[:, None, None]
        out.index_add_(0, nd.reshape(-1), share.reshape(-1, V.shape[1]))
    return out


def _residual(case, t, X, U, geo=None):
    vol, en, fn = geo if geo is not None else t.geometry(X)
    V = _prim(U)
    Ub = torch.from_numpy(_freestream6(case["mach"])).cuda()
    rec = case["rec"]
    G = None if rec == "constant" else t.gradients(X, V)
    R = torch.zeros(t.N, U.shape[1], dtype=U.dtype, device=U.device)
    for c in range(0, t.i.numel(), CHUNK):
        i, j = t.i[c:c + CHUNK], t.j[c:c + CHUNK]
        a = (rec, i, j, X, V, G, en[c:c + CHUNK])
        f = checkpoint(_edge_chunk, *a, use_reentrant=False) if R.requires_grad or U.requires_grad else _edge_chunk(*a)
        R = R.index_add(0, i, f).index_add(0, j, -f)
    for k in range(3):
        nd = t.faces[:, k]
        R = R.index_add(0, nd, _face_flux(t.wall, fn / 3.0, V[nd], Ub))
    if case.get("model"):
        d2w = torch.from_numpy(_wall_distance(_mesh(case))).cuda()
        R = R + _galerkin(case, t, X, V, d2w)
    return R / vol[:, None]


def _timestep(t, geo, U, cfl):
    vol, en, fn = geo
    V = _prim(U)
    s = torch.zeros(t.N, dtype=U.dtype, device=U.device)
    S = (en * en).sum(1).sqrt()
    Vm = 0.5 * (V[t.i] + V[t.j])
    a, un = (GAMMA * Vm[:, 4] / Vm[:, 0]).sqrt(), (Vm[:, 1:4] * en).sum(1) / S
    s.index_add_(0, t.i, torch.clamp(un - a, max=0.0) * S).index_add_(0, t.j, torch.clamp(-un - a, max=0.0) * S)
    for k in range(3):
        v = V[t.faces[:, k]]
        a, S = (GAMMA * v[:, 4] / v[:, 0]).sqrt(), (fn * fn).sum(1).sqrt()
        s.index_add_(0, t.faces[:, k], torch.clamp((v[:, 1:4] * fn).sum(1) / S - a, max=0.0) * S / 3.0)
    return -cfl * vol / s


class _FirstOrder:
    """The first-order operator: approximate Roe Jacobians on the edges,
    face Jacobians (analytic wall, forward differences of the far-field flux
    with the step 1e-6 |V_k|), 1/vol, + I/dt; block-Jacobi and GMRES."""

    def __init__(self, case, t, geo, U, dt):
        vol, en, fn = geo
        self.t, self.V, self.iv = t, _prim(U), 1.0 / vol
        V, dev = self.V, U.device
        S = (en * en).sum(1).sqrt()
        e = en / S[:, None]
        eye = torch.eye(5, dtype=U.dtype, device=dev)
        D = torch.diag_embed((1.0 / dt)[:, None].expand(-1, 5)).contiguous()
        self.Aij, self.Aji = [], []
        for c in range(0, S.numel(), CHUNK):
            i, j, s, n = t.i[c:c + CHUNK], t.j[c:c + CHUNK], S[c:c + CHUNK], e[c:c + CHUNK, None]
            u, H, cs = (q[:, None] for q in _roe_average(V[i], V[j]))
            un, Q = (u * n).sum(-1), eye.expand(s.numel(), 5, 5)
            ab = _apply(un.abs(), (un + cs).abs(), (un - cs).abs(), n, u, H, cs, Q).transpose(1, 2)
            half = 0.5 * s[:, None, None]
            Hi, Hj = (self._flux_jac(V[k], e[c:c + CHUNK]) for k in (i, j))
            D.index_add_(0, i, (Hi + ab) * half * self.iv[i][:, None, None])
            D.index_add_(0, j, (ab - Hj) * half * self.iv[j][:, None, None])
            self.Aij.append((Hj - ab) * half * self.iv[i][:, None, None])
            self.Aji.append(-(Hi + ab) * half * self.iv[j][:, None, None])
        Ub = torch.from_numpy(_freestream6(case["mach"])).cuda()
        for k in range(3):
            nd = t.faces[:, k]
            D.index_add_(0, nd, self._face_jac(V[nd], fn / 3.0, Ub) * self.iv[nd][:, None, None])
        self.Aij, self.Aji, self.D, self.Dinv = torch.cat(self.Aij), torch.cat(self.Aji), D, torch.linalg.inv(D)

    @staticmethod
    def _flux_jac(V, n):
        eye = torch.eye(5, dtype=V.dtype, device=V.device).expand(V.shape[0], 5, 5)
        u, un, c = V[:, None, 1:4], (V[:, 1:4] * n).sum(1)[:, None], (GAMMA * V[:, 4] / V[:, 0]).sqrt()[:, None]
        H = ((_cons5(V)[:, 4] + V[:, 4]) / V[:, 0])[:, None]
        return _apply(un, un + c, un - c, n[:, None], u, H, c, eye).transpose(1, 2)

    def _face_jac(self, V, n, Ub):
        f0, cols = _face_flux(self.t.wall, n, V, Ub), []
        for k in range(5):
            e = torch.where(V[:, k].abs() < 1e-10, torch.full_like(V[:, k], 1e-6), 1e-6 * V[:, k])
            Ve = V.clone()
            Ve[:, k] += e
            fd = (_face_flux(self.t.wall, n, Ve, Ub) - f0) / e[:, None]
            wall = torch.cat([torch.zeros_like(n[:, :1]), n if k == 4 else torch.zeros_like(n), torch.zeros_like(n[:, :1])], 1)
            cols.append(torch.where(self.t.wall[:, None], wall, fd))
        dV = torch.zeros(V.shape[0], 5, 5, dtype=V.dtype, device=V.device)
        dV[:, 0, 0] = 1.0
        for a in (1, 2, 3):
            dV[:, a, 0], dV[:, a, a], dV[:, 4, a] = -V[:, a] / V[:, 0], 1.0 / V[:, 0], -(GAMMA - 1.0) * V[:, a]
        dV[:, 4, 0], dV[:, 4, 4] = 0.5 * (GAMMA - 1.0) * (V[:, 1:4] ** 2).sum(1), GAMMA - 1.0
        return torch.stack(cols, 2) @ dV

    def product(self, p):
        y = (self.D @ p[..., None])[..., 0]
        y.index_add_(0, self.t.i, (self.Aij @ p[self.t.j][..., None])[..., 0])
        return y.index_add_(0, self.t.j, (self.Aji @ p[self.t.i][..., None])[..., 0])

    def gmres(self, b, its):
        beta = b.norm()
        Q, Hm = [b / beta], torch.zeros(its + 1, its, dtype=b.dtype)
        for k in range(its):
            w = self.product((self.Dinv @ Q[k][..., None])[..., 0])
            for i in range(k + 1):
                h = (w * Q[i]).sum()
                Hm[i, k] = h
                w = w - h * Q[i]
            Hm[k + 1, k] = w.norm()
            Q.append(w / w.norm())
        g = torch.zeros(its + 1, 1, dtype=b.dtype)
        g[0, 0] = beta
        y = torch.linalg.lstsq(Hm, g).solution
        x = sum(float(y[k, 0]) * Q[k] for k in range(its))
        return (self.Dinv @ x[..., None])[..., 0], float((Hm @ y - g).norm())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("newton", "sensitivities"):
        return None
    t, s = _topology(case), _inputs(case, seed)
    X = torch.from_numpy(_mesh(case)["X"]).cuda()
    U = s["U"]
    if kind == "residual":
        R = _residual(case, t, X, U)
        return [R.cpu().numpy() if case["host"] else R, 0]
    if kind == "galerkin":
        return [_residual(case, t, X, U), 0]
    if kind == "gradients":
        return list(t.gradients(X, s["V"]).unbind(1))
    if kind == "rk2":
        geo = t.geometry(X)
        for _ in range(case["steps"]):
            dt = _timestep(t, geo, U, 0.8)[:, None]
            k1 = dt * _residual(case, t, X, U, geo)
            U = U - 0.5 * (k1 + dt * _residual(case, t, X, U - k1, geo))
        return [U, 0]
    if kind == "pseudo_step":
        geo = t.geometry(X)
        R, dt = _residual(case, t, X, U, geo), _timestep(t, geo, U, case["cfl"])
        x, res = _FirstOrder(case, t, geo, U, dt).gmres(-R, case["its"])
        return {"R": R, "bad": 0, "dt": dt, "dU": x, "its": case["its"], "res": res}
    if kind == "adjoint":
        Ug, Xg = U.clone().requires_grad_(), X.clone().requires_grad_()
        (_residual(case, t, Xg, Ug) * s["lam"]).sum().backward()
        return [Ug.grad, Xg.grad]
    f = lambda x, u: _residual(case, t, x, u)  # noqa: E731
    zX, zU = torch.zeros_like(X), torch.zeros_like(U)
    jv = torch.func.jvp(f, (X, U), (zX, s["v"]))[1]
    if case["stored"]:
        Ug = U.clone().requires_grad_()
        (_residual(case, t, X, Ug) * s["w"]).sum().backward()
        return [jv, Ug.grad]
    return [jv, torch.func.jvp(f, (X, U), (s["Xdot"][0], zU))[1]]
