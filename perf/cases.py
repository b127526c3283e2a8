"""Performance cases: the calls a user of this framework makes, at the sizes they make them.

The framework is a nonlinear-solve library, so most cases are whole solves through the public Python binding
(the nonlinear drivers with their multigrid or Jacobi preconditioners), beside the building blocks a program
calls on its own: an operator's evaluations and one multigrid V-cycle.  Sizes and parameters are those of the
benchmark, the published calibration campaigns and the tests; draw() varies them over the same ranges, with
ragged hierarchies (95 = 47, 23, 11, 5, 2 and the like) and even operator grids among them.  The learned
preconditioner is not a case: the solver is used without it.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parents[1] / "chebyshev-nonlinear-lab_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import numa_gpu as G  # noqa: E402

_CTX = None


def _ctx():
    """One context for the program, as an application keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = G.Context(0)
    return _CTX


class _Cai:
    """A device vector's memory for torch (CUDA array interface)."""

    def __init__(self, vec):
        self.vec = vec
        self.__cuda_array_interface__ = {"shape": (vec.n,), "typestr": "<f8", "data": (vec.device_ptr(), False),
                                         "version": 3, "strides": None}


def _tensor(vec):
    return torch.as_tensor(_Cai(vec), device="cuda")


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # The smallest calls: F(u), F'(u) v and F''(u)[v, v] of a 31^3 operator, as a program with its own
        # nonlinear loop makes them; launches and latency decide.
        {"name": "ops_31", "kind": "ops", "n": 31, "mode": "analytic"},
        # One application of the multigrid preconditioner inside somebody else's Krylov solver: the FP64 V(2,2)
        # that equals the reference's, and the FP32 one of the mixed path.
        {"name": "vcycle_fp64_63", "kind": "vcycle", "n": 63, "prec": "fp64"},
        {"name": "vcycle_fp32_127", "kind": "vcycle", "n": 127, "prec": "fp32"},
        # The drop-in solve (FP64, GMRES(30) with modified Gram-Schmidt, V(2,2), rtol 1e-10) at the campaign's
        # smallest and at an ordinary size.
        {"name": "nk_fp64_31", "kind": "nk", "n": 31, "lam": 6.0, "path": "fp64", "method": "nk"},
        {"name": "nk_fp64_127", "kind": "nk", "n": 127, "lam": 6.0, "path": "fp64", "method": "nk"},
        # The Chebyshev driver with a recycled Krylov space, on a hierarchy that ends in an even grid.
        {"name": "rec_fp64_95", "kind": "nk", "n": 95, "lam": 4.0, "path": "fp64", "method": "rec"},
        # The mixed path end to end from pinned host buffers (a service that solves one instance per request).
        {"name": "host_mixed_63", "kind": "host", "n": 63, "lam": 6.0},
        # The mixed path at the benchmark's size, start and solution on the device.
        {"name": "nk_mixed_255", "kind": "nk", "n": 255, "lam": 6.0, "path": "mixed", "method": "nk"},
        # The published calibration runs: point-Jacobi, GMRES(30) with up to 200 iterations a linear solve.
        {"name": "jacobi_31", "kind": "jacobi", "n": 31, "lam": 6.93, "method": "nk"},
        # The second problem family: an implicit Burgers step with the 2D Helmholtz multigrid (calibration runs).
        {"name": "burgers_255", "kind": "burgers", "n": 255, "nu": 0.02, "dt": 0.04, "method": "nk"},
        # The third: implicit steps of the periodic two-species Brusselator, mixed path.
        {"name": "bruss_2048", "kind": "bruss", "n": 2048, "steps": 2},
        # Many independent instances in one batched solver, solutions wanted on the host.
        {"name": "batch_32", "kind": "batch", "count": 32, "big": 63},
    ]


# grids whose halving chain reaches n <= 15 by odd sizes: (m + 1) 2^k - 1
_GRIDS = [31, 39, 47, 55, 63, 79, 95, 111, 127, 159, 191, 223, 255]


def draw(rng):
    kind = rng.choice(["ops", "vcycle", "vcycle", "fp64", "fp64", "host", "mixed", "jacobi", "burgers", "bruss",
                       "batch"])
    grid = lambda top: rng.choice([g for g in _GRIDS if g <= top])  # noqa: E731
    lam = round(rng.uniform(1.0, 6.5), 3)
    if kind == "ops":
        return {"kind": "ops", "n": int(round(math.exp(rng.uniform(math.log(8), math.log(200))))),
                "mode": rng.choice(["analytic", "analytic", "fd"])}
    if kind == "vcycle":
        prec = rng.choice(["fp64", "fp32"])
        return {"kind": "vcycle", "n": grid(127 if prec == "fp64" else 255), "prec": prec}
    if kind == "fp64":
        method = rng.choice(["nk", "nk", "cheb", "rec"])
        return {"kind": "nk", "n": grid(111 if method == "nk" else 79), "lam": lam, "path": "fp64", "method": method}
    if kind == "host":
        return {"kind": "host", "n": rng.choice([31, 63, 127]), "lam": lam}
    if kind == "mixed":
        return {"kind": "nk", "n": grid(223), "lam": lam, "path": "mixed", "method": "nk"}
    if kind == "jacobi":
        return {"kind": "jacobi", "n": rng.randint(12, 31), "lam": lam, "method": "nk"}
    if kind == "burgers":
        return {"kind": "burgers", "n": rng.choice([31, 47, 63, 95, 127, 191, 255]), "nu": rng.choice([0.02, 0.05, 0.08]),
                "dt": rng.choice([0.01, 0.02, 0.04]), "method": rng.choice(["nk", "cheb"])}
    if kind == "bruss":
        return {"kind": "bruss", "n": rng.choice([96, 128, 160, 256, 320, 512, 768, 1024]), "steps": rng.randint(1, 3)}
    return {"kind": "batch", "count": rng.randint(4, 32), "big": rng.choice([31, 63])}


# ------------------------------------------------------------------------------------------------ inputs
def _rng(case, seed):
    return np.random.default_rng([int(seed), int(case.get("n", case.get("count", 0)))])


def _axis(n):
    return np.arange(1, n + 1) / (n + 1.0)


def _smooth3(case, seed, scale, modes=3):
    """A sum of low sine modes with seeded amplitudes: a smooth field that is zero on the boundary."""
    n, r = case["n"], _rng(case, seed)
    s = [np.sin(math.pi * (m + 1) * _axis(n)) for m in range(modes)]
    u = np.zeros((n, n, n))
    for _ in range(4):
        a, b, c = r.integers(0, modes, 3)
        u += r.uniform(-scale, scale) * (s[a][:, None, None] * s[b][None, :, None] * s[c][None, None, :])
    return u.ravel()


def _start3(case, seed):
    """A Newton start: a positive bump of seeded height with a little of the low modes."""
    s = np.sin(math.pi * _axis(case["n"]))
    bump = s[:, None, None] * s[None, :, None] * s[None, None, :]
    return _rng(case, seed + 1).uniform(0.0, 0.3) * bump.ravel() + 0.2 * _smooth3(case, seed, 0.1)


def _rhs3(case, seed):
    """What a Krylov solver hands the preconditioner: a smooth part and a rough one, norm near 1."""
    r = _rng(case, seed).standard_normal(case["n"] ** 3)
    v = _smooth3(case, seed + 1, 1.0) + 0.3 * r
    return v / np.linalg.norm(v)


def _params(case):
    if case["kind"] in ("nk", "host"):
        p = dict(rtol_nl=1e-10, gmres_restart=30)
        if case["kind"] == "host" or case["path"] == "mixed":
            p.update(flexible=1, jvp_precision=G.FP32, orth=G.CGS1, jvp_tight=1)
        return G.default_params(**p)
    if case["kind"] == "bruss":
        return G.default_params(rtol_nl=1e-6, gmres_restart=40, gmres_max_iters=400, flexible=1, jvp_precision=G.FP32,
                                orth=G.CGS1)
    if case["kind"] == "batch":
        return G.default_params(rtol_nl=1e-10, gmres_restart=30, flexible=1, jvp_precision=G.FP32, orth=G.CGS1,
                                jvp_tight=1, coarse_jacobian=1)
    # the calibration campaign's setting t01
    return G.default_params(rtol_nl=1e-8, eta_init=0.25, gmres_restart=30, gmres_max_iters=200)


def _instances(case, seed):
    r = np.random.default_rng([int(seed), case["count"]])
    sizes = [31 if i % 3 else case["big"] for i in range(case["count"])]
    return [(n, float(lm)) for n, lm in zip(sizes, r.uniform(1.0, 6.5, case["count"]))]


def _burgers_exact(n):
    s1, s2 = np.sin(math.pi * _axis(n)), np.sin(2.0 * math.pi * _axis(n))
    return np.concatenate([np.outer(s1, s1).ravel(), np.outer(s1, s2).ravel()])


def _burgers_start(case, seed):
    """Near the rest state: the campaign starts at zero."""
    n, r = case["n"], _rng(case, seed)
    s = [np.sin(math.pi * (m + 1) * _axis(n)) for m in range(3)]
    w = [sum(r.uniform(-0.1, 0.1) * np.outer(s[a], s[b]) for a in range(3) for b in range(3)).ravel() for _ in range(2)]
    return np.concatenate(w)


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    st = {"kind": kind, "ctx": ctx}
    if kind == "batch":
        st["solver"] = G.BatchSolver(ctx, _instances(case, seed), _params(case))
        return st
    n = case["n"]
    if kind == "ops":
        st["op"] = G.Bratu3D(ctx, n, 6.0)
        st["mode"] = G.FD if case["mode"] == "fd" else G.ANALYTIC
        st["u"], st["v"] = ctx.from_numpy(_start3(case, seed)), ctx.from_numpy(_rhs3(case, seed))
        st["out"] = [ctx.vec(n ** 3) for _ in range(3)]
        st["t"] = [_tensor(o) for o in st["out"]]
    elif kind == "vcycle":
        st["mg"] = G.PoissonMG(ctx, n, precision=G.FP32 if case["prec"] == "fp32" else G.FP64)
        st["r"], st["z"] = ctx.from_numpy(_rhs3(case, seed)), ctx.vec(n ** 3)
        st["t"] = _tensor(st["z"])
    elif kind == "host":
        st.update(n=n, lam=case["lam"], p=_params(case))
        st["x0"] = torch.from_numpy(_start3(case, seed)).pin_memory().numpy()
        st["out"] = torch.empty(n ** 3, dtype=torch.float64, pin_memory=True).numpy()
    else:
        st["p"] = _params(case)
        if kind in ("nk", "jacobi"):
            op = G.Bratu3D(ctx, n, case["lam"])
            x0 = _start3(case, seed)
            if kind == "jacobi":
                pc = G.Provider.jacobi(op)
            elif case["path"] == "fp64":
                pc = G.Provider.poisson_mg(ctx, n)
            elif (n & (n + 1)) == 0:  # 2^k - 1: the Jacobian-aware hierarchy
                pc = G.Provider.jacobian_mg(ctx, n)
            else:
                pc = G.Provider.poisson_mg(ctx, n, precision=G.FP32)
        elif kind == "burgers":
            op = G.Burgers2D(ctx, n, case["nu"], case["dt"], 1.0)
            pc, x0 = G.Provider.burgers_mg(ctx, n, case["nu"], case["dt"]), _burgers_start(case, seed)
        else:
            op = G.Brusselator2D(ctx, n)
            pc, x0 = G.Provider.brusselator_mg(op, G.FP32), G.brusselator2d_initial(n, seed=int(seed))
            st["steps"] = case["steps"]
        st["method"] = case.get("method", "nk")
        st["op"], st["pc"] = op, pc
        st["x0"], st["x"] = ctx.from_numpy(x0), ctx.vec(x0.size)
        st["t"] = _tensor(st["x"])
    return st


_COUNTS = ("converged", "iters", "n_F", "n_JVP", "n_D2", "n_lin_iters", "n_prec")


def run(st):
    kind = st["kind"]
    if kind == "ops":
        op, u, v, o = st["op"], st["u"], st["v"], st["out"]
        op.eval(u, o[0])
        op.jvp(u, v, o[1], st["mode"])
        op.d2(u, v, o[2], st["mode"])
        return list(st["t"])
    if kind == "vcycle":
        st["mg"](st["r"], st["z"])
        return st["t"]
    if kind == "host":
        x, r = G.solve_bratu3d_host(st["ctx"], st["n"], st["lam"], st["x0"], st["out"], "nk", "jacobian_mg", G.FP32,
                                    st["p"])
        return {"x": x, "counts": [int(r[k]) for k in _COUNTS]}
    if kind == "batch":
        r, _, xs = st["solver"].solve(want_x=True)
        return {"x": xs, "counts": np.array([[int(q[k]) for k in ("converged", "iters", "n_F", "n_lin_iters")] for q in r])}
    st["x"].copy_from(st["x0"])
    if kind == "bruss":
        r = st["op"].advance(st["x"], st["steps"], "nk", st["p"], st["pc"])
        return {"x": st["t"], "counts": [[int(q[k]) for k in _COUNTS] for q in r]}
    r = G.solve(st["op"], st["x"], st["method"], st["p"], st["pc"])
    return {"x": st["t"], "counts": [int(r[k]) for k in _COUNTS]}


# ------------------------------------------------------------------------------------------------ least work
def work(case):
    """Inputs read once and results written once; the operations of the algorithm as the method needs them (an
    evaluation or product ~20 a point, a V(2,2) cycle ~60 a point over its levels)."""
    kind = case["kind"]
    if kind == "batch":
        N = sum(n ** 3 for n, _ in _instances(case, 0))
        return {"bytes": 8.0 * N, "flops": 9 * 80.0 * N}
    n = case["n"]
    if kind == "ops":
        return {"bytes": 8.0 * 5 * n ** 3, "flops": 50.0 * n ** 3}
    if kind == "vcycle":
        return {"bytes": 16.0 * n ** 3, "flops": 60.0 * n ** 3}
    if kind == "burgers":
        return {"bytes": 16.0 * 2 * n * n, "flops": 18 * 70.0 * 2 * n * n}
    if kind == "bruss":
        return {"bytes": 16.0 * 2 * n * n, "flops": case["steps"] * 5 * 90.0 * 2 * n * n}
    cycles = 190 if kind == "jacobi" else (24 if case.get("method") in ("cheb", "rec") else 12)
    per = 60.0 if kind == "jacobi" else 90.0
    return {"bytes": 16.0 * n ** 3, "flops": cycles * per * n ** 3}


# ------------------------------------------------------------------------------------------------ 64-bit answers
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _lap3(u, n):
    """-Lap_h u of an n^3 tensor with zero boundary values."""
    h2 = (n + 1.0) ** 2
    s = 6.0 * u
    s[1:] -= u[:-1]
    s[:-1] -= u[1:]
    s[:, 1:] -= u[:, :-1]
    s[:, :-1] -= u[:, 1:]
    s[:, :, 1:] -= u[:, :, :-1]
    s[:, :, :-1] -= u[:, :, 1:]
    return h2 * s


class _Poisson3:
    """(-Lap_h)^-1 by the sine transform, as dense products along the three axes."""

    def __init__(self, n):
        k = torch.arange(1, n + 1, dtype=torch.float64, device=_dev())
        self.S = torch.sin(math.pi * k[:, None] * k[None, :] / (n + 1)) * math.sqrt(2.0 / (n + 1))
        e = 4.0 * (n + 1.0) ** 2 * torch.sin(0.5 * math.pi * k / (n + 1)) ** 2
        self.w = 1.0 / (e[:, None, None] + e[None, :, None] + e[None, None, :])
        self.n = n

    def _t(self, u):
        n, S = self.n, self.S
        u = (u.reshape(n * n, n) @ S).reshape(n, n, n)
        u = torch.matmul(S, u)
        return (S @ u.reshape(n, n * n)).reshape(n, n, n)

    def __call__(self, u):
        return self._t(self._t(u) * self.w)


def _bratu_exact(n, lam, x0):
    """The discrete solution on the branch of the start: Newton with conjugate gradients preconditioned by the exact
    Laplacian inverse (the Jacobian is positive definite there)."""
    P, u = _Poisson3(n), torch.from_numpy(np.array(x0)).to(_dev()).reshape(n, n, n)
    res0 = None
    for _ in range(12):
        c = lam * torch.exp(u)
        F = _lap3(u, n) - c
        z = torch.zeros_like(u)
        r, y = F.clone(), P(F)
        p, rho = y.clone(), float((r * y).sum())
        rho0 = rho
        res0 = res0 or rho
        if rho <= 1e-26 * res0:
            break
        for _ in range(60):
            q = _lap3(p, n) - c * p
            a = rho / float((p * q).sum())
            z += a * p
            r -= a * q
            y = P(r)
            new = float((r * y).sum())
            if new <= 1e-20 * rho0:
                break
            p = y + (new / rho) * p
            rho = new
        u = u - z
    return u.reshape(-1)


def _vcycle64(n, r):
    """One V(2,2) of the full hierarchy in FP64: red-black Gauss-Seidel, full weighting, trilinear interpolation."""
    i = torch.arange(n, device=_dev())
    colour = (i[:, None, None] + i[None, :, None] + i[None, None, :]) % 2
    masks = [colour == 0, colour == 1]
    b = r.reshape(n, n, n)

    def sweep(x, b, n, order):
        h2 = (n + 1.0) ** 2
        for c in (order, 1 - order):
            m = masks_of[n][c]
            x = torch.where(m, x + (b - _lap3(x, n)) / (6.0 * h2), x)
        return x

    def interp(nc, nf):
        W = torch.zeros(nf, nc, dtype=torch.float64, device=_dev())
        for k in range(nc):
            W[2 * k + 1, k] = 1.0
            W[2 * k, k] = 0.5
            if 2 * k + 2 < nf:
                W[2 * k + 2, k] = 0.5
        return W

    def along(W, u):
        u = torch.einsum("ai,ijk->ajk", W, u)
        u = torch.einsum("bj,ajk->abk", W, u)
        return torch.einsum("ck,abk->abc", W, u)

    masks_of = {n: masks}

    def cycle(b, n):
        if n not in masks_of:
            i = torch.arange(n, device=_dev())
            col = (i[:, None, None] + i[None, :, None] + i[None, None, :]) % 2
            masks_of[n] = [col == 0, col == 1]
        if n == 1:
            return b / 24.0
        x = torch.zeros_like(b)
        if n % 2 == 0:
            for s in range(30):
                x = sweep(x, b, n, s % 2)
            return x
        for _ in range(2):
            x = sweep(x, b, n, 0)
        nc = (n - 1) // 2
        W = interp(nc, n)
        x = x + along(W, cycle(along(0.5 * W.T, b - _lap3(x, n)), nc))
        for _ in range(2):
            x = sweep(x, b, n, 1)
        return x

    return cycle(b, n).reshape(-1)


def _bruss_exact(case, seed):
    """Each implicit step by a fixed point on the Fourier inverse of the Jacobian at the mean state."""
    n, q = case["n"], G.brusselator_params()
    w = torch.from_numpy(G.brusselator2d_initial(n, seed=int(seed))).to(_dev()).reshape(2, n, n)
    h2 = float(n) * n
    k = 4.0 * h2 * torch.sin(math.pi * torch.arange(n, dtype=torch.float64, device=_dev()) / n) ** 2
    eig = k[:, None] + k[None, : n // 2 + 1]

    def lap(a):
        return h2 * ((torch.roll(a, 1, 0) - a) + (torch.roll(a, -1, 0) - a) + (torch.roll(a, 1, 1) - a) +
                     (torch.roll(a, -1, 1) - a))

    for _ in range(case["steps"]):
        prev = w.clone()
        for _ in range(14):
            u, v = w[0], w[1]
            uuv = u * u * v
            Fu = (u - prev[0]) / q.dt - q.Du * lap(u) - (q.A + uuv - (q.B + 1.0) * u)
            Fv = (v - prev[1]) / q.dt - q.Dv * lap(v) - (q.B * u - uuv)
            uv, uu = float((u * v).mean()), float((u * u).mean())
            k11, k12 = 1.0 / q.dt + q.B + 1.0 - 2.0 * uv + q.Du * eig, -uu
            k21, k22 = 2.0 * uv - q.B, 1.0 / q.dt + uu + q.Dv * eig
            det = k11 * k22 - k12 * k21
            a, b = torch.fft.rfft2(Fu), torch.fft.rfft2(Fv)
            w = torch.stack([u - torch.fft.irfft2((k22 * a - k12 * b) / det, s=(n, n)),
                             v - torch.fft.irfft2((k11 * b - k21 * a) / det, s=(n, n))])
    return w.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"x": [_bratu_exact(n, lm, np.zeros(n ** 3)) for n, lm in _instances(case, seed)], "counts": None}
    n = case["n"]
    if kind == "ops":
        u, v = (torch.from_numpy(f(case, seed)).to(_dev()).reshape(n, n, n) for f in (_start3, _rhs3))
        c = 6.0 * torch.exp(u)
        F, J, D = _lap3(u, n) - c, _lap3(v, n) - c * v, -c * v * v
        if case["mode"] == "fd":  # the quotients have no value but their own
            return [F.reshape(-1), None, None]
        return [t.reshape(-1) for t in (F, J, D)]
    if kind == "vcycle":
        return _vcycle64(n, torch.from_numpy(_rhs3(case, seed)).to(_dev()))
    counts = [None] * len(_COUNTS)
    if kind == "burgers":
        return {"x": _burgers_exact(n), "counts": counts}
    if kind == "bruss":
        return {"x": _bruss_exact(case, seed), "counts": [counts] * case["steps"]}
    return {"x": _bratu_exact(n, case["lam"], _start3(case, seed)), "counts": counts}
