"""Performance cases of the GB300 ADI framework: what a user's program asks of it.

Six kinds of work, each through the package's public classes:

* ``single``  -- one 2-D Heston problem, ``ImplicitHestonSolver.solve`` (host surface and value);
* ``adjoint`` -- value, dV/d(kappa, theta, sigma, rho, r) and dV/d(payoff) of one problem;
* ``batch``   -- many uneven Heston calls advanced together (values and status);
* ``grads``   -- the same with the adjoint (values, the five sensitivities of every instance);
* ``heat1d``  -- a batch of uneven 1-D Black-Scholes calls.

Model parameters are drawn from the seed inside the region where the splitting schemes are
stable (no growing modes): a priced surface is bounded by S_max there, as a user wants it.
"""
import math
import random

import numpy as np
import torch

import linear_system_solvers_gb300 as lss
from linear_system_solvers_gb300 import heat1d

# grid sizes of the batches: the ones that the package's own batch generator draws, and odd ones
NXS = (64, 77, 96, 128, 161, 192, 256)
NYS = (32, 45, 48, 64, 96, 101, 128)
NS_1D = (101, 128, 200, 256, 333, 384, 512)


def listed():
    return [
        # one Heston call on the plain 100 x 50 grid, as the reference's own tests price it: the
        # smallest call, where latency and launches count.  The plain call, without graph replay.
        dict(name="dr_100x50_call", kind="single", scheme="dr", nx=100, ny=50, steps=200, precision="f64",
             arith="fast", graph=False, nonuniform=False),
        # the same problem in the arithmetic that is bit-identical to the reference's host solver
        # (what the C++ drop-in runs)
        dict(name="dr_100x50_bitwise", kind="single", scheme="dr", nx=100, ny=50, steps=200, precision="f64",
             arith="reference", graph=True, nonuniform=False),
        # a fine sinh grid with the Hundsdorfer-Verwer scheme: one ordinary accurate price
        dict(name="hv_400x200", kind="single", scheme="hv", nx=400, ny=200, steps=500, precision="f64",
             arith="fast", graph=True, nonuniform=True),
        # the same class of problem in FP32 on an odd grid
        dict(name="mcs_301x151_f32", kind="single", scheme="mcs", nx=301, ny=151, steps=300, precision="f32",
             arith="fast", graph=True, nonuniform=True),
        # the largest single grid: larger than the L2 cache
        dict(name="hv_4096x2048", kind="single", scheme="hv", nx=4096, ny=2048, steps=40, precision="f64",
             arith="fast", graph=True, nonuniform=True),
        # price and sensitivities of one call (calibration step)
        dict(name="adjoint_mcs_128x64", kind="adjoint", model="heston", scheme="mcs", nx=128, ny=64, steps=200,
             rate=0.02),
        # SABR with a rate: coefficients that change with time, forward and adjoint
        dict(name="adjoint_sabr_512x256", kind="adjoint", model="sabr", scheme="dr", nx=512, ny=256, steps=100,
             rate=0.03),
        # a book of uneven calls, prices only
        dict(name="batch_mcs_1024", kind="batch", scheme="mcs", count=1024, steps_lo=100, steps_hi=400,
             precision="f64"),
        dict(name="batch_dr_768_f32", kind="batch", scheme="dr", count=768, steps_lo=100, steps_hi=400,
             precision="f32"),
        # a book of uneven calls with every sensitivity (the package's headline work)
        dict(name="grads_mcs_768", kind="grads", scheme="mcs", count=768, steps_lo=50, steps_hi=200,
             precision="f64"),
        # 1-D Black-Scholes books, both precisions
        dict(name="bs1d_4096", kind="heat1d", count=4096, nt_lo=100, nt_hi=1000, precision="f64"),
        dict(name="bs1d_8192_f32", kind="heat1d", count=8192, nt_lo=100, nt_hi=1000, precision="f32"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["single", "single", "adjoint", "batch", "grads", "heat1d"])
    if kind == "single":
        nx = _log_int(rng, 48, 2048)
        ny = _log_int(rng, max(24, nx // 4), min(1024, nx))
        arith = "reference" if nx * ny < 60000 and rng.random() < 0.25 else "fast"
        steps = min(_log_int(rng, 20, 500), max(10, int(3.0e8 / (nx * ny))))
        if arith == "reference":
            steps = min(steps, 200)
        return dict(kind=kind, scheme=rng.choice(["dr", "mcs", "hv"]), nx=nx, ny=ny, steps=steps,
                    precision="f64" if arith == "reference" else rng.choice(["f64", "f64", "f32"]), arith=arith,
                    graph=rng.random() < 0.7, nonuniform=rng.random() < 0.7)
    if kind == "adjoint":
        model = rng.choice(["heston", "sabr"])
        nx = _log_int(rng, 48, 512)
        ny = _log_int(rng, max(24, nx // 4), min(256, nx))
        return dict(kind=kind, model=model, scheme="dr" if model == "sabr" else rng.choice(["dr", "mcs", "hv"]), nx=nx,
                    ny=ny, steps=min(_log_int(rng, 20, 200), max(10, int(1.3e7 / (nx * ny)))),
                    rate=rng.choice([0.0, 0.03]) if model == "sabr" else 0.02)
    if kind in ("batch", "grads"):
        lo = rng.randint(20, 100)
        return dict(kind=kind, scheme=rng.choice(["dr", "mcs", "hv"]), count=_log_int(rng, 24, 768), steps_lo=lo,
                    steps_hi=rng.randint(lo, 400 if kind == "batch" else 200),
                    precision=rng.choice(["f64", "f32"]) if kind == "batch" else "f64")
    lo = rng.randint(50, 200)
    return dict(kind=kind, count=_log_int(rng, 48, 4096), nt_lo=lo, nt_hi=rng.randint(lo, 1000),
                precision=rng.choice(["f64", "f32"]))


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _heston(r, nx, ny, steps, scheme, nonuniform=True, precision="f64", rate=None):
    strike = r.uniform(85.0, 115.0)
    # the reference's Craig-Sneyd variants grow for strongly negative correlation on fine grids
    rho_lo = {"dr": -0.9, "hv": -0.7}.get(scheme, -0.25)
    kappa, theta_v = r.uniform(0.8, 4.0), r.uniform(0.02, 0.09)
    # the v = 0 line is advanced explicitly: its Courant number stays below the scheme's limit
    slope = 1.2 / 24.0 * math.asinh(24.0) if nonuniform else 1.2 * math.asinh(1.0)
    longest = 0.25 * 2.0 * slope * steps / (kappa * theta_v * (ny - 1))
    kw = dict(kappa=kappa, theta_v=theta_v, sigma=r.uniform(0.15, 0.5), rho=r.uniform(rho_lo, 0.0),
              rate=r.uniform(0.005, 0.05) if rate is None else rate, maturity=min(r.uniform(0.4, 1.5), longest),
              strike=strike, nx=nx, ny=ny, nt=steps + 1, scheme=scheme, eval_s=100.0, eval_v=0.04,
              fp64_tables=precision == "f32")
    if nonuniform:
        kw.update(nonuniform=True, acc_point=strike, alpha_scale=10.0, beta_scale=24.0)
    return lss.HestonProblem(**kw)


def _problems(case, seed):
    """The problem, or the list of problems, of a 2-D case."""
    r = random.Random("adi %d" % seed)
    if case["kind"] == "single":
        return _heston(r, case["nx"], case["ny"], case["steps"], case["scheme"], case["nonuniform"], case["precision"])
    if case["kind"] == "adjoint":
        if case["model"] == "sabr":
            return lss.HestonProblem(model="sabr", sabr_beta=0.5, sigma=r.uniform(0.25, 0.45), rho=r.uniform(-0.4, 0.2),
                                     rate=case["rate"], strike=r.uniform(0.045, 0.055), maturity=1.0, s_lo=0.0, s_hi=0.2,
                                     v_lo=0.0, v_hi=1.0, nx=case["nx"], ny=case["ny"], nt=case["steps"] + 1,
                                     scheme=case["scheme"], nonuniform=True, acc_point=0.05, alpha_scale=3.0,
                                     beta_scale=5.0, eval_s=0.05, eval_v=0.3)
        return _heston(r, case["nx"], case["ny"], case["steps"], case["scheme"], rate=case["rate"])
    # the sizes of a book belong to the case, the market data to the seed
    z = random.Random("sizes %d" % case["count"])
    return [_heston(r, z.choice(NXS), z.choice(NYS), z.randint(case["steps_lo"], case["steps_hi"]), case["scheme"],
                    precision=case["precision"]) for _ in range(case["count"])]


def _bs_problems(case, seed):
    r, z = random.Random("bs %d" % seed), random.Random("sizes %d" % case["count"])
    out = []
    for _ in range(case["count"]):
        strike = r.uniform(80.0, 120.0)
        out.append(heat1d.BlackScholesProblem(sigma=r.uniform(0.1, 0.6), rate=r.uniform(0.0, 0.1),
                                              maturity=r.uniform(0.25, 2.0), strike=strike, put=r.random() < 0.3,
                                              s_lo=0.0, s_hi=4.0 * strike, n=z.choice(NS_1D),
                                              nt=z.randint(case["nt_lo"], case["nt_hi"]),
                                              theta_scheme="cn" if r.random() < 0.8 else "euler", nonuniform=True,
                                              acc_point=strike, alpha_scale=3.0, eval_s=strike))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "heat1d":
        return dict(case=case, b=heat1d.black_scholes_batch(_bs_problems(case, seed), precision=case["precision"]))
    ps = _problems(case, seed)
    if kind == "single":
        s = lss.ImplicitHestonSolver(ps, precision=case["precision"], arith=case["arith"])
        x, _ = s.grid()
        pay = np.repeat(np.maximum(x - ps.strike, 0.0).astype(s.dtype)[:, None], ps.ny, axis=1)
        return dict(case=case, s=s, payoff=pay)
    if kind == "adjoint":
        return dict(case=case, s=lss.ImplicitHestonSolver(ps))
    b = lss.BatchSolver(ps, precision=case["precision"])
    if kind == "grads":
        b.set_workspace(3.0e10)
    return dict(case=case, b=b)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "single":
        surface, value = state["s"].solve(state["payoff"], graph=case["graph"])
        return {"surface": surface, "value": value}
    if kind == "adjoint":
        value, grads, dpay = state["s"].adjoint()
        return {"value": value, "grads": grads, "payoff_gradient": dpay}
    b = state["b"]
    if kind == "heat1d":
        b.run()
        values, status = b.results()
        return {"values": values, "status": status, "solution": b.solution(0)}
    b.run(1 if kind == "grads" else 0, graph=True)
    values, grads, status = b.results()
    out = {"values": values, "status": status, "surface": b.surface(0)}
    if kind == "grads":
        out.update(grads=grads, payoff_gradient=b.payoff_gradient(0))
    return out


# ------------------------------------------------------------------------------------------------
# unavoidable work of one pass
# ------------------------------------------------------------------------------------------------
# Floating-point operations of one grid point and one step: the right-hand sides and one
# multiply-add each way (and one scaling) per line solve; the adjoint transposes them and sums the
# parameter sensitivities.
FWD = {"dr": 26, "cs": 44, "mcs": 44, "hv": 58}
ADJ = {"dr": 62, "cs": 102, "mcs": 102, "hv": 122}


def work(case):
    kind = case["kind"]
    w = 4 if case.get("precision") == "f32" else 8
    if kind == "heat1d":
        ps = _bs_problems(case, 1)
        return {"bytes": float(w * 2 * sum(p.n for p in ps)), "flops": float(6 * sum(p.n * (p.nt - 1) for p in ps))}
    ps = _problems(case, 1)
    ps = ps if isinstance(ps, list) else [ps]
    n = sum(p.nx * p.ny for p in ps)
    gps = sum(p.nx * p.ny * p.steps for p in ps)
    per = FWD[case["scheme"]] + (ADJ[case["scheme"]] if kind in ("adjoint", "grads") else 0)
    return {"bytes": float(w * 2 * n), "flops": float(per * gps)}


# ------------------------------------------------------------------------------------------------
# the same results in plain torch, FP64: dense inverses of the line matrices, autograd for the adjoint
# ------------------------------------------------------------------------------------------------
class _LineSolve(torch.autograd.Function):
    """x of tridiagonal systems (..., e) given their dense inverse; the adjoint is the transposed solve."""

    @staticmethod
    def forward(ctx, inv, lo, dg, up, f):
        x = torch.matmul(inv, f.unsqueeze(-1)).squeeze(-1)
        ctx.save_for_backward(inv, x)
        ctx.need = lo.requires_grad
        return x

    @staticmethod
    def backward(ctx, xb):
        inv, x = ctx.saved_tensors
        g = torch.matmul(inv.transpose(-1, -2), xb.unsqueeze(-1)).squeeze(-1)
        if not ctx.need:
            return None, None, None, None, g
        z = torch.zeros_like(x[..., :1])
        dlo = -g * torch.cat([z, x[..., :-1]], -1)
        dup = -g * torch.cat([x[..., 1:], z], -1)
        return None, dlo, -g * x, dup, g


def _inverse(lo, dg, up):
    a = torch.diag_embed(dg) + torch.diag_embed(lo[..., 1:], -1) + torch.diag_embed(up[..., :-1], 1)
    return torch.linalg.inv(a.detach())


class _Same2d:
    """Problems of one size, scheme and model advanced together."""

    def __init__(self, ps, dev, params=None):
        p0 = ps[0]
        self.ps, self.dev, self.nx, self.ny, self.scheme = ps, dev, p0.nx, p0.ny, p0.scheme
        self.sabr = p0.model == "sabr"
        t = lambda f: torch.tensor([f(p) for p in ps], dtype=torch.float64, device=dev)  # noqa: E731
        self.par = params if params is not None else [t(lambda p, n=n: getattr(p, n)) for n in
                                                      ("kappa", "theta_v", "sigma", "rho", "rate")]
        self.steps = torch.tensor([p.steps for p in ps], device=dev)
        nx, ny = p0.nx, p0.ny
        k = t(lambda p: p.maturity / p.steps)
        h1, h2 = 1.0 / (nx - 1), 1.0 / (ny - 1)
        self.k, self.h1, self.h2 = k, h1, h2
        self.al, self.be, self.ga, self.de, self.ni = k / (h1 * h1), k / (h2 * h2), 0.25 * k / (h1 * h2), 0.5 * k / h1, 0.5 * k / h2
        self.th, self.ze = 0.5, p0.zeta
        z = torch.arange(nx, dtype=torch.float64, device=dev) * h1
        e = torch.arange(ny, dtype=torch.float64, device=dev) * h2
        pt = t(lambda p: p.acc_point)
        slo, shi, vlo, vhi = t(lambda p: p.s_lo), t(lambda p: p.s_hi), t(lambda p: p.v_lo), t(lambda p: p.v_hi)
        a = t(lambda p: (p.acc_point - p.s_lo) / p.alpha_scale if p.nonuniform else p.s_hi - p.s_lo)
        b = t(lambda p: (p.v_hi - p.v_lo) / p.beta_scale if p.nonuniform else p.v_hi - p.v_lo)
        c0, c1, d = torch.asinh((shi - pt) / a), torch.asinh((slo - pt) / a), torch.asinh((vhi - vlo) / b)
        arg = c0[:, None] * z + c1[:, None] * (1.0 - z)
        cd = (c0 - c1)[:, None]
        self.x = pt[:, None] + a[:, None] * torch.sinh(arg)
        self.A, self.A2 = a[:, None] * cd * torch.cosh(arg), a[:, None] * cd * cd * torch.sinh(arg)
        dd = d[:, None]
        self.y = vlo[:, None] + b[:, None] * torch.sinh(dd * e)
        self.B, self.B2 = b[:, None] * dd * torch.cosh(dd * e), b[:, None] * dd * dd * torch.sinh(dd * e)
        self.neu = t(lambda p: p.neumann_value)[:, None] * self.A[:, -1:]
        # the neighbour line that a truncating index_of((h i) / h) picks
        self.im = torch.tensor([int((h1 * i) / h1) for i in range(nx)], device=dev)
        self.jm = torch.tensor([int((h2 * j) / h2) for j in range(ny)], device=dev)
        self.tdep = self.sabr and any(p.rate != 0.0 for p in ps)
        self.T = t(lambda p: p.maturity)
        if not self.tdep:
            self.tables(self.T - k)

    def tables(self, time):
        ka, tv, sg, rh, rt = [q[:, None, None] for q in self.par]
        x, y, A, B, A2, B2 = self.x[:, :, None], self.y[:, None, :], self.A[:, :, None], self.B[:, None, :], self.A2[:, :, None], self.B2[:, None, :]
        if self.sabr:
            bt = self.ps[0].sabr_beta
            D = torch.exp(-rt * (self.T - time)[:, None, None])
            a = 0.5 * y * y * x ** (2 * bt) * D ** (2 * (1 - bt))
            b, c, e = 0.5 * sg * sg * y * y, rh * sg * y * y * x ** bt * D ** (1 - bt), 0.0 * ka
        else:
            a, b, c, e = 0.5 * y * x * x, 0.5 * sg * sg * y, rh * sg * y * x, ka * (tv - y)
        ah, bh, ch = a / (A * A), b / (B * B), c / (A * B)
        dh, eh, fh = rt * x / A - a * A2 / A ** 3, e / B - b * B2 / B ** 3, -rt
        q = lambda v: v[:, None, None]  # noqa: E731
        full = torch.zeros((len(self.ps), self.nx, self.ny), dtype=torch.float64, device=self.dev)
        self.M, self.P = q(self.al) * ah - q(self.de) * dh + full, q(self.al) * ah + q(self.de) * dh + full
        self.Z = 2 * q(self.al) * ah - 0.5 * q(self.k) * fh + full
        self.Mt, self.Pt = q(self.be) * bh - q(self.ni) * eh + full, q(self.be) * bh + q(self.ni) * eh + full
        self.W = 2 * q(self.be) * bh - 0.5 * q(self.k) * fh + full
        self.gC = q(self.ga) * ch + full
        self.D0, self.E0, self.F0 = (dh + full)[:, :, 0], (eh + full)[:, :, 0], (fh + full)[:, :, 0]
        tr = lambda v: v[:, 1:-1, 1:-1].transpose(1, 2)  # noqa: E731
        th = self.th
        self.sl = [tr(-th * self.M), tr(1 + th * self.Z), tr(-th * self.P)]
        self.sinv = _inverse(*self.sl)
        if not hasattr(self, "vinv"):
            iv = lambda v: v[:, 1:-1, 1:-1]  # noqa: E731
            self.vl = [iv(-th * self.Mt), iv(1 + th * self.W), iv(-th * self.Pt)]
            self.vinv = _inverse(*self.vl)

    def s_solve(self, f, lo, hi):
        """f: (B, nx-2, ny-2); lo, hi: (B, ny-2) values on rows 0 and nx-1; returns the interior."""
        f = f.transpose(1, 2)
        f = torch.cat([f[..., :1] - (self.sl[0][..., :1] * lo[..., None]), f[..., 1:-1],
                       f[..., -1:] - (self.sl[2][..., -1:] * hi[..., None])], -1)
        return _LineSolve.apply(self.sinv, *self.sl, f).transpose(1, 2)

    def v_solve(self, f, lo, hi):
        f = torch.cat([f[..., :1] - (self.vl[0][..., :1] * lo[..., None]), f[..., 1:-1],
                       f[..., -1:] - (self.vl[2][..., -1:] * hi[..., None])], -1)
        return _LineSolve.apply(self.vinv, *self.vl, f)

    def step(self, U):
        i = lambda v: v[:, 1:-1, 1:-1]  # noqa: E731
        mix = lambda v: v[:, :-2, :-2] - v[:, :-2, 2:] - v[:, 2:, :-2] + v[:, 2:, 2:]  # noqa: E731
        w, e, s, n = (lambda v: v[:, :-2, 1:-1]), (lambda v: v[:, 2:, 1:-1]), (lambda v: v[:, 1:-1, :-2]), (lambda v: v[:, 1:-1, 2:])
        M, P, Z, Mt, Pt, W, gC = [i(v) for v in (self.M, self.P, self.Z, self.Mt, self.Pt, self.W, self.gC)]
        th, ze = self.th, self.ze
        ni, de, k = self.ni[:, None], self.de[:, None], self.k[:, None]
        # the explicit v = v_lo column and the v_hi column
        c0, c1, c2 = U[:, :, 0], U[:, :, 1], U[:, :, 2]
        ctr = (1 - 3 * ni * self.E0 + k * self.F0) * c0 + 4 * ni * self.E0 * c1 - ni * self.E0 * c2
        mid = ctr[:, 1:-1] + (de * self.D0)[:, 1:-1] * (c0[:, 2:] - c0[:, :-2])
        top = ctr[:, -1:] - de * 2 * self.h1 * self.neu * self.D0[:, -1:]
        b0 = torch.cat([torch.zeros_like(top), mid, top], 1)
        vlo, vhi = b0[:, self.im[1:-1]], self.x[:, self.im[1:-1]]
        jm = self.jm[1:-1]
        slo, shi = U[:, 0, jm], U[:, -1, jm]

        def frame(inner, row0, row1, col0, col1):
            v = torch.cat([col0[:, :, None], inner, col1[:, :, None]], 2)
            return torch.cat([row0[:, None], v, row1[:, None]], 1)

        def v_rhs(a):
            return -th * (Mt * s(a) - W * i(a) + Pt * n(a))

        f1 = gC * mix(U) + (1 - th) * (M * w(U) - Z * i(U) + P * e(U)) + Mt * s(U) + (1 - W) * i(U) + Pt * n(U)
        y1 = self.s_solve(f1, slo, shi)
        if self.scheme == "dr":
            v = self.v_solve(v_rhs(U) + y1, vlo, vhi)
        else:
            zr = torch.zeros_like(U[:, 0])
            y2 = frame(self.v_solve(v_rhs(U) + y1, vlo, vhi), zr, zr, vlo, vhi)
            d = y2 - U
            if self.scheme == "hv":
                y1f = torch.cat([slo[:, None], y1, shi[:, None]], 1)
                f = y1 - th * (M * y1f[:, :-2] - Z * y1 + P * y1f[:, 2:]) - th * (M * w(d) - Z * i(d) + P * e(d))
                f = f + ze * (gC * mix(d) + M * w(d) - (W + Z) * i(d) + P * e(d) + Mt * s(d) + Pt * n(d))
                y3 = self.s_solve(f, slo, shi)
                v = self.v_solve(v_rhs(y2) + y3, vlo, vhi)
            else:
                f = -th * (M * w(U) - Z * i(U) + P * e(U)) + y1 + ze * gC * mix(d)
                if self.scheme == "mcs" and ze != th:
                    f = f + (ze - th) * (M * w(d) - (Z + W) * i(d) - P * e(d) + Mt * s(d) + Pt * n(d))
                y3 = self.s_solve(f, slo, shi)
                v = self.v_solve(v_rhs(U) + y3, vlo, vhi)
        v = torch.cat([vlo[:, :, None], v, vhi[:, :, None]], 2)
        last = (4 * v[:, -1][:, self.jm] - v[:, -2][:, self.jm] - 2 * self.h1 * self.neu) / 3
        return torch.cat([torch.zeros_like(last)[:, None], v, last[:, None]], 1)

    def solve(self, U):
        time = self.T - self.k
        for m in range(int(self.steps.max())):
            if self.tdep:
                self.tables(time)
                time = time - self.k
            new = self.step(U)
            done = (self.steps <= m)[:, None, None]
            U = torch.where(done, U, new) if bool(done.any()) else new
        return U

    def payoff(self):
        K = torch.tensor([p.strike for p in self.ps], dtype=torch.float64, device=self.dev)
        return torch.clamp(self.x - K[:, None], min=0.0)[:, :, None].expand(-1, -1, self.ny).contiguous()

    def values(self, U):
        out = []
        for q, p in enumerate(self.ps):
            x, y = self.x[q].tolist(), self.y[q].tolist()

            def cell(g, at):
                i0 = 0
                while i0 + 2 < len(g) and g[i0 + 1] <= at:
                    i0 += 1
                return i0, min(1.0, max(0.0, (at - g[i0]) / (g[i0 + 1] - g[i0])))

            (a, s), (b, v) = cell(x, p.eval_s), cell(y, p.eval_v)
            out.append((1 - s) * (1 - v) * U[q, a, b] + s * (1 - v) * U[q, a + 1, b] + (1 - s) * v * U[q, a, b + 1] +
                       s * v * U[q, a + 1, b + 1])
        return torch.stack(out)


PARAMS = ("kappa", "theta_v", "sigma", "rho", "rate")


def _with_grads(ps, dev):
    """values, grads (B, 5), dV/d(payoff) and final surfaces of problems of one size."""
    par = [torch.tensor([getattr(p, n) for p in ps], dtype=torch.float64, device=dev, requires_grad=True) for n in PARAMS]
    s = _Same2d(ps, dev, par)
    pay = s.payoff().requires_grad_(True)
    U = s.solve(pay)
    val = s.values(U)
    g = torch.autograd.grad(val.sum(), par + [pay], allow_unused=True)
    zero = torch.zeros_like(par[0])
    return val.detach(), torch.stack([zero if q is None else q for q in g[:5]], 1), g[5], U.detach()


def _cost(p):
    return p.steps * p.nx * p.ny * (p.nx + p.ny)


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    kind = case["kind"]
    if kind == "heat1d":
        return _exact_1d(case, seed, dev)
    ps = _problems(case, seed)
    if kind == "single":
        if _cost(ps) > 3.0e10 or ps.nx * ps.ny * (ps.nx + ps.ny) > 4.0e8:
            return None
        s = _Same2d([ps], dev)
        U = s.solve(s.payoff())
        return {"surface": U[0].cpu().numpy(), "value": float(s.values(U)[0])}
    if kind == "adjoint":
        if ps.model == "sabr" and ps.rate != 0.0 and ps.nx * ps.ny > 20000 or _cost(ps) > 1.0e10:
            return None
        val, g, dp, _ = _with_grads([ps], dev)
        return {"value": float(val[0]), "grads": g[0].cpu().numpy(), "payoff_gradient": dp[0].cpu().numpy()}
    grads = kind == "grads"
    if sum(_cost(p) for p in ps) > (1.2e12 if grads else 2.0e12):
        return None
    values = np.empty(len(ps))
    gr = np.empty((len(ps), 5))
    surface = dpay = None
    groups = {}
    for q, p in enumerate(ps):
        groups.setdefault((p.nx, p.ny), []).append(q)
    for (nx, ny), idx in groups.items():
        # autograd keeps about 40 grids per step
        most = max(1, int(6.0e10 / (320.0 * nx * ny * max(ps[q].steps for q in idx)))) if grads else 64
        idx.sort(key=lambda q: ps[q].steps)
        for a in range(0, len(idx), most):
            part = idx[a:a + most]
            sub = [ps[q] for q in part]
            if grads:
                val, g, dp, U = _with_grads(sub, dev)
                gr[part] = g.cpu().numpy()
            else:
                s = _Same2d(sub, dev)
                U = s.solve(s.payoff())
                val = s.values(U)
            values[part] = val.cpu().numpy()
            if 0 in part:
                surface = U[part.index(0)].cpu().numpy()
                if grads:
                    dpay = dp[part.index(0)].cpu().numpy()
    out = {"values": values, "status": None, "surface": surface}
    if grads:
        out.update(grads=gr, payoff_gradient=dpay)
    return out


def _exact_1d(case, seed, dev):
    ps = _bs_problems(case, seed)
    values, solution = np.empty(len(ps)), None
    groups = {}
    for q, p in enumerate(ps):
        groups.setdefault(p.n, []).append(q)
    for n, idx in groups.items():
        idx.sort(key=lambda q: -ps[q].nt)
        sub = [ps[q] for q in idx]
        t = lambda f: torch.tensor([f(p) for p in sub], dtype=torch.float64, device=dev)  # noqa: E731
        h = 1.0 / (n - 1)
        k, strike, rate, T = t(lambda p: p.maturity / (p.nt - 1)), t(lambda p: p.strike), t(lambda p: p.rate), t(lambda p: p.maturity)
        sig, th, put = t(lambda p: p.sigma), t(lambda p: 1.0 if p.theta_scheme == "euler" else 0.5), t(lambda p: float(p.put))
        z = torch.arange(n, dtype=torch.float64, device=dev) * h
        slo, shi, pt = t(lambda p: p.s_lo), t(lambda p: p.s_hi), t(lambda p: p.acc_point)
        al = t(lambda p: (p.acc_point - p.s_lo) / p.alpha_scale)
        c0, c1 = torch.asinh((shi - pt) / al), torch.asinh((slo - pt) / al)
        arg, cd = c0[:, None] * z + c1[:, None] * (1 - z), (c0 - c1)[:, None]
        x = pt[:, None] + al[:, None] * torch.sinh(arg)
        A, A2 = al[:, None] * cd * torch.cosh(arg), al[:, None] * cd * cd * torch.sinh(arg)
        ua, ub, uc = 0.5 * sig[:, None] ** 2 * x * x, rate[:, None] * x, -rate[:, None]
        lam, gam, dlt = (k / (h * h))[:, None], (k / (2 * h))[:, None], (0.5 * k)[:, None]
        ta, tb = ua / (A * A), ub / A - ua * A2 / A ** 3
        cA, cB, cD = lam * ta - gam * tb, lam * ta - dlt * uc, lam * ta + gam * tb
        th_ = th[:, None]
        lo, dg, up = [v[:, 1:-1] for v in (-th_ * cA, 1 + 2 * th_ * cB, -th_ * cD)]
        inv = _inverse(lo, dg, up)
        sgn = (1 - 2 * put)[:, None]
        U = torch.clamp(sgn * (x - strike[:, None]), min=0.0)
        time = T - k
        steps = torch.tensor([p.nt - 1 for p in sub], device=dev)
        host = steps.tolist()
        live = len(sub)
        for m in range(host[0]):
            while live and host[live - 1] <= m:
                live -= 1
            c = slice(0, live)
            disc = strike[c] * torch.exp(-rate[c] * (T[c] - time[c]))
            lv, hv = put[c] * disc, (1 - put[c]) * (shi[c] - disc)
            u, om = U[c], (1 - th_)[c]
            f = om * cA[c, 1:-1] * u[:, :-2] + (1 - 2 * om * cB[c, 1:-1]) * u[:, 1:-1] + om * cD[c, 1:-1] * u[:, 2:]
            f = torch.cat([f[:, :1] - lo[c, :1] * lv[:, None], f[:, 1:-1], f[:, -1:] - up[c, -1:] * hv[:, None]], 1)
            v = torch.matmul(inv[c], f[:, :, None]).squeeze(-1)
            U[c] = torch.cat([lv[:, None], v, hv[:, None]], 1)
            time = time - k
        X, S = x.cpu().numpy(), U.cpu().numpy()
        for r, q in enumerate(idx):
            p = ps[q]
            i0 = int(np.searchsorted(X[r, 1:-1], p.eval_s, side="right"))
            w = min(1.0, max(0.0, (p.eval_s - X[r, i0]) / (X[r, i0 + 1] - X[r, i0])))
            values[q] = (1 - w) * S[r, i0] + w * S[r, i0 + 1]
            if q == 0:
                solution = S[r].copy()
    return {"values": values, "status": None, "solution": solution}
