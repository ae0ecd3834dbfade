"""The work this framework is timed on: whole simulations through the public calls.

A case is one use of the library as a program makes it: a simulation run from
its initial field for some steps and read back (Solver), a group of
simulations admitted into a batch, stepped together and read back (Batch), or
single steps on a host array (the drop-in for a solver that keeps its state on
the host).  Sizes, degrees and initial fields are those of the four named
workloads and of the seeded request mix (aderdg/workloads.py): degrees 2 to 5,
sides 32 to 512, every initial-field parameter jittered by 10%; 20 steps a
request, as bench.py serves them, fewer where a step is long.

exact() restates the scheme in plain torch FP64 over all cells at once.
"""
import dataclasses
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ader-dg_gb300"))
import aderdg  # noqa: E402
from aderdg import workloads  # noqa: E402

PRECISION = {"fp64": aderdg.FP64, "fp32_mixed": aderdg.FP32_MIXED, "fp32_wide": aderdg.FP32_WIDE}


def case(name, call, workload, N, imax, jmax, precision, steps, count=1):
    return dict(name=name, call=call, workload=workload, N=N, imax=imax, jmax=jmax, precision=precision, steps=steps,
                count=count)


def listed():
    return [
        # the smallest call: scalar transport on a 64 x 64 grid, every step a handful of tiny launches
        case("ad_sine_64_n3_mixed", "run", "ad_sine", 3, 64, 64, "fp32_mixed", 100),
        # the smallest request of the mix, with the limiter
        case("euler_rp2d_32_n2_mixed", "run", "euler_rp2d", 2, 32, 32, "fp32_mixed", 20),
        # smooth Euler flow at its named size, FP32-mixed and the reference's FP64
        case("euler_vortex_256_n4_mixed", "run", "euler_vortex", 4, 256, 256, "fp32_mixed", 40),
        case("euler_vortex_256_n4_fp64", "run", "euler_vortex", 4, 256, 256, "fp64", 20),
        # shocks and contacts at the named size, a few thousand cells limited each step
        case("euler_rp2d_512_n3_mixed", "run", "euler_rp2d", 3, 512, 512, "fp32_mixed", 20),
        # the same flow in FP64 on a ragged grid
        case("euler_rp2d_257x193_n3_fp64", "run", "euler_rp2d", 3, 257, 193, "fp64", 20),
        # the two-phase cylinder at its named size; in FP64 on a quarter of the cells
        case("bn_cylinder_400_n3_mixed", "run", "bn_cylinder", 3, 400, 400, "fp32_mixed", 20),
        case("bn_cylinder_200_n3_fp64", "run", "bn_cylinder", 3, 200, 200, "fp64", 20),
        # the highest degree, odd sides
        case("euler_rp2d_301x275_n5_mixed", "run", "euler_rp2d", 5, 301, 275, "fp32_mixed", 20),
        # a serving group: eight two-phase requests of mixed size stepped together
        case("bn_batch_8_n2_mixed", "batch", "bn_cylinder", 2, 300, 300, "fp32_mixed", 20, 8),
        # the all-FP32 split on a small two-phase grid
        case("bn_cylinder_97x61_n4_wide", "run", "bn_cylinder", 4, 97, 61, "fp32_wide", 20),
        # a host program that keeps its state on the host and calls one step at a time
        case("euler_vortex_128_n3_fp64_host", "host_step", "euler_vortex", 3, 128, 128, "fp64", 10),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    workload = rng.choice(["ad_sine", "euler_vortex", "euler_rp2d", "bn_cylinder"])
    call = rng.choice(["run"] * 5 + ["batch", "batch", "host_step"])
    precision = rng.choice(["fp64", "fp32_mixed", "fp32_mixed", "fp32_wide"])
    N = rng.randint(2, 5)
    steps = rng.randint(8, 20)
    count = rng.randint(3, 8) if call == "batch" else 1
    while True:
        c = dict(call=call, workload=workload, N=N, imax=side(24, 512), jmax=side(24, 512), precision=precision,
                 steps=steps, count=count)
        # no dearer than the largest listed case of its arithmetic
        w = work(c)
        if w["bytes"] <= 5e9 and w["flops"] <= (0.8e11 if precision == "fp64" else 2.7e11):
            return c


def sides(case):
    """The grids of the case's simulations: a batch's shrink by a quarter from one to the next."""
    return [(max(8, int(case["imax"] * 0.75 ** k)), max(8, int(case["jmax"] * 0.75 ** k))) for k in range(case["count"])]


def problems(case, seed):
    """(Config, initial field id, parameters) of every simulation: the workload's parameters jittered by 10%."""
    rng = random.Random(seed * 1009 + 17)
    out = []
    for imax, jmax in sides(case):
        cfg, ic, params, _ = workloads.make(case["workload"], side=imax, N=case["N"],
                                            precision=PRECISION[case["precision"]])
        cfg = dataclasses.replace(cfg, imax=imax, jmax=jmax)
        out.append((cfg, ic, tuple(p * rng.uniform(0.9, 1.1) for p in params)))
    return out


def prepare(case, seed):
    sims = problems(case, seed)
    # page-locked host memory for the results (the arrays keep their tensors alive)
    pinned = [torch.empty(cfg.dofs, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy() for cfg, _, _ in sims]
    state = dict(case=case, sims=sims, pinned=pinned)
    cfg, ic, params = sims[0]
    if case["call"] == "batch":
        state["batch"] = aderdg.Batch(cfg.system, cfg.N, cfg.precision, cfg.limiter,
                                      capacity_units=sum(aderdg.Batch.units(c) for c, _, _ in sims) + 64,
                                      max_instances=len(sims))
    else:
        state["solver"] = aderdg.Solver(cfg)
        if case["call"] == "host_step":
            state["initial"], state["lh"] = aderdg.project_initial_condition(cfg, ic, params)
    return state


def run(state):
    c, sims, pinned = state["case"], state["sims"], state["pinned"]
    if c["call"] == "batch":
        b = state["batch"]
        slots = [b.admit_ic(cfg, ic, params, 1e30, c["steps"]) for cfg, ic, params in sims]
        b.launch(c["steps"])
        b.sync()
        times = [b.query(s)["time"] for s in slots]
        uh = [b.download(s, p) for s, p in zip(slots, pinned)]
        status = [b.download_status(s) for s in slots]
        for s in slots:
            b.release(s)
        return dict(uh=uh, status=status, time=times)
    s, (cfg, ic, params), uh = state["solver"], sims[0], pinned[0]
    if c["call"] == "host_step":
        s.upload(state["initial"])
        s.init_limiter(state["lh"])
        uh[:] = state["initial"]
        t = 0.0
        for _ in range(c["steps"]):
            t, dt, n = s.step_host(uh, t, 1e30)
        return dict(uh=uh, time=t)
    s.initial_condition(ic, params)
    t, _ = s.run(0.0, 1e30, c["steps"])
    s.download_into(uh)
    out = dict(uh=uh, time=t)
    if cfg.limiter and cfg.system != aderdg.SYS_ADVDIFF:
        out["status"] = s.get(aderdg.A_STATUS)
    return out


def work(case):
    """Per step every degree of freedom is read and written once in FP64 (the
    global time step keeps steps apart); the flops are the predictor's
    contractions, its time update and its fluxes, the rest of a step being of
    lower order."""
    V = {"ad_sine": 1, "euler_vortex": 4, "euler_rp2d": 4, "bn_cylinder": 9}[case["workload"]]
    P = case["N"] + 1
    cells = sum(i * j for i, j in sides(case))
    flux = {1: 10, 4: 25, 9: 75}[V]
    per_node = P * (4 * P * V + 2 * P * V + flux) * (P - 2) + 2 * (4 * P * V + 2 * P * V + P * flux)
    return {"bytes": 16.0 * V * P * P * cells * case["steps"], "flops": float(per_node) * P * P * cells * case["steps"]}


# ---------------------------------------------------------------------------
# the scheme in 64 bits, all cells of a grid at once: arrays [j, i, y, x, v]


def legendre_operators(N):
    P, S = N + 1, 2 * N + 1
    x, w = np.polynomial.legendre.leggauss(P)
    x, w = 0.5 * (x + 1), 0.5 * w

    def basis(at):  # [point, k]
        at = np.atleast_1d(at)
        return np.array([[np.prod([(s - x[j]) / (x[k] - x[j]) for j in range(P) if j != k]) for k in range(P)] for s in at])

    D = np.array([[sum(np.prod([(s - x[j]) / (x[k] - x[j]) for j in range(P) if j != k and j != m]) / (x[k] - x[m])
                       for m in range(P) if m != k) for k in range(P)] for s in x])  # D[i, k] = phi_k'(x_i)
    left, right = basis(0.0)[0], basis(1.0)[0]
    stiff = (w[:, None] * D).T                    # stiff[a, b] = w_b phi_a'(x_b)
    K1inv = np.linalg.inv(np.outer(right, right) - stiff)
    sub = np.array([w @ basis((s + x) / S) for s in range(S)])       # subcell averages
    A = np.block([[2 * sub.T @ sub, -w[:, None]], [w[None, :], np.zeros((1, 1))]])
    back = np.linalg.solve(A, np.vstack([2 * sub.T, np.full((1, S), 1.0 / S)]))[:P]
    c = np.zeros(P)
    c[-1] = 1.0
    inner = np.polynomial.legendre.Legendre(c).deriv().roots() if P > 2 else np.array([])
    lob = basis(0.5 * (np.concatenate([[-1.0], np.sort(inner.real), [1.0]]) + 1))
    return dict(x=x, w=w, D=D, left=left, right=right, stiff=stiff, T=K1inv * w[None, :], g=K1inv @ left, sub=sub,
                back=back, lob=lob, bary=(np.arange(S) + 0.5) / S)


def euler_prim(Q, gamma):
    rho, mx, my, E = Q.unbind(-1)
    return rho, mx / rho, my / rho, (gamma - 1) * (E - 0.5 * (mx * mx + my * my) / rho)


class Exact:
    """One simulation in FP64; the flow of main.f90's loop body."""

    def __init__(self, cfg, ic, params, device):
        self.cfg, self.ic, self.p = cfg, ic, params
        self.P, self.S, self.V = cfg.N + 1, 2 * cfg.N + 1, cfg.nvar
        self.dx, self.dy = (cfg.xr[0] - cfg.xl[0]) / cfg.imax, (cfg.xr[1] - cfg.xl[1]) / cfg.jmax
        self.op = {k: torch.tensor(v, dtype=torch.float64, device=device) for k, v in legendre_operators(cfg.N).items()}
        self.device = device
        self.limiter = bool(cfg.limiter) and cfg.system != aderdg.SYS_ADVDIFF
        self.u = self.field(self.op["x"])
        self.time = 0.0
        if self.limiter:
            self.status = torch.zeros(cfg.jmax, cfg.imax, dtype=torch.bool, device=device)
            self.lh = self.field(self.op["bary"])
            lo, hi = self.u.amin((2, 3)), self.u.amax((2, 3))
            self.status = self.troubled(self.u, lo, hi, 0.1)

    # -- initial fields
    def field(self, at):
        c, p = self.cfg, self.p

        def grid(n, lo, d):
            k = torch.arange(n, dtype=torch.float64, device=self.device)
            return ((lo + (k + 0.5) * d) - 0.5 * d)[:, None] + at[None, :] * d

        X = grid(c.imax, c.xl[0], self.dx)[None, :, None, :]
        Y = grid(c.jmax, c.xl[1], self.dy)[:, None, :, None]
        X, Y = torch.broadcast_tensors(X, Y)
        if c.system == aderdg.SYS_ADVDIFF:
            return (p[0] * torch.sin(2 * math.pi * X) * torch.sin(2 * math.pi * Y))[..., None]
        if self.ic == aderdg.IC_EULER_VORTEX:
            g, eps = c.gamma, p[0]
            rx, ry = X - p[1], Y - p[2]
            r2 = rx * rx + ry * ry
            amp = eps / (2 * math.pi) * torch.exp(0.5 * (1 - r2))
            T0 = p[6] / p[3]
            T = T0 - (g - 1) * eps * eps / (8 * g * math.pi ** 2) * torch.exp(1 - r2)
            rho = p[3] * (T / T0) ** (1 / (g - 1))
            prim = [rho, p[4] - amp * ry, p[5] + amp * rx, rho * T]
        elif self.ic == aderdg.IC_EULER_RP2D:
            q = torch.where(Y >= p[1], torch.where(X >= p[0], 0, 1), torch.where(X < p[0], 2, 3))
            table = torch.tensor(p[2:18], dtype=torch.float64, device=self.device).reshape(4, 4)
            prim = list(table[q].unbind(-1))
        else:
            inside = (X - p[0]) ** 2 + (Y - p[1]) ** 2 < p[2] ** 2
            both = torch.tensor(p[3:13], dtype=torch.float64, device=self.device).reshape(2, 5)
            a, rs, ps, rg, pg = both[torch.where(inside, 0, 1)].unbind(-1)
            z = torch.zeros_like(a)
            es = rs * a * (ps + c.gamma_s * c.pi_s) / (rs * (c.gamma_s - 1))
            eg = (1 - a) * rg * (pg + c.gamma_g * c.pi_g) / (rg * (c.gamma_g - 1))
            return torch.stack([a * rs, z, z, es, (1 - a) * rg, z, z, eg, a], -1)
        r, ux, uy, pr = prim
        return torch.stack([r, r * ux, r * uy, pr / (c.gamma - 1) + 0.5 * r * (ux * ux + uy * uy)], -1)

    # -- physics
    def phases(self, Q):
        """Baer-Nunziato: (fraction, fraction * density, momenta, energy, pressure, sound speed) of both phases."""
        c, out = self.cfg, []
        for k, a, g, pi in ((0, Q[..., 8], c.gamma_s, c.pi_s), (4, 1 - Q[..., 8], c.gamma_g, c.pi_g)):
            m, mx, my, E = (Q[..., k + n] for n in range(4))
            p = (g - 1) * (E - 0.5 * (mx * mx + my * my) / m) / a - g * pi
            out.append((a, m, mx, my, E, p, g * (p + pi) * a / m, pi))
        return out

    def flux(self, Q):
        if self.cfg.system == aderdg.SYS_EULER:
            r, ux, uy, p = euler_prim(Q, self.cfg.gamma)
            E = Q[..., 3]
            return (torch.stack([r * ux, r * ux * ux + p, r * ux * uy, ux * (E + p)], -1),
                    torch.stack([r * uy, r * ux * uy, r * uy * uy + p, uy * (E + p)], -1))
        fx, fy = [], []
        for a, m, mx, my, E, p, _, _ in self.phases(Q):
            ux, uy = mx / m, my / m
            fx += [mx, mx * ux + a * p, my * ux, ux * (E + a * p)]
            fy += [my, mx * uy, my * uy + a * p, uy * (E + a * p)]
        z = torch.zeros_like(Q[..., 8])
        return torch.stack(fx + [z], -1), torch.stack(fy + [z], -1)

    def speed(self, Q, d):
        if self.cfg.system == aderdg.SYS_EULER:
            r, ux, uy, p = euler_prim(Q, self.cfg.gamma)
            waves = [((ux, uy)[d], self.cfg.gamma * p / r)]
        else:
            waves = [((mx, my)[d] / m, c2) for _, m, mx, my, _, _, c2, _ in self.phases(Q)]
        fastest = torch.zeros_like(Q[..., 0])
        for un, c2 in waves:  # the larger speed, a NaN left out as Fortran's max does
            fastest = torch.fmax(fastest, torch.fmax(un.abs(), un.abs() + torch.sqrt(c2)))
        return fastest

    def column(self, Q, gx, gy):
        """Non-conservative product with the volume-fraction gradient (gx, gy)."""
        (_, ms, mx, my, _, _, _, _), gas = self.phases(Q)
        p, un = gas[5], (mx * gx + my * gy) / ms
        z = torch.zeros_like(p)
        return torch.stack([z, -p * gx, -p * gy, -p * un, z, p * gx, p * gy, p * un, un], -1)

    def fluctuation(self, QL, QR, d):
        jump, D = QR - QL, 0
        one, z = torch.ones_like(jump[..., 8]), torch.zeros_like(jump[..., 8])
        for s, w in ((0.5 - math.sqrt(15) / 10, 5 / 18), (0.5, 8 / 18), (0.5 + math.sqrt(15) / 10, 5 / 18)):
            D = D + w * self.column(QL + s * jump, one if d == 0 else z, one if d == 1 else z)
        return D * jump[..., 8:9]

    def positive(self, Q):
        if self.cfg.system == aderdg.SYS_EULER:
            r, _, _, p = euler_prim(Q, self.cfg.gamma)
            return ~((r <= 1e-12) | (p <= 1e-12))
        bad = (Q[..., 8] <= 0) | (Q[..., 8] >= 1)
        for a, m, _, _, _, p, _, pi in self.phases(Q):
            bad = bad | (m / a <= 1e-12) | (p + pi <= 1e-12)
        return ~bad

    # -- the step
    def time_step(self):
        c = self.cfg
        pnpm = (1.0, 0.33, 0.17, 0.1, 0.069, 0.045)[c.N]
        if c.system == aderdg.SYS_ADVDIFF:
            f = 2 * c.N + 1
            den = (abs(c.cx) + 2 * c.a * f / self.dx) / self.dx + (abs(c.cy) + 2 * c.a * f / self.dy) / self.dy
        else:
            den = float((self.speed(self.u, 0) / self.dx + self.speed(self.u, 1) / self.dy).max())
        return c.cfl * pnpm / den

    def predictor(self, dt):
        """Time averages (q, Fx, Fy, -NCP or gradient) of the space-time predictor."""
        o, c, P = self.op, self.cfg, self.P
        grad = lambda q: (torch.einsum("ak,...kv->...av", o["D"], q) / self.dx,          # noqa: E731
                          torch.einsum("bk,...kav->...bav", o["D"], q) / self.dy)
        q = self.u[None].expand(P, *self.u.shape)
        for _ in range(P):
            if c.system == aderdg.SYS_ADVDIFF:
                gx, gy = grad(q)
                Fx, Fy = -c.a * gx, -c.a * gy
                if c.ad_flux_mode:
                    Fx, Fy = Fx + c.cx * q, Fy + c.cy * q
                extra = (gx, gy)
            else:
                Fx, Fy = self.flux(q)
                extra = ()
            b = grad(Fx)[0] + grad(Fy)[1]
            if c.system == aderdg.SYS_BN:
                ax, ay = grad(q[..., 8:9])
                extra = (-self.column(q, ax[..., 0], ay[..., 0]),)
                b = b - extra[0]
            q = o["g"].reshape(-1, *[1] * self.u.dim()) * self.u - dt * torch.einsum("ml,l...->m...", o["T"], b)
        mean = lambda f: torch.einsum("l,l...->...", o["w"], f)                         # noqa: E731
        return mean(q), mean(Fx), mean(Fy), tuple(mean(e) for e in extra)

    def across(self, f, side, d):
        """Values of face field f[side] on the left / right of every face along d, boundaries included."""
        lo, hi = f
        ax = 1 if d == 0 else 0
        first, last = lo.narrow(ax, 0, 1), hi.narrow(ax, -1 % hi.shape[ax], 1)
        wrap = self.cfg.bc[2 * d] == 3
        return (torch.cat([last if wrap else first, hi], ax) if side == 0
                else torch.cat([lo, first if wrap else last], ax))

    def faces(self, q, F, extra, d):
        """Numerical flux on every face along d: (seen from the left cell, seen from the right cell)."""
        o, c = self.op, self.cfg
        eq = "k,jiykv->jiyv" if d == 0 else "k,jikxv->jixv"
        ends = lambda f: (torch.einsum(eq, o["left"], f), torch.einsum(eq, o["right"], f))  # noqa: E731
        qs = ends(q)
        QL, QR = self.across(qs, 0, d), self.across(qs, 1, d)
        if c.system == aderdg.SYS_ADVDIFF:
            gs = ends(extra[d])
            gL, gR = self.across(gs, 0, d), self.across(gs, 1, d)
            speed = (c.cx, c.cy)[d]
            smax = abs(speed) + 2 * c.a * (2 * c.N + 1) / (self.dx * math.sqrt(0.5 * math.pi))
            f = 0.5 * (speed * (QL + QR) - c.a * (gL + gR)) - 0.5 * smax * (QR - QL)
            return f, f
        fs = ends(F)
        smax = torch.fmax(self.speed(QL, d), self.speed(QR, d))[..., None]
        f = 0.5 * (self.across(fs, 0, d) + self.across(fs, 1, d)) - 0.5 * smax * (QR - QL)
        if c.system != aderdg.SYS_BN:
            return f, f
        D = self.fluctuation(QL, QR, d)
        return f + 0.5 * D, f - 0.5 * D

    def step(self):
        o, c = self.op, self.cfg
        dt = self.time_step()
        if self.limiter:
            lo, hi = self.bounds()
            self.was = self.status
        q, Fx, Fy, extra = self.predictor(dt)
        w = o["w"]
        r = torch.einsum("ak,jiykv->jiyav", o["stiff"], Fx) / (self.dx * w[:, None])
        r = r + torch.einsum("bk,jikxv->jibxv", o["stiff"], Fy) / (self.dy * w[:, None, None])
        if c.system == aderdg.SYS_BN:
            r = r + extra[0]
        # a cell sees its right (top) face from that face's left (lower) side
        seen_left, seen_right = self.faces(q, Fx, extra, 0)
        right, left = seen_left[:, 1:, :, None], seen_right[:, :-1, :, None]
        r = r - (right * o["right"][:, None] - left * o["left"][:, None]) / (self.dx * w[:, None])
        seen_left, seen_right = self.faces(q, Fy, extra, 1)
        top, bottom = seen_left[1:, :, None], seen_right[:-1, :, None]
        r = r - (top * o["right"][:, None, None] - bottom * o["left"][:, None, None]) / (self.dy * w[:, None, None])
        new = self.u + dt * r
        if self.limiter:
            new = self.limit(new, lo, hi, dt)
        self.u = new
        self.time += dt

    # -- limiter
    def project(self, u):
        s = torch.einsum("sy,...yxv->...sxv", self.op["sub"], u)
        return torch.einsum("sx,...yxv->...ysv", self.op["sub"], s)

    def extremes(self, u):
        s = self.project(u)
        lob = torch.einsum("sy,...yxv->...sxv", self.op["lob"], u)
        lob = torch.einsum("sx,...yxv->...ysv", self.op["lob"], lob)
        every = torch.cat([f.flatten(-3, -2) for f in (u, s, lob)], -2)
        return s, every.nan_to_num(math.inf, math.inf, -math.inf).amin(-2), every.nan_to_num(-math.inf, math.inf, -math.inf).amax(-2)

    def troubled(self, u, lo, hi, floor=0.0):
        s, mn, mx = self.extremes(u)
        tol = torch.clamp(1e-3 * (hi - lo), min=max(1e-4, floor))
        return ((mn < lo - tol) | (mx > hi + tol)).any(-1) | ~self.positive(s).all(-1).all(-1)

    def shift(self, f, dj, di):
        for ax, d in ((0, dj), (1, di)):
            if d:
                n = f.shape[ax]
                k = torch.arange(n, device=f.device) + d
                f = f.index_select(ax, k % n if self.cfg.bc[2 if ax == 0 else 0] == 3 else k.clamp(0, n - 1))
        return f

    def bounds(self):
        _, lo, hi = self.extremes(self.u)
        st = self.status[..., None]
        lo, hi = torch.where(st, self.lh.amin((2, 3)), lo), torch.where(st, self.lh.amax((2, 3)), hi)
        at = [(j, i) for j in (-1, 0, 1) for i in (-1, 0, 1)]
        return (torch.stack([self.shift(lo, j, i) for j, i in at]).amin(0),
                torch.stack([self.shift(hi, j, i) for j, i in at]).amax(0))

    def limit(self, new, lo, hi, dt):
        o, S = self.op, self.S
        bad = self.troubled(new, lo, hi)
        near = torch.zeros_like(bad)
        for dj, di in ((0, -1), (0, 1), (-1, 0), (1, 0)):
            near = near | self.shift(bad, dj, di)
        js, is_ = torch.nonzero(bad | near, as_tuple=True)
        self.status = bad.clone()
        if js.numel() == 0:
            return new
        # subcell data of the 3 x 3 neighbourhood, two rings of it
        n_j, n_i = bad.shape
        wrap = self.cfg.bc[0] == 3, self.cfg.bc[2] == 3
        rows = []
        for dj in (-1, 0, 1):
            row = []
            for di in (-1, 0, 1):
                a, b = js + dj, is_ + di
                a = a % n_j if wrap[1] else a.clamp(0, n_j - 1)
                b = b % n_i if wrap[0] else b.clamp(0, n_i - 1)
                row.append(torch.where(self.was[a, b][:, None, None, None], self.lh[a, b], self.project(self.u[a, b])))
            rows.append(torch.cat(row, 2))
        s = torch.cat(rows, 1)[:, S - 2:2 * S + 2, S - 2:2 * S + 2]  # subcells -1 .. S+2
        sub = self.subcells(s, dt)
        poly = torch.einsum("ys,nsxv->nyxv", o["back"], sub)
        poly = torch.einsum("xs,nysv->nyxv", o["back"], poly)
        fails = self.troubled(poly, lo[js, is_], hi[js, is_])
        limited = bad[js, is_] | fails
        new = new.clone()
        new[js, is_] = poly
        self.status[js, is_] = limited
        self.lh[js[limited], is_[limited]] = sub[limited]
        return new

    def subcells(self, s, dt):
        """MUSCL-Hancock step of the S x S subcells from s[cell, y, x, v] with two rings around them."""
        hx, hy = self.dx / self.S, self.dy / self.S
        bn = self.cfg.system == aderdg.SYS_BN

        def slope(a, b):
            return torch.where(a * b <= 0, 0.0, torch.where(a.abs() < b.abs(), a, b))

        c = s[:, 1:-1, 1:-1]  # subcells 0 .. S+1
        sx = slope(s[:, 1:-1, 2:] - c, c - s[:, 1:-1, :-2])
        sy = slope(s[:, 2:, 1:-1] - c, c - s[:, :-2, 1:-1])
        if not bn:  # Euler reconstructs the cell's own subcells only
            own = torch.zeros_like(c[:1, :, :, :1])
            own[:, 1:-1, 1:-1] = 1
            sx, sy = sx * own, sy * own
        rate = -(self.flux(c + 0.5 * sx)[0] - self.flux(c - 0.5 * sx)[0]) / hx
        rate = rate - (self.flux(c + 0.5 * sy)[1] - self.flux(c - 0.5 * sy)[1]) / hy
        if bn:
            rate = rate - self.column(c, sx[..., 8] / hx, sy[..., 8] / hy)
        half = c + 0.5 * dt * rate
        out = c[:, 1:-1, 1:-1]
        for d, sl, h in ((0, sx, hx), (1, sy, hy)):
            ax = 2 - d
            plus, minus = half + 0.5 * sl, half - 0.5 * sl
            inner = (slice(None), slice(1, -1)) if d == 0 else (slice(None), slice(None), slice(1, -1))
            plus, minus = plus[inner], minus[inner]
            m = plus.shape[ax]
            QL, QR = plus.narrow(ax, 0, m - 1), minus.narrow(ax, 1, m - 1)
            smax = torch.fmax(self.speed(QL, d), self.speed(QR, d))[..., None]
            F = 0.5 * (self.flux(QL)[d] + self.flux(QR)[d]) - 0.5 * smax * (QR - QL)
            k = F.shape[ax]
            out = out - dt / h * (F.narrow(ax, 1, k - 1) - F.narrow(ax, 0, k - 1))
            if bn:
                D = self.fluctuation(QL, QR, d)
                out = out - 0.5 * dt / h * (D.narrow(ax, 1, k - 1) + D.narrow(ax, 0, k - 1))
        if bn:
            mid = half[:, 1:-1, 1:-1]
            out = out - dt * self.column(mid, sx[:, 1:-1, 1:-1, 8] / hx, sy[:, 1:-1, 1:-1, 8] / hy)
        return out


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    uh, times = [], []
    for cfg, ic, params in problems(case, seed):
        e = Exact(cfg, ic, params, device)
        for _ in range(case["steps"]):
            e.step()
        uh.append(e.u.reshape(-1).cpu().numpy())
        times.append(e.time)
    if case["call"] == "batch":
        return dict(uh=uh, status=None, time=times)
    out = dict(uh=uh[0], time=times[0])
    if case["call"] == "run" and cfg.limiter and cfg.system != aderdg.SYS_ADVDIFF:
        out["status"] = None
    return out
