"""Timed cases of the time-stepping and Newton paths, over the sizes their users run.

A case is one call a user's program makes on a prepared plan: a run of IMEX steps of one shell or of a batch,
a batch of uneven shells replayed from its captured graph, the Newton residual, the Jacobian products of a
Krylov solve, steps with their per-step diagnostics, a whole Newton-GMRES solve.  ``exact`` restates the same
operations in dense FP64 numpy (transforms as matrices, chains as plain recurrences).
"""
import math

import numpy as np
import torch

from spectraldoublediffusiveconvection_gb300.batch import ShellBatch
from spectraldoublediffusiveconvection_gb300.plan import Plan

D_GAP, PR, RA_S = 2.0, 1.0, 500.0      # the shell's gap parameter, Prandtl number, solutal Rayleigh number

#: theta modes whose 3/2-padded transform length has only the factors 2, 3, 5, 7
MODES = (24, 32, 40, 48, 56, 64, 80, 90, 96, 112, 120, 128, 150, 160, 180, 192, 210, 240, 256, 288, 320, 336,
         384, 420, 450, 480, 512, 540)


def _case(name, kind, N_r, M, batch, precision="fp64", nsteps=1, symmetric=False, linear=False, dt=1e-3, tau=0.01):
    return dict(name=name, kind=kind, N_r=N_r, M=M, batch=batch, precision=precision, nsteps=nsteps,
                symmetric=symmetric, linear=linear, dt=dt, tau=tau)


def listed():
    return [
        # the smallest call: one step of a small shell, e.g. a driver that looks at the state after every step
        _case("step_one_20x64", "step", 20, 64, 1),
        # the production-size shell, 100 steps a call: the headline workload
        _case("steps_shell_30x256", "step", 30, 256, 1, nsteps=100, dt=5e-4),
        # a quantum of the request server: a few shells of one shape, mixed precision
        _case("quantum_mixed_28x128", "step", 28, 128, 3, "mixed", nsteps=50, tau=1.0),
        # the largest shape a plan takes, one shell
        _case("steps_largest_65x540", "step", 65, 540, 1, nsteps=20, dt=5e-4),
        # many shells of one shape, plain and mixed
        _case("steps_batch64_30x256", "step", 30, 256, 64, nsteps=10),
        _case("steps_batch64_mixed_30x256", "step", 30, 256, 64, "mixed", nsteps=10),
        # 64 shells of 16 shapes in one captured graph of 10 steps
        _case("uneven64_mixed", "uneven", 0, 0, 64, "mixed", nsteps=10),
        # time stepping with the per-step norm, kinetic energy and Nusselt records, equatorially symmetric, ragged
        _case("steps_diag_sym_23x90", "diag", 23, 90, 1, nsteps=20, symmetric=True),
        # the Newton residual of one shell and the Jacobian products of a batch (dt = 1 operators)
        _case("residual_30x256", "residual", 30, 256, 1, dt=1.0),
        _case("jacobian_batch16_mixed_36x192", "jacobian", 36, 192, 16, "mixed", dt=1.0),
        # a whole steady-state solve from a time-stepped convecting state, plain FP64 and batched mixed
        _case("newton_20x64", "newton", 20, 64, 1, dt=1.0, tau=1.0),
        _case("newton_batch8_mixed_24x64", "newton", 24, 64, 8, "mixed", dt=1.0, tau=1.0),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "diag", "residual", "jacobian"])
    while True:
        N_r = int(round(math.exp(rng.uniform(math.log(8), math.log(65)))))
        M = rng.choice(MODES)
        batch = int(round(math.exp(rng.uniform(0.0, math.log(64)))))
        nsteps = int(round(math.exp(rng.uniform(0.0, math.log(100))))) if kind in ("step", "diag") else 1
        sym = rng.random() < 0.25
        c = dict(kind=kind, N_r=N_r, M=M, batch=batch, precision=rng.choice(["fp64", "mixed"]), nsteps=nsteps,
                 symmetric=sym, linear=kind == "step" and rng.random() < 0.1,
                 dt=1.0 if kind in ("residual", "jacobian") else rng.choice([5e-4, 1e-3]),
                 tau=rng.choice([0.01, 1.0]))
        if work(c)["flops"] <= 4e9 and batch * M * N_r <= 64 * 256 * 40:
            return c


# ---- inputs ---------------------------------------------------------------------------------------


def _state(M, nr, batch, symmetric, rng, amp):
    """Smooth convecting fields: modes decaying in theta, radial profiles that vanish at the walls (psi with its
    slope), (batch, 3 M nr)."""
    s = 0.5 * (1.0 - np.cos(np.pi * np.arange(1, nr + 1) / (nr + 1)))
    m = np.arange(1, 5)[:, None]
    prof = np.sin(np.pi * m * s[None, :])
    X = np.zeros((batch, 3, M, nr))
    k = np.arange(M)[None, :, None]
    for f in range(3):
        c = rng.standard_normal((batch, M, 4)) * np.exp(-k / 6.0) * np.exp(-np.arange(4) / 1.5)
        X[:, f] = amp * (c @ (prof * (np.sin(np.pi * s) if f == 0 else 1.0)))
    if symmetric:
        X[:, 0, 0::2] = 0.0
        X[:, 1:, 1::2] = 0.0
    return X.reshape(batch, -1)


def _shells(seed, n):
    """Shells of mixed shapes (the same for every seed) with seeded Rayleigh numbers and states."""
    shape, rng = np.random.default_rng(1234), np.random.default_rng(seed)
    N_r = shape.choice([20, 24, 30, 36], size=n)
    M = shape.choice([64, 128, 256, 384], size=n)
    Ra = rng.uniform(6000.0, 12000.0, size=n)
    return [dict(N_r=int(a), N_theta=int(b), Ra=float(c), X=_state(int(b), int(a) - 1, 1, False, rng, 0.05)[0])
            for a, b, c in zip(N_r, M, Ra)]


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    M, nr, B = case["M"], case["N_r"] - 1, case["batch"]
    Ra = rng.uniform(6000.0, 9000.0, size=B)
    X = _state(M, nr, B, case["symmetric"], rng, 0.05)
    dv = _state(M, nr, B, case["symmetric"], rng, 1.0)
    return X, dv, Ra


def prepare(case, seed):
    if case["kind"] == "uneven":
        shells = _shells(seed, case["batch"])
        sb = ShellBatch(shells, d=D_GAP, dt=case["dt"], Pr=PR, Tau=case["tau"], Ra_s=RA_S, precision=case["precision"])
        sb.capture(case["nsteps"])
        return dict(kind="uneven", batch=sb)
    plan = Plan(case["M"], case["N_r"], D_GAP, case["dt"], PR, case["tau"], symmetric=case["symmetric"],
                precision=case["precision"])
    plan.reserve(case["batch"])
    X, dv, Ra = _inputs(case, seed)
    st = dict(kind=case["kind"], plan=plan, X=torch.from_numpy(X).cuda(), Ra=torch.from_numpy(Ra).cuda(),
              nsteps=case["nsteps"], linear=case["linear"])
    if case["kind"] == "jacobian":
        st["dv"] = torch.from_numpy(dv).cuda()
        st["base"] = plan.new_base(case["batch"])
        plan.pfx(st["X"], st["Ra"], RA_S, base=st["base"])     # the residual of the same X leaves its grid fields
    elif case["kind"] == "newton":
        # a convecting state near its steady branch: 6 diffusion times of stepping from the seeded state
        Ra = 9000.0 + 50.0 * np.arange(case["batch"]) + (seed % 7)
        st["Ra"] = torch.from_numpy(Ra).cuda()
        stepper = Plan(case["M"], case["N_r"], D_GAP, 2e-3, PR, case["tau"])
        st["X"] = stepper.step(st["X"], st["Ra"], RA_S, nsteps=3000)
        torch.cuda.synchronize()
        stepper.close()
        st["mv"] = 3 if case["precision"] == "mixed" else 0
    else:
        st["out"] = torch.empty_like(st["X"])
    return st


def run(state):
    kind = state["kind"]
    if kind == "uneven":
        state["batch"].replay()
        return [g.X for g in state["batch"].groups]
    plan, X, Ra = state["plan"], state["X"], state["Ra"]
    if kind == "step":
        return plan.step(X, Ra, RA_S, nsteps=state["nsteps"], linear=state["linear"], out=state["out"])
    if kind == "diag":
        return plan.step_diag(X, Ra, RA_S, nsteps=state["nsteps"], out=state["out"])
    if kind == "residual":
        return plan.pfx(X, Ra, RA_S, out=state["out"])
    if kind == "jacobian":
        return plan.pdfx(state["dv"], X, Ra, RA_S, base=state["base"])
    Xs = X.clone()
    plan.newton(Xs, Ra, RA_S, tol=1e-12, mixed_matvec=state["mv"])
    return Xs


def _step_work(M, nr):
    P = 3 * M // 2
    return 21.0 * M * nr * nr + 30.0 * nr * P * math.log2(P) + 11.0 * nr * P + 40.0 * nr * M


def work(case):
    """Bytes: the states in and out and the plan's implicit-solve blocks once each; flops: the transforms as FFTs,
    the radial contractions, the solves' two matvecs per mode (a Newton solve: 30 products of the Krylov space)."""
    if case["kind"] == "uneven":
        sh = [(s["N_theta"], s["N_r"] - 1) for s in _shells(0, case["batch"])]
        return {"bytes": sum(48.0 * M * nr for M, nr in sh) + sum(24.0 * M * nr * nr for M, nr in set(sh)),
                "flops": case["nsteps"] * sum(_step_work(M, nr) for M, nr in sh)}
    M, nr, B = case["M"], case["N_r"] - 1, case["batch"]
    f = _step_work(M, nr) * B
    io = 48.0 * M * nr * B
    n = case["nsteps"]
    if case["kind"] == "jacobian":
        io += 24.0 * M * nr * B
    if case["kind"] == "newton":
        n = 30
    return {"bytes": io + 24.0 * M * nr * nr, "flops": n * f}


# ---- the same operations in dense FP64 numpy ------------------------------------------------------


class _Dense:
    """Operators of one shell shape: Chebyshev collocation in r, sine (psi) and cosine (T, S) modes in theta."""

    def __init__(self, M, N_r, dt, Tau, d=D_GAP, Pr=PR):
        ri, ro, nr = 1.0 / d, (1.0 + d) / d, N_r - 1
        self.M, self.nr, self.dt, self.Pr, self.Tau = M, nr, dt, Pr, Tau
        n = np.arange(N_r + 1)
        r = 0.5 * (ri + ro) + 0.5 * (ri - ro) * np.cos(np.pi * n / N_r)
        c = np.where((n == 0) | (n == N_r), 2.0, 1.0) * (-1.0) ** n
        D = np.outer(c, 1.0 / c) / (r[:, None] - r[None, :] + np.eye(N_r + 1))
        D -= np.diag(D.sum(axis=1))
        i = slice(1, -1)
        self.r, self.D = r, D
        x = self.x = r[i]
        D2 = D @ D
        self.Dr, self.D2 = D[i, i], D2[i, i]
        self.dT0 = (ri * ro / (ri - ro)) / x ** 2
        self.gr = ri ** 2 / x ** 2
        # psi solve: A^2 - dt Pr A^4, block diagonal part per sine mode j; T, S: r^2 - dt r^2 Lap
        b, cc = -(ri + ro), ri * ro
        q = r ** 2 + b * r + cc
        qi = np.zeros_like(q)
        qi[1:-1] = 1.0 / q[1:-1]
        D3 = D @ D2
        L4 = ((q[:, None] * (D2 @ D2) + 4.0 * (2.0 * r + b)[:, None] * D3 + 12.0 * D2) * qi[None, :])[i, i]
        self.ir2, self.ir4 = 1.0 / x ** 2, 1.0 / x ** 4
        self.D2A = ((2.0 * D2 - 4.0 * D / r[:, None] + 6.0 * np.diag(1.0 / r ** 2)) / (r ** 2)[:, None])[i, i]
        j = (M - np.arange(M))[:, None, None].astype(float)
        bj = -j * (j + 1.0)
        I2, I4 = np.diag(self.ir2), np.diag(self.ir4)
        h = Pr * dt
        self.LA = np.linalg.inv((self.D2 + bj * I2) - h * (L4 + bj * (self.D2A + bj * I4)))
        lap = (r[:, None] ** 2 * D2 + 2.0 * r[:, None] * D)[i, i]
        j = j - 1.0
        bj = -j * (j + 1.0)
        R2, eye = np.diag(x ** 2), np.eye(nr)
        self.LT = np.linalg.inv(R2 - dt * (lap + bj * eye))
        self.LS = np.linalg.inv(R2 - Tau * dt * (lap + bj * eye))
        P = 3 * M // 2
        th = np.pi * (2.0 * np.arange(P) + 1.0) / (2.0 * P)
        self.P = P
        self.C = np.cos(np.outer(np.arange(M), th))                # cosine modes 0 .. M-1
        self.S = np.sin(np.outer(np.arange(1, M + 1), th))         # sine slot s is wavenumber s + 1
        self.S[-1] = 0.0                                           # the top slot is not evaluated

    def suffix(self, G):
        out = np.empty_like(G)
        for p in (0, 1):
            out[:, p::2] = np.cumsum(G[:, p::2][:, ::-1], axis=1)[:, ::-1]
        return out

    def jtheta(self, psi):
        s = np.zeros_like(psi)
        s[:, :-1] = self.suffix(psi)[:, 1:]
        f = 2.0 * s
        f[:, 1:] += np.arange(2.0, self.M + 1.0)[:, None] * psi[:, :-1]
        f[:, 0] = s[:, 0]
        return f

    def a2(self, psi, D2, ir):
        s = np.zeros_like(psi)
        s[:, :-2] = self.suffix(psi)[:, 2:]
        j = np.arange(1.0, self.M + 1.0)[:, None]
        return psi @ D2.T - j * ir * ((j + 1.0) * psi + 2.0 * s)

    def fields(self, X, sym):
        psi, T, S = X[:, 0], X[:, 1], X[:, 2]
        k = np.arange(self.M)[:, None]
        ks = k + 1.0
        jt, om, dp = self.jtheta(psi), self.a2(psi, self.D2 / self.x[:, None] ** 2, self.ir4), psi @ self.Dr.T
        spec_c = [jt, ks * om, ks * dp, T @ self.Dr.T, S @ self.Dr.T]
        spec_s = [om, dp, -k * T, -k * S]
        if sym:
            for a in (om, dp, spec_c[1], spec_c[2]):
                a[:, 0::2] = 0.0
            for a in (jt, spec_c[3], spec_c[4], spec_s[2], spec_s[3]):
                a[:, 1::2] = 0.0
        to = lambda a, E: np.einsum("bkn,kp->bnp", a, E, optimize=True)
        up = np.zeros_like(self.C)
        up[:-1] = self.C[1:]                                       # sine-slot quantities times cos((s+1) theta)
        sn = np.zeros_like(self.C)
        sn[1:] = self.S[:-1]                                       # cosine-slot quantities times sin(k theta)
        JT, DT, DC = (to(spec_c[q], self.C) for q in (0, 3, 4))
        kO, kD = to(spec_c[1], up), to(spec_c[2], up)
        O, Dp = to(om, self.S), to(dp, self.S)
        kT, kC = to(spec_s[2], sn), to(spec_s[3], sn)
        return JT, kO, kD, DT, DC, O, Dp, kT, kC

    def nlin(self, a, b, sym):
        """The bilinear term of grid fields a and b, in modes (batch, 3, M, nr)."""
        JT, kO, kD, DT, DC, O, Dp, kT, kC = b
        aJT, akO, akD, aDT, aDC, aO, aDp, akT, akC = a
        if a is b:
            q, r = JT * O, kD * O + Dp * kO
            nt, ns = JT * DT - Dp * kT, JT * DC - Dp * kC
        else:
            q = aJT * O + JT * aO
            r = akD * O + aDp * kO + kD * aO + Dp * akO
            nt = JT * aDT - Dp * akT + aJT * DT - aDp * kT
            ns = JT * aDC - Dp * akC + aJT * DC - aDp * kC
        back = lambda g, E: np.einsum("bnp,kp->bkn", g, E, optimize=True) * (2.0 / self.P)
        F = np.stack([back(q, self.S) @ self.Dr.T - back(r, self.S), back(nt, self.C), back(ns, self.C)], axis=1)
        F[:, 1:, 0] *= 0.5
        if sym:
            F[:, 0, 0::2] = 0.0
            F[:, 1:, 1::2] = 0.0
        return F

    def solve(self, G, sym):
        """The three mode-coupled solves, both parities of each from the top mode down."""
        M, F, h = self.M, np.zeros_like(G), self.Pr * self.dt
        mv = lambda A, x: x @ A.T
        for p in ((0,) if sym else (0, 1)):
            fe, bf = np.zeros_like(G[:, 0, 0]), np.zeros_like(G[:, 0, 0])
            for jj in range(p, M, 2):
                row, j = M - 1 - jj, float(M - jj)
                bj, bt = -j * (j + 1.0), -2.0 * j
                g = G[:, 0, row]
                if jj > p:
                    fe = fe + F[:, 0, row + 2]
                    g = g + h * bt * (mv(self.D2A, fe) + bj * self.ir4 * fe + self.ir4 * bf) - bt * self.ir2 * fe
                F[:, 0, row] = mv(self.LA[jj], g)
                bf = bf + bj * F[:, 0, row] + (bt * fe if jj > p else 0.0)
        for f, L, h in ((1, self.LT, self.dt), (2, self.LS, self.Tau * self.dt)):
            for p in ((1,) if sym else (0, 1)):
                b = np.zeros_like(G[:, 0, 0])
                for jj in range(p, M, 2):
                    j = M - 1 - jj
                    if jj > p:
                        b = b + 2.0 * h * (j + 2.0) * F[:, f, j + 2]
                    F[:, f, j] = mv(L[jj], G[:, f, j] - (0.5 if j == 0 else 1.0) * b)
        return F

    def rhs(self, X, NX, Ra, sym):
        psi, T, S = X[:, 0], X[:, 1], X[:, 2]
        G = NX.copy()
        k1 = np.arange(1.0, self.M)[:, None]
        buoy = np.zeros_like(psi)
        buoy[:, :-1] = -k1 * self.gr * (Ra[:, None, None] * T[:, 1:] - RA_S * S[:, 1:])
        G[:, 0] += self.a2(psi, self.D2, self.ir2) + self.dt * self.Pr * buoy
        t0 = self.dT0 * self.jtheta(psi)
        G[:, 1] += self.x ** 2 * T - self.dt * t0
        G[:, 2] += self.x ** 2 * S - self.dt * t0
        return G

    def step(self, X, Ra, sym, linear=False):
        NX = np.zeros_like(X)
        if not linear:
            a = self.fields(X, sym)
            NX = -self.dt * self.nlin(a, a, sym)
        return self.solve(self.rhs(X, NX, Ra, sym), sym)

    def diagnostics(self, X, sym):
        """|X|, volume-mean kinetic energy, the inner-wall Nusselt sums of T and S of one shell (3, M, nr)."""
        M, r, n3 = self.M, self.r, 3 * self.M
        th = np.pi * (2.0 * np.arange(n3) + 1.0) / (2.0 * n3)
        J = self.jtheta(X[None, 0])[0]
        if sym:
            J = J.copy()
            J[1::2] = 0.0
        k = np.arange(M)
        sn = np.sin(np.outer(k + 1, th))
        sn[-1] = 0.0
        u = (J / self.x).T @ np.cos(np.outer(k, th))
        v = (X[0] @ self.Dr.T).T @ sn
        ke = np.trapezoid(np.trapezoid(u ** 2 + v ** 2, x=self.x, axis=0) * np.sin(th), x=th)
        ke *= 0.5 / ((2.0 / 3.0) * (r[-1] ** 3 - r[0] ** 3))
        at = r[0] * r[-1] / (r[0] - r[-1])
        ev = np.arange(0, M, 2)
        w = (r[0] ** 2 / at) * self.D[0, 1:-1]
        nus = [float(((X[f, ev] @ w) / (1.0 - ev ** 2.0)).sum()) for f in (1, 2)]
        return [float(np.sqrt((X ** 2).sum())), float(ke)] + nus


def exact(case, seed):
    kind = case["kind"]
    if kind == "newton":
        return None                    # its start is a state stepped for thousands of steps
    if kind == "uneven":
        shells = _shells(seed, case["batch"])
        groups = {}
        for s in shells:
            groups.setdefault((s["N_r"], s["N_theta"]), []).append(s)
        out = []
        for (N_r, M), g in sorted(groups.items(), key=lambda kv: -kv[0][1] * kv[0][0]):
            ops = _Dense(M, N_r, case["dt"], case["tau"])
            X = np.stack([s["X"] for s in g]).reshape(len(g), 3, M, N_r - 1)
            Ra = np.array([s["Ra"] for s in g])
            for _ in range(case["nsteps"]):
                X = ops.step(X, Ra, False)
            out.append(X.reshape(len(g), -1))
        return out
    M, nr, B, sym = case["M"], case["N_r"] - 1, case["batch"], case["symmetric"]
    if case["nsteps"] * B * M * nr > 8e6:
        return None                    # over the time such a check may take
    X, dv, Ra = _inputs(case, seed)
    ops = _Dense(M, case["N_r"], case["dt"], case["tau"])
    X, dv = X.reshape(B, 3, M, nr), dv.reshape(B, 3, M, nr)
    if kind == "residual":
        return (ops.step(X, Ra, sym) - X).reshape(B, -1)
    if kind == "jacobian":
        NX = -ops.dt * ops.nlin(ops.fields(X, sym), ops.fields(dv, sym), sym)
        return (ops.solve(ops.rhs(dv, NX, Ra, sym), sym) - dv).reshape(B, -1)
    diag = []
    for _ in range(case["nsteps"]):
        X = ops.step(X, Ra, sym, case["linear"])
        if kind == "diag":
            diag.append([ops.diagnostics(X[b], sym) for b in range(B)])
    if kind == "diag":
        return X.reshape(B, -1), np.array(diag)
    return X.reshape(B, -1)
