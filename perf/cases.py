"""The work that users of this package have it do, as cases that can be timed and compared.

A case is one call (or one short run of calls) through the package's public entry points:
a run of time steps from given initial data with the final state read back, a whole short
solve, one right-hand side over host arrays (the drop-in boundary), a batch of uneven solves,
a served set of requests. Sizes are those of the package's configurations, tests and
benchmark: Kelvin-Helmholtz on 32^2 and 256^2 quads, the double Mach reflection on 480x120,
four-quadrant Riemann problems, the 5x5 vortex of the smoke test, the Sedov example on Gauss
nodes, the Shu-Osher line. The initial data carry seeded noise or seeded parameters.
"""
import math
import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "p2de.jl_gb300"))

import p2de  # noqa: E402
from p2de import problems  # noqa: E402
from p2de import solver as S  # noqa: E402
from p2de.batch import Batch, Server  # noqa: E402
from p2de.workloads import build_case, Case  # noqa: E402

GAMMA = 1.4


def listed():
    return [
        # the smallest real solve of the test-suite: 25 elements, a whole time loop; launches
        # and host calls are what it costs
        dict(name="vortex5_n2_solve", kind="solve", problem="vortex", N=2, Kx=5, Ky=5, precision="fp64",
             bound="cell_entropy", intended=False, steps=0),
        # the plain small configuration: Kelvin-Helmholtz 32x32, N=3, FP64
        dict(name="kh32_n3_fp64", kind="advance", problem="kh", N=3, Kx=32, Ky=32, precision="fp64",
             bound="cell_entropy", intended=False, steps=40),
        # the large limiter-heavy configuration and the benchmark's workload
        dict(name="dmr480_n3_fp64", kind="advance", problem="dmr", N=3, Kx=480, Ky=120, precision="fp64",
             bound="cell_entropy", intended=False, steps=25),
        # the same solve in mixed precision
        dict(name="dmr480_n3_mixed", kind="advance", problem="dmr", N=3, Kx=480, Ky=120, precision="mixed",
             bound="cell_entropy", intended=False, steps=25),
        # the accurate mixed precision mode at the highest degree, the most nodes of the set
        dict(name="kh256_n5_acc64", kind="advance", problem="kh", N=5, Kx=256, Ky=256, precision="mixed-acc64",
             bound="cell_entropy", intended=False, steps=8),
        # the intended reading of the bounds, under which the limiter blends and the cell
        # entropy repair runs
        dict(name="riemann64_n4_intended", kind="advance", problem="riemann", N=4, Kx=64, Ky=64, precision="fp64",
             bound="cell_entropy", intended=True, steps=10),
        # the min-entropy bound (a bisection per contested face)
        dict(name="riemann64_n3_minentropy", kind="advance", problem="riemann", N=3, Kx=64, Ky=64, precision="fp64",
             bound="min_entropy", intended=False, steps=10),
        # the drop-in boundary: the caller owns the state on the host and asks for one
        # right-hand side (a ragged mesh that is no multiple of any block)
        dict(name="rhs97x83_n3_host", kind="rhs", problem="riemann", N=3, Kx=97, Ky=83, precision="fp64",
             bound="cell_entropy", intended=False, steps=0),
        # uneven solves advanced together: added, stepped, read back, removed
        dict(name="batch12_mixed", kind="batch", problem="riemann", N=0, Kx=0, Ky=0, precision="mixed",
             bound="cell_entropy", intended=False, steps=8, members=12, largest=96),
        # a served set of short requests from the three families
        dict(name="serve16_acc64", kind="serve", problem="mixed", N=0, Kx=0, Ky=0, precision="mixed-acc64",
             bound="cell_entropy", intended=False, steps=0, members=16, largest=64),
        # the Sedov example: Gauss nodes, scaled extrapolation, Zhang-Shu limiter
        dict(name="sedov80_n3_gauss", kind="advance", problem="sedov", N=3, Kx=80, Ky=80, precision="fp64",
             bound="zhang_shu", intended=False, steps=8),
        # the one-dimensional example at its own size
        dict(name="shu_osher64_n3", kind="advance", problem="shu_osher", N=3, Kx=64, Ky=1, precision="fp64",
             bound="positivity", intended=True, steps=60),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["advance"] * 7 + ["solve", "rhs", "batch", "serve", "line"])
    c = dict(kind=kind, problem="kh", N=rng.randint(1, 5), Kx=0, Ky=0, precision="fp64", bound="cell_entropy",
             intended=False, steps=0)
    if kind == "line":
        c.update(kind="advance", problem="shu_osher", Kx=_log_int(rng, 40, 20000), Ky=1, bound="positivity",
                 intended=True, steps=rng.randint(10, 40))
    elif kind in ("batch", "serve"):
        c.update(problem="riemann" if kind == "batch" else "mixed", N=0, members=rng.randint(3, 14),
                 largest=_log_int(rng, 24, 90), precision=rng.choice(["fp64", "mixed", "mixed-acc64"]),
                 steps=rng.randint(4, 8) if kind == "batch" else 0)
    elif kind == "solve":
        c.update(problem="vortex", Kx=rng.randint(4, 9), Ky=rng.randint(4, 9), N=rng.randint(1, 4))
    else:
        nodes = math.exp(rng.uniform(math.log(4e3), math.log(6e5)))
        kx = max(5, int(math.sqrt(nodes / (c["N"] + 1) ** 2) * rng.uniform(0.7, 1.4)))
        ky = max(5, int(nodes / (c["N"] + 1) ** 2 / kx))
        c.update(Kx=kx, Ky=ky, problem=rng.choice(["kh", "riemann", "dmr"]))
        if kind == "advance":
            c.update(steps=rng.randint(4, 12), precision=rng.choice(["fp64", "fp64", "mixed", "mixed-acc64"]))
            form = rng.choice(["plain", "plain", "intended", "gauss"])
            if form == "intended":
                # the entropy repair acts at rounding level on smooth data, so it is drawn on
                # the problem with well separated states
                c.update(problem="riemann", intended=True, precision="fp64", steps=rng.randint(3, 6))
            elif form == "gauss":
                c.update(problem="sedov", bound="zhang_shu", precision="fp64", steps=rng.randint(3, 6),
                         Kx=min(c["Kx"], 90), Ky=min(c["Ky"], 90))
    return c


# --- initial data (this file's own, so that exact() needs nothing of the package) ---------
def _conservative(rho, u, v, p):
    return np.stack([rho, rho * u, rho * v, p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)], axis=-1)


def _vortex_parameters(seed):
    r = np.random.Generator(np.random.PCG64(seed))
    return r.uniform(1.0, 5.0), r.uniform(0.0, 1.0), r.uniform(0.0, 1.0)


def _initial(problem, seed):
    """initial_condition(param, x, y) of a two-dimensional problem."""

    def condition(_param, x, y):
        r = np.random.Generator(np.random.PCG64(seed))
        if problem == "kh":  # shear layer, noise of 1e-3 on the velocity
            inner = np.abs(y - 0.5) < 0.25
            u = np.where(inner, 0.5, -0.5) + r.uniform(-1e-3, 1e-3, x.shape)
            v = 0.1 * np.sin(4 * np.pi * x) + r.uniform(-1e-3, 1e-3, x.shape)
            return _conservative(np.where(inner, 2.0, 1.0), u, v, np.full(x.shape, 2.5))
        if problem == "riemann":  # four constant states
            rho, p = r.uniform(0.1, 2.0, 4), r.uniform(0.02, 2.0, 4)
            u, v = r.uniform(-1.0, 1.0, 4), r.uniform(-1.0, 1.0, 4)
            q = np.where(x >= 0.5, np.where(y >= 0.5, 0, 3), np.where(y >= 0.5, 1, 2))
            return _conservative(rho[q], u[q], v[q], p[q])
        if problem == "dmr":  # the oblique Mach 10 shock, noise of 1e-3 on the state
            behind = (x < 1.0 / 6.0 + y / math.sqrt(3.0))[..., None]
            s = np.where(behind, _DMR_POST, _DMR_PRE)
            return s * (1.0 + 1e-3 * r.uniform(-1.0, 1.0, x.shape))[..., None]
        if problem == "vortex":
            beta, ux, uy = _vortex_parameters(seed)
            xs, ys = x - 4.5, y - 5.0
            e = np.exp(1 - xs * xs - ys * ys)
            rho = (1 - (GAMMA - 1) / (16 * GAMMA * np.pi ** 2) * (beta * e) ** 2) ** (1 / (GAMMA - 1))
            return _conservative(rho, ux - beta * e * ys / (2 * np.pi), uy + beta * e * xs / (2 * np.pi), rho ** GAMMA)
        if problem == "sedov":  # a blast at the centre of [-1.5, 1.5]^2, noise of 1e-3 on the density
            r0 = 0.15
            p = np.where(np.hypot(x, y) < r0, (GAMMA - 1) / np.pi / r0 / r0, 1e-5)
            one = 1.0 + 1e-3 * r.uniform(-1.0, 1.0, x.shape)
            return _conservative(one, 0 * x, 0 * x, p)
        raise ValueError(problem)

    return condition


_DMR_POST = _conservative(np.float64(8.0), np.float64(8.25 * math.cos(math.pi / 6)),
                          np.float64(-8.25 * math.sin(math.pi / 6)), np.float64(116.5))
_DMR_PRE = _conservative(np.float64(1.4), np.float64(0.0), np.float64(0.0), np.float64(1.0))

_T = {"kh": 0.1, "riemann": 0.2, "dmr": 0.2, "vortex": 0.02}


def _setup(case, seed):
    """initialize_DG of a case's problem: what a program does once before it steps."""
    if case["problem"] == "shu_osher":
        param, _, bc, _ = problems.shu_osher(N=case["N"], K=case["Kx"])
        phase = float(np.random.Generator(np.random.PCG64(seed)).uniform(0.0, 2 * np.pi))

        def condition(param, x):
            left = x < -4.0
            rho = np.where(left, 3.857143, 1 + 0.2 * np.sin(5 * x + phase))
            u, p = np.where(left, 2.629369, 0.0), np.where(left, 10.3333, 1.0)
            return np.stack([rho, rho * u, p / (GAMMA - 1) + 0.5 * rho * u * u], axis=-1)

        return p2de.initialize_DG(param, condition, bc), condition
    condition = _initial(case["problem"], seed)
    kw = dict(N=case["N"], Kx=case["Kx"], Ky=case["Ky"])
    if case["problem"] == "sedov":
        param, _, bc, _ = problems.sedov(**kw)
        return p2de.initialize_DG(param, condition, bc), condition
    bound = {"cell_entropy": p2de.PositivityAndCellEntropyBound, "min_entropy": p2de.PositivityAndMinEntropyBound,
             "positivity": p2de.PositivityBound}[case["bound"]]()
    make = {"kh": problems.kelvin_helmholtz, "riemann": problems.riemann2d, "dmr": problems.double_mach_reflection,
            "vortex": problems.isentropic_vortex}[case["problem"]]
    param, _, bc = make(bound=bound, precision=case["precision"], reference_semantics=not case["intended"], **kw)[:3]
    return p2de.initialize_DG(param, condition, bc), condition


def _members(case, seed):
    """The solves of a batch or of a served set: degree, mesh and family drawn from the seed
    of the sizes (not of the values), so that every seed has the same work."""
    sizes = np.random.Generator(np.random.PCG64(1000 + case["members"]))
    meshes = [max(8, case["largest"] // q) for q in (1, 2, 3, 4)]
    out = []
    for i in range(case["members"]):
        k = int(meshes[int(sizes.integers(0, 4))]) if i else case["largest"]
        if case["kind"] == "batch":
            out.append(Case("riemann", int(sizes.integers(2, 5)), k, 0.2, seed * 1000 + i))
        else:
            n = int(sizes.integers(2, 6))
            fam = ("kh", "riemann", "vortex")[i % 3]
            length = 10.0 if fam == "vortex" else 1.0
            extra = {}
            if fam == "vortex":
                beta, ux, uy = _vortex_parameters(seed * 1000 + i)
                extra = dict(strength=beta, ux=ux, uy=uy)
            # about thirty steps at the CFL step of this mesh and degree
            out.append(Case(fam, n, k, length * 1.2 / k / n ** 2, seed * 1000 + i, extra=extra))
    return out


class _State:
    pass


def prepare(case, seed):
    st = _State()
    st.case = case
    if case["kind"] in ("batch", "serve"):
        st.jobs = []
        for m in _members(case, seed):
            _, _, _, desc, U0 = build_case(m, precision=case["precision"])
            st.jobs.append((desc, U0))
        if case["kind"] == "batch":
            st.batch = Batch(2 << 30, max_solves=64, precision=case["precision"])
        else:
            st.server = Server(2 << 30, max_active=64, steps_per_tick=8, precision=case["precision"])
        return st
    (st.solver, st.state, st.state_param), condition = _setup(case, seed)
    md = st.solver.md
    st.U0 = S.evaluate_initial_condition(st.solver.param, md, condition)
    if case["kind"] == "rhs":
        st.host = p2de.HostState(st.solver, st.U0)
    return st


def run(st):
    case = st.case
    if case["kind"] == "batch":
        slots = [st.batch.add(desc, U0) for desc, U0 in st.jobs]
        st.batch.step(case["steps"])
        out = [st.batch.Uq(s) for s in slots]
        for s in slots:
            st.batch.remove(s)
        return out
    if case["kind"] == "serve":
        ids = [st.server.submit(desc, U0) for desc, U0 in st.jobs]
        states = [st.server.wait(i) for i in ids]
        return {"states": states, "Uq": [st.server.result(i) for i in ids]}
    ts = st.solver.param.timestepping_param
    if case["kind"] == "rhs":
        # L_local is filled too, but its element-boundary entries are 0 or 1 by the rounding
        # of two equal fluxes and do not reach rhsU, so they are no output to compare
        dt = p2de.rhs_bang(st.host, st.solver, st.state_param, p2de.TimeParam(0.0, ts.CFL * ts.dt0, 1))
        return {"dt": dt, "rhsU": st.host.preallocation.rhsU}
    st.solver.set_Uq(st.U0)
    if case["kind"] == "solve":
        t, steps, dt = S.ssp33(st.solver)
        return {"t": t, "steps": steps, "Uq": st.state.Uq}
    t, done = S.c_double(ts.t0), S.c_int64()
    st.solver._check(st.solver.lib.p2de_ssp33_advance(st.solver.handle, case["steps"], S.byref(t), S.byref(done)))
    return {"t": t.value, "steps": done.value, "Uq": st.state.Uq}


# --- the work of a pass ------------------------------------------------------------------
def _element_stage_flops(n):
    """Operations that one right-hand side of one element asks for (divisions, roots and
    logarithms as one each): node values, low- and high-order two-point fluxes, faces, bounds
    of the interior subcell faces, limited sums and the stage update."""
    return 75 * n * n + 24 * 2 * n * (n - 1) + 50 * 4 * n + 50 * n * n * (n - 1) + 45 * 2 * n * (n - 1)


def _solves(case):
    """(elements, nodes per line, right-hand sides) of every solve of a pass."""
    if case["kind"] in ("batch", "serve"):
        steps = case["steps"] or 30
        return [(m.K1d * m.K1d, m.N + 1, 3 * steps) for m in _members(case, 0)]
    steps = {"solve": 8, "rhs": 0}.get(case["kind"], case["steps"])
    return [(case["Kx"] * case["Ky"], case["N"] + 1, 3 * steps or 1)]


def work(case):
    byts = flops = 0
    for K, n, rhs in _solves(case):
        if case["problem"] == "shu_osher":
            byts += 2 * 24 * K * n * (rhs + 1)
            flops += K * rhs * (75 * n + 24 * n + 100 + 25 * n * (n + 3))
        else:
            # each right-hand side reads the state and writes one; plus the state in and out
            byts += 2 * 32 * K * n * n * (rhs + 1)
            flops += K * rhs * _element_stage_flops(n)
    return {"bytes": byts, "flops": flops}


# --- the same scheme in plain numpy, 64 bits ----------------------------------------------
def _gll(N):
    """LGL nodes, weights and differentiation matrix on [-1, 1]."""
    P = np.polynomial.legendre.Legendre.basis(N)
    x = np.concatenate([[-1.0], np.sort(P.deriv().roots().real), [1.0]])
    for _ in range(3):  # polish the roots of P'
        x[1:-1] -= P.deriv()(x[1:-1]) / P.deriv(2)(x[1:-1])
    x = 0.5 * (x - x[::-1])
    w = 2.0 / (N * (N + 1) * P(x) ** 2)
    n = N + 1
    c = np.array([np.prod([x[i] - x[j] for j in range(n) if j != i]) for i in range(n)])
    D = np.array([[c[i] / (c[j] * (x[i] - x[j])) if i != j else 0.0 for j in range(n)] for i in range(n)])
    np.fill_diagonal(D, -D.sum(axis=1))
    return x, w, D


def _pressure(U):
    return (GAMMA - 1) * (U[..., 3] - 0.5 * (U[..., 1] ** 2 + U[..., 2] ** 2) / U[..., 0])


def _phi(U):
    return (U[..., 3] - 0.5 * (U[..., 1] ** 2 + U[..., 2] ** 2) / U[..., 0]) * U[..., 0] ** -GAMMA


def _flux(U, d):
    p, un = _pressure(U), U[..., 1 + d] / U[..., 0]
    F = U * un[..., None]
    F[..., 1 + d] += p
    F[..., 3] += p * un
    return F


def _speed(U, d):
    r = U[..., 0]
    pe = U[..., 3] - 0.5 * U[..., 1 + d] ** 2 / r
    return np.abs(U[..., 1 + d] / r) + np.sqrt(GAMMA * (GAMMA - 1) * pe / r)


def _log_mean(a, b, la, lb):
    da, av = b - a, 0.5 * (a + b)
    f = da / av
    v = f * f
    series = av * (1 + v * (-0.2 - v * (0.0512 - v * 0.026038857142857)))
    near = np.abs(f) < 1e-4
    return np.where(near, series, -da / np.where(near, 1.0, la - lb))


def _two_point(V, i, j, d):
    """Chandrashekar's flux of line nodes i and j in direction d; V = rho, u, v, beta, log rho, log beta."""
    a, b = [q[..., i] for q in V], [q[..., j] for q in V]
    rl, bl = _log_mean(a[0], b[0], a[4], b[4]), _log_mean(a[3], b[3], a[5], b[5])
    ua, va = 0.5 * (a[1] + b[1]), 0.5 * (a[2] + b[2])
    pa = 0.5 * (a[0] + b[0]) / (a[3] + b[3])
    f4 = rl / (2 * (GAMMA - 1) * bl) + pa + 0.5 * rl * (a[1] * b[1] + a[2] * b[2])
    un = va if d else ua
    m = [rl * un, rl * un * ua, rl * un * va, f4 * un]
    m[1 + d] = m[1 + d] + pa
    return np.stack(m, axis=-1)


class _Scheme:
    """SSP-RK3 of the subcell-limited LGL scheme on a uniform mesh; U is (Ky, Kx, s, r, 4)."""

    def __init__(self, case, seed):
        self.case, N = case, case["N"]
        self.n = n = N + 1
        Kx, Ky = case["Kx"], case["Ky"]
        size = {"vortex": (10.0, 10.0), "dmr": (4.0, 1.0)}.get(case["problem"], (1.0, 1.0))
        self.h = (size[0] / Kx, size[1] / Ky)
        self.x1, self.w, self.D = _gll(N)
        self.J = self.h[0] * self.h[1] / 4
        self.g = (self.h[1] / 2, self.h[0] / 2)  # rxJ, syJ
        x = self.h[0] * np.arange(Kx)[:, None] + 0.5 * (self.x1 + 1) * self.h[0]
        y = self.h[1] * np.arange(Ky)[:, None] + 0.5 * (self.x1 + 1) * self.h[1]
        X = np.broadcast_to(x[None, :, None, :], (Ky, Kx, n, n)).reshape(Ky * Kx, n * n)
        Y = np.broadcast_to(y[:, None, :, None], (Ky, Kx, n, n)).reshape(Ky * Kx, n * n)
        self.x, self.y = x, y
        self.U = _initial(case["problem"], seed)(None, X, Y).reshape(Ky, Kx, n, n, 4)
        self.wJ = self.J * self.w[:, None] * self.w[None, :]
        if case["problem"] == "vortex":
            self.CFL, self.dt0 = 1.0, 1e-2
        else:
            self.CFL, self.dt0 = 0.5, _T[case["problem"]]
        self.T = _T[case["problem"]]

    def outside(self, U, d, t):
        """Across the low and high faces of direction d: exterior flux states, states for the
        wavespeed, and where the dissipation of the high-order flux is off; (Ky, Kx, n, 4)."""
        k = 1 - d  # axis of the elements in direction d
        node = (slice(None),) * (3 - d)  # axis of the nodes in direction d: r is axis 3, s axis 2
        low, high = U[node + (0,)], U[node + (-1,)]
        out = []
        for own, far, shift, edge in ((low, high, 1, 0), (high, low, -1, -1)):
            P = np.roll(far, shift, axis=k)
            Q, off = P.copy(), np.zeros(own.shape[:-1], bool)
            if self.case["problem"] in ("riemann", "dmr"):
                at = (slice(None),) * k + (edge,)
                Q[at] = own[at]  # a boundary face is its own neighbour
                P[at] = own[at]
                off[at] = True
                if self.case["problem"] == "dmr":
                    if d == 0 and edge == 0:
                        P[at] = _DMR_POST
                    elif d == 1 and edge == 0:
                        wall = own[at].copy()
                        wall[..., 2] *= -1
                        inflow = (self.x < 1.0 / 6.0)
                        P[at] = np.where(inflow[..., None], _DMR_POST, wall)
                        off[at] = inflow
                    elif d == 1:
                        post = self.x < 1.0 / 6.0 + (1.0 + 20.0 * t) / math.sqrt(3.0)
                        P[at] = np.where(post[..., None], _DMR_POST, _DMR_PRE)
            out.append((own, P, Q, off))
        return out

    def rhs(self, U, t, dt, first):
        """rhsU and, at the first stage, the time step of the positivity CFL condition."""
        n, w, wJ = self.n, self.w, self.wJ
        rho, p = U[..., 0], _pressure(U)
        beta = rho / (2 * p)
        V = [rho, U[..., 1] / rho, U[..., 2] / rho, beta, np.log(rho), np.log(beta)]
        lam = np.zeros(rho.shape)
        low, high = [], []
        for d in (0, 1):
            if d == 0:
                L = lambda q: q  # noqa: E731  lines along the axis before the components
            else:
                L = lambda q: np.moveaxis(q, 3, 2)  # noqa: E731
            Ud, Vd, gd = L(U), [L(q) for q in V], self.g[d]
            F, ws, lamd = _flux(Ud, d), _speed(Ud, d), L(lam)
            fl, fh = np.empty(Ud.shape[:3] + (n + 1, 4)), np.empty(Ud.shape[:3] + (n + 1, 4))
            for side, (own, P, Q, off) in enumerate(self.outside(U, d, t)):
                at, sg = -side, 1.0 if side else -1.0
                lb = 0.5 * gd * w * np.maximum(ws[..., at], _speed(Q, d))
                b = sg * 0.5 * gd * w[:, None] * (F[..., at, :] + _flux(P, d))
                lf = lb[..., None] * (P - own)
                lamd[..., at] += lb
                fl[..., at, :] = -sg * (b - lf)
                fh[..., at, :] = -sg * (b - np.where(off[..., None], 0.0, lf))
            for i in range(1, n):
                lm = 0.5 * gd * w * np.maximum(ws[..., i], ws[..., i - 1])
                fl[..., i, :] = (-0.5 * gd * w[:, None] * (F[..., i, :] + F[..., i - 1, :])
                                 + lm[..., None] * (Ud[..., i, :] - Ud[..., i - 1, :]))
                lamd[..., i] += lm
                lamd[..., i - 1] += lm
            fh[..., 1:n, :] = 0.0
            for i in range(n):
                for j in range(i):
                    s = (w[i] * self.D[i, j] - w[j] * self.D[j, i]) * gd
                    f = (s * w)[:, None] * _two_point(Vd, i, j, d)
                    fh[..., j + 1:i + 1, :] += f[..., None, :]
            low.append(fl)
            high.append(fh)
        # the dissipation enters with the sign of the face-flux convention: fbar[i+1] - fbar[i]
        step = None
        if first:
            step = min(min(self.CFL * self.dt0, self.T - t), float((self.CFL * 0.5 * wJ / lam).min()))
        turn = lambda q: np.moveaxis(q, 2, 3)  # noqa: E731  y lines back to (s, r)
        diff = lambda fx, fy: (np.diff(fx, axis=3) + turn(np.diff(fy, axis=3))) / wJ[..., None]  # noqa: E731
        uL = U + dt * diff(low[0], low[1])
        floor = self.entropy_floor(U, t) if self.case["bound"] == "min_entropy" else None
        factors = [self.factors(*((q if d == 0 or q is None else np.moveaxis(q, 3, 2)) for q in (uL, floor)),
                                low[d], high[d], dt) for d in (0, 1)]
        if self.case["bound"] == "cell_entropy":
            for d in (0, 1):
                self.entropy(U, low[d], high[d], factors[d], d)
        for d in (0, 1):  # one factor per element face
            l, k = factors[d], 1 - d
            lo, hi = l[..., 0].copy(), l[..., -1].copy()
            a, b = np.minimum(lo, np.roll(hi, 1, axis=k)), np.minimum(hi, np.roll(lo, -1, axis=k))
            if self.case["problem"] in ("riemann", "dmr"):
                a[(slice(None),) * k + (0,)] = lo[(slice(None),) * k + (0,)]
                b[(slice(None),) * k + (-1,)] = hi[(slice(None),) * k + (-1,)]
            l[..., 0], l[..., -1] = a, b
        f = [low[d] + factors[d][..., None] * (high[d] - low[d]) for d in (0, 1)]
        return diff(f[0], f[1]), step

    def entropy_floor(self, U, t):
        """The smallest rho e rho^-gamma of a node and its four neighbours, across faces too."""
        phi = _phi(U)
        least = phi.copy()
        for d in (0, 1):
            node = (slice(None),) * (3 - d)
            inner = [node + (slice(1, None),), node + (slice(None, -1),)]
            least[inner[0]] = np.minimum(least[inner[0]], phi[inner[1]])
            least[inner[1]] = np.minimum(least[inner[1]], phi[inner[0]])
            for at, (_, _, Q, _) in zip((0, -1), self.outside(U, d, t)):
                least[node + (at,)] = np.minimum(least[node + (at,)], _phi(Q))
        return least

    def factors(self, uL, floor, fl, fh, dt):
        """Bound factors of the subcell faces of one direction."""
        n = self.n
        l = np.ones(fl.shape[:-1])
        q = 4 * dt / self.wJ
        lower = uL[..., 0] * 0.1
        lower_e = 0.1 * (uL[..., 3] - 0.5 * (uL[..., 1] ** 2 + uL[..., 2] ** 2) / uL[..., 0])
        upper = 0.0 if not self.case["intended"] and floor is None else np.inf
        df = fh - fl
        with np.errstate(all="ignore"):
            for h in (0, 1):
                P = (df[..., h:n + h, :] * q[..., None]) * (1.0 if h else -1.0)
                up = uL[..., 0] + P[..., 0]
                a = np.where(up < lower, np.maximum((lower - uL[..., 0]) / P[..., 0], 0.0), 1.0)
                b = np.where(up > upper, np.maximum((upper - uL[..., 0]) / P[..., 0], 0.0), 1.0)
                b = np.where((P[..., 0] == 0) & (up > upper), np.where(np.signbit(P[..., 0]), 1.0, 0.0), b)
                v = np.minimum(np.minimum(a, b), 1.0)
                A = P[..., 0] * P[..., 3] - 0.5 * (P[..., 1] ** 2 + P[..., 2] ** 2)
                B = (uL[..., 3] * P[..., 0] + uL[..., 0] * P[..., 3] - uL[..., 1] * P[..., 1]
                     - uL[..., 2] * P[..., 2] - P[..., 0] * lower_e)
                C = uL[..., 3] * uL[..., 0] - 0.5 * (uL[..., 1] ** 2 + uL[..., 2] ** 2) - uL[..., 0] * lower_e
                disc = B * B - 4 * A * C
                s = np.sqrt(np.maximum(disc, 0.0))
                r1, r2 = (-B + s) / (2 * A), (-B - s) / (2 * A)
                e = 5e-16
                root = np.where((r1 > e) & (r2 > e), np.minimum(r1, r2),
                                np.where((r1 > e) & (r2 < -e), r1, np.where((r2 > e) & (r1 < -e), r2, 1.0)))
                v = np.minimum(v, np.where((disc >= 0) & np.isfinite(root), root, 1.0))
                if floor is not None:  # the largest factor of 21 halvings that keeps the floor
                    bad = np.nonzero(~(_phi(uL + v[..., None] * P) >= floor - 1e-14))
                    u, P, least = uL[bad], P[bad], floor[bad] - 1e-14
                    good, over = np.zeros(least.shape), v[bad]
                    for _ in range(21):
                        mid = 0.5 * (good + over)
                        ok = _phi(u + mid[:, None] * P) >= least
                        good, over = np.where(ok, mid, good), np.where(ok, over, mid)
                    v[bad] = good
                l[..., h:n + h] = np.minimum(l[..., h:n + h], v)
        return l

    def entropy(self, U, fl, fh, l, d):
        """The cell entropy repair of one direction, on the interior factors in place."""
        n = self.n
        p = _pressure(U)
        s = np.log(p) - GAMMA * np.log(U[..., 0])
        v = np.stack([GAMMA + 1 - s - (GAMMA - 1) * U[..., 3] / p, U[..., 1] * (GAMMA - 1) / p,
                      U[..., 2] * (GAMMA - 1) / p, -U[..., 0] * (GAMMA - 1) / p], axis=-1)
        psi = (GAMMA - 1) * U[..., 1 + d]
        if d:
            v, psi = np.moveaxis(v, 3, 2), np.moveaxis(psi, 3, 2)
        sB = (self.g[d] * self.w * (psi[..., -1] - psi[..., 0])).sum(-1)
        dv = v[..., :-1, :] - v[..., 1:, :]
        i_l, i_h = fl[..., 1:n, :], fh[..., 1:n, :]
        dvdf = (dv * (i_h - i_l)).sum(-1)
        sdl = (dv * i_l).sum((-1, -2, -3))
        lin = l[..., 1:n]
        # face numbers of the reference's order: x faces along the line first, y faces across it
        ix = np.arange(n * (n - 1)).reshape(n, n - 1) if d == 0 else np.arange(n * (n - 1)).reshape(n - 1, n).T
        total = (lin * dvdf).sum((-1, -2))
        target, tol = sB - sdl, np.maximum(0.0, sdl - sB)
        back = np.argsort(ix.ravel())  # flattened (line, face) places in the order of the numbers
        for ky, kx in np.argwhere(total - target > tol):
            df, ll = dvdf[ky, kx].ravel()[back], lin[ky, kx].ravel()[back]
            order = sorted(range(df.size), key=lambda q: (df[q], q), reverse=True)
            left, goal, used = total[ky, kx], target[ky, kx] + tol[ky, kx], []
            for q in order:
                if not left > goal or df[q] < 5e-16:
                    break
                left -= ll[q] * df[q]
                used.append(q)
            for i, q in enumerate(used):
                ll[q] = min(ll[q], max((goal - left) / df[q], 0.0) if i == len(used) - 1 else 0.0)
            put = np.empty_like(ll)
            put[back] = ll
            lin[ky, kx] = put.reshape(lin.shape[2:])

    def advance(self, steps):
        t, U, done = 0.0, self.U, 0
        while t < self.T and (steps is None or done < steps):
            dt = min(self.CFL * self.dt0, self.T - t)
            R, dt = self.rhs(U, t, dt, True)
            V = U + dt * R
            V = 0.75 * U + 0.25 * (V + dt * self.rhs(V, t, dt, False)[0])
            U = U / 3 + 2 / 3 * (V + dt * self.rhs(V, t, dt, False)[0])
            t, done = t + dt, done + 1
        return t, done, U


def exact(case, seed):
    """run() of the two-dimensional LGL solves in plain numpy. None for the largest ones and
    the batches (minutes of numpy), and for the Gauss and line solves, which are other schemes."""
    K, n, rhs = _solves(case)[0]
    if (case["kind"] not in ("advance", "solve", "rhs") or case["bound"] not in ("cell_entropy", "min_entropy")
            or K * n * n * (n + 2) * rhs > 3.2e7):
        return None
    s = _Scheme(case, seed)
    if case["kind"] == "rhs":
        R, dt = s.rhs(s.U, 0.0, s.CFL * s.dt0, True)
        return {"dt": dt, "rhsU": R.reshape(K, n * n, 4)}
    t, done, U = s.advance(None if case["kind"] == "solve" else case["steps"])
    return {"t": t, "steps": done, "Uq": U.reshape(K, n * n, 4)}
