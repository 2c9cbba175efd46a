"""Workloads of the time-step engine, measured through its public entry points.

One pass is a span of steps from a given state to its read-out, the unit a
user's program works in:

* call "span": the state goes up through page-locked host buffers, the span
  runs on the device and the state comes back (Context.step_host_inner), as a
  driver does between two output steps or restarts.
* call "loop": Solver.load_state, one Solver.step per time step (a driver
  that looks at dt after each one, as the C++ drop-in does), then
  Solver.field of the state.

Grids are the repository's own families: the curvilinear periodic box, the
tiled slab between a Solid_Surface and a Farfield, the spherical shell with
Pole patches, and sweeps of independent shells or slabs in one batch.  The
physics options are ideal MHD, the implicit resistive solve, the explicit
resistive sub-cycles and the implicit Hall solve; FP64 or the mixed form;
forward Euler or SSP-RK2.
"""
import functools
import math

import numpy as np
import torch

from beta1_b200 import case as case_mod
from beta1_b200 import mhd, physics, solver

FIELDS = ("U_H", "B_xi", "B_eta", "B_zeta")
RES_PEAK = 1e-3  # peak of the resistive shell profile, in units of U L (the slab workload's)


def listed():
    return [
        # a correctness-size box stepped one call at a time: launches and call latency only
        dict(name="box_tiny", kind="box", ni=12, nj=10, nk=9, mode="ideal", integrator="euler", precision="fp64",
             call="loop", steps=20),
        # the 64^3 curvilinear block with SSP-RK2, the smallest of the benchmark's configurations
        dict(name="box_64_rk2", kind="box", ni=64, nj=64, nk=64, mode="ideal", integrator="rk2", precision="fp64",
             call="span", steps=100),
        # a box of odd sizes in mixed precision
        dict(name="box_odd_mixed", kind="box", ni=101, nj=67, nk=83, mode="ideal", integrator="euler",
             precision="mixed", call="span", steps=100),
        # four small slab blocks with walls, far field and block interfaces, stepped one call at a time
        dict(name="slab_small", kind="slab", nr=16, nj=8, nk=8, tj=2, tk=2, mode="ideal", precision="fp64",
             call="loop", steps=50),
        # the six-block slab with the implicit resistive solve in every step
        dict(name="slab_implicit", kind="slab", nr=80, nj=40, nk=40, tj=3, tk=2, mode="implicit", precision="fp64",
             call="span", steps=100),
        # ragged slab blocks with the explicit resistive sub-cycles
        dict(name="slab_explicit", kind="slab", nr=57, nj=27, nk=31, tj=2, tk=2, mode="explicit", precision="fp64",
             call="span", steps=100),
        # one spherical shell with Poles, FP64
        dict(name="shell_fp64", kind="shell", nr=96, nth=64, nph=64, mode="ideal", precision="fp64", call="span",
             steps=100),
        # a small shell with the explicit resistive sub-cycles, stepped one call at a time
        dict(name="shell_resistive", kind="shell", nr=33, nth=25, nph=26, mode="explicit", precision="fp64",
             call="loop", steps=50),
        # a parameter sweep of shells in one batch, mixed precision: the benchmark's default workload on fewer runs
        dict(name="sweep_shell_mixed", kind="sweep", grid="shell", runs=6, draws=5, mode="ideal", precision="mixed",
             call="span", steps=100),
        # the same kind of sweep on slab blocks, FP64, other draws
        dict(name="sweep_slab_fp64", kind="sweep", grid="slab", runs=3, draws=11, mode="ideal", precision="fp64",
             call="span", steps=100),
        # Hall MHD on the six-block slab, half the benchmark's size per direction, the implicit solve in every step
        dict(name="hall_slab", kind="slab", nr=64, nj=32, nk=32, tj=3, tk=2, mode="hall", precision="fp64",
             call="span", steps=20),
        # a small ragged Hall slab in a mixed-precision context
        dict(name="hall_small_mixed", kind="slab", nr=37, nj=21, nk=25, tj=2, tk=1, mode="hall", precision="mixed",
             call="span", steps=20),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """A case of the listed ranges: sizes from the correctness tests' to the
    benchmark configurations', odd and even alike."""
    kind = rng.choice(("box", "slab", "slab", "shell", "sweep", "hall"))
    precision = rng.choice(("fp64", "mixed"))
    call = rng.choice(("span", "span", "loop"))
    steps = rng.randint(20, 100)
    if kind == "box":
        return dict(kind="box", ni=_log_int(rng, 8, 100), nj=_log_int(rng, 8, 100), nk=_log_int(rng, 8, 100),
                    mode="ideal", integrator=rng.choice(("euler", "rk2")), precision=precision, call=call, steps=steps)
    if kind == "shell":
        return dict(kind="shell", nr=_log_int(rng, 16, 96), nth=_log_int(rng, 12, 64),
                    nph=2 * _log_int(rng, 6, 32), mode=rng.choice(("ideal", "explicit")), precision=precision,
                    call=call, steps=steps)
    if kind == "sweep":
        return dict(kind="sweep", grid=rng.choice(("shell", "slab")), runs=rng.randint(2, 3),
                    draws=rng.randint(1, 1000), mode="ideal", precision=precision, call="span", steps=steps)
    tj, tk = rng.choice(((1, 1), (2, 1), (2, 2), (3, 2)))
    if kind == "hall":
        return dict(kind="slab", nr=_log_int(rng, 24, 64), nj=_log_int(rng, 8, 32), nk=_log_int(rng, 8, 32), tj=tj,
                    tk=tk, mode="hall", precision=precision, call="span", steps=rng.randint(4, 20))
    return dict(kind="slab", nr=_log_int(rng, 16, 96), nj=_log_int(rng, 8, 48), nk=_log_int(rng, 8, 48), tj=tj, tk=tk,
                mode=rng.choice(("ideal", "implicit", "explicit")), precision=precision, call=call, steps=steps)


# --------------------------------------------------------------------------
# what a program has in hand before the call
# --------------------------------------------------------------------------

@functools.lru_cache(maxsize=2)
def _plan(key):
    """Grid and parameters of a case (and a sweep's compiled tables): they
    depend on the case alone, not on the state."""
    c = dict(key)
    if c["kind"] == "box":
        return case_mod.periodic_box_case((c["ni"], c["nj"], c["nk"])), "periodic", None
    over = {}
    if c["mode"] in ("implicit", "explicit"):
        sc = case_mod.ref_scales()
        over = dict(is_Lunar_resistance=1, use_implicit_lunar_resistance=int(c["mode"] == "implicit"),
                    eta_max_lunar=RES_PEAK * case_mod.MU0 * sc["U"] * sc["L_ref"], implicit_resistive_ksp_rtol=1e-10,
                    n_resistive_subcycles=2)
    if c["kind"] == "slab":
        return case_mod.slab_case(c["nr"], (c["nj"], c["nk"]), (c["tj"], c["tk"]), **over), "tiled", None
    if c["kind"] == "shell":
        return case_mod.shell_case(c["nr"], c["nth"], c["nph"], **over), "shell", None
    topo = "shell" if c["grid"] == "shell" else "tiled"
    runs = [(spec, topo) for spec, _ in case_mod.sweep_cases(c["runs"], seed=c["draws"], grid=c["grid"])]
    return runs, topo, [solver.host_setup(spec, topo, "device") for spec, topo in runs]


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


def _state_of(case, spec, seed):
    if case["kind"] == "box":
        return case_mod.initial_state(spec, seed=seed)
    return case_mod.inflow_state(spec, seed=seed)


def _inner(fa):
    """the inner points of a restart array (its ghost layers are -lo deep on both sides)"""
    g = [-x for x in fa.lo]
    return fa.data[g[0]:fa.data.shape[0] - g[0], g[1]:fa.data.shape[1] - g[1], g[2]:fa.data.shape[2] - g[2]]


class _Span:
    """a context with its page-locked state buffers"""

    def __init__(self, engine, states, steps):
        self.engine, self.ctx, self.steps = engine, engine.ctx, steps
        self.loop = False
        parts, self.names, self.shapes = [], [], []
        for st in states:
            for b in range(len(st.fields["U_H"].blocks)):
                for f in FIELDS:
                    a = _inner(st.fields[f].blocks[b])
                    self.names.append("%s_%02d" % (f, len(self.names) // len(FIELDS)))
                    self.shapes.append(a.shape)
                    parts.append(a.reshape(-1))
        n = sum(p.size for p in parts)
        self.src = torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()
        self.dst = torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()
        np.concatenate(parts, out=self.src)


class _Loop:
    """a solver and the restart state it starts from"""

    def __init__(self, engine, state, steps):
        self.engine, self.state, self.steps = engine, state, steps
        self.loop = True
        self.nblocks = len(engine.spec.blocks)


def prepare(case, seed):
    """The solver (geometry, boundary tables, solve set-up) and a state of
    the seed in host memory: page-locked for a span."""
    plan, topo, host = _plan(_key(case))
    precision = mhd.PREC_MIXED if case["precision"] == "mixed" else mhd.PREC_FP64
    if case["kind"] == "sweep":
        eng = solver.Batch(plan, precision=precision, host=iter(host))
        return _Span(eng, [_state_of(case, spec, 100 * seed + r) for r, (spec, _) in enumerate(plan)], case["steps"])
    eng = solver.Solver(plan, topology=topo, precision=precision, geometry_on="device")
    if case["mode"] == "hall":
        eng.install_hall_implicit(topo, rtol=1e-10, maxit=10, ksp_rtol=1e-5, ksp_maxit=200)
    if case.get("integrator") == "rk2":
        eng.ctx.set_integrator(mhd.INTEGRATOR_SSPRK2)
    st = _state_of(case, plan, seed)
    return _Loop(eng, st, case["steps"]) if case["call"] == "loop" else _Span(eng, [st], case["steps"])


def run(state):
    """One span of steps and the state after it: U_H and the face B of every
    block, and the last step's dt."""
    if state.loop:
        s = state.engine
        s.load_state(state.state)
        for _ in range(state.steps):
            dt, _ = s.step()
        out = {"%s_%02d" % (f, b): s.field(f, b) for b in range(state.nblocks) for f in FIELDS}
        out["dt"] = dt
        return out
    dt = state.ctx.step_host_inner(state.steps, state.src, state.dst)
    out, off = {}, 0
    for name, shape in zip(state.names, state.shapes):
        n = math.prod(shape)
        out[name] = state.dst[off:off + n].reshape(shape)
        off += n
    out["dt"] = dt
    return out


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------

def _cells(case):
    if case["kind"] == "box":
        return case["ni"] * case["nj"] * case["nk"]
    if case["kind"] == "slab":
        return case["nr"] * case["nj"] * case["nk"] * case["tj"] * case["tk"]
    if case["kind"] == "shell":
        return case["nr"] * case["nth"] * case["nph"]
    total = 0
    for spec, _ in case_mod.sweep_cases(case["runs"], seed=case["draws"], grid=case["grid"]):
        total += sum(b.ncell[0] * b.ncell[1] * b.ncell[2] for b in spec.blocks)
    return total


def work(case):
    """Per stage and cell: the state (5 fluid components, 3 face fluxes) read
    and written once, and the grid's metric read once: face vectors 9,
    volume, applied field 3, face and edge ratios 6, and the reconstruction
    weights of B (18) and J (36), in 4 bytes each in the mixed form.  The
    explicit sub-cycles read and write B and read its metric once more each;
    a Hall step evaluates its residual once per Krylov iteration and Newton
    step (12 at these tolerances), each reading B, the two ratio sets, the
    weights and the edge vectors and writing the edge field."""
    cells = _cells(case)
    w = 4 if case["precision"] == "mixed" else 8
    stage = (2 * 8 + 9 + 1 + 3 + 6) * 8 + 54 * w
    flops = 900
    if case["mode"] == "explicit":
        stage += 2 * ((2 * 3 + 6 + 3 + 9) * 8 + 54 * w)
        flops += 2 * 250
    if case["mode"] == "hall":
        stage += 12 * ((3 + 6 + 3 + 6 + 9 + 3 + 3) * 8 + 54 * 8)
        flops += 12 * 500
    stages = case["steps"] * (2 if case.get("integrator") == "rk2" else 1)
    return {"bytes": stages * cells * stage + 2 * 8 * 8 * cells, "flops": stages * cells * flops}


# --------------------------------------------------------------------------
# the periodic box in plain numpy
# --------------------------------------------------------------------------

def exact(case, seed):
    """The periodic box's steps in 64-bit numpy on one period (faces and
    edges of index n are those of index 0); None for the bounded grids, whose
    wall, far-field and Pole rules and solves would be a second solver, and
    for boxes that would take too long."""
    if case["kind"] != "box":
        return None
    stages = case["steps"] * (2 if case["integrator"] == "rk2" else 1)
    if stages * _cells(case) > 2.5e6:
        return None
    spec = case_mod.periodic_box_case((case["ni"], case["nj"], case["nk"]))
    st = case_mod.initial_state(spec, seed=seed)
    n = (case["ni"], case["nj"], case["nk"])
    U = np.moveaxis(_inner(st.fields["U_H"].blocks[0]), -1, 0).copy()
    B = [_inner(st.fields[f].blocks[0])[:n[0], :n[1], :n[2], 0].copy() for f in FIELDS[1:]]
    box = _PeriodicBox(spec)
    for _ in range(case["steps"]):
        dt = box.time_step(U, B)
        U1, B1 = box.euler(U, B, dt)
        if case["integrator"] == "rk2":
            U2, B2 = box.euler(U1, B1, dt)
            U1, B1 = 0.5 * (U + U2), [0.5 * (a + b) for a, b in zip(B, B2)]
        U, B = U1, B1
    out = {"dt": dt}
    for f, a, plus in [("U_H", U, (0, 0, 0))] + [(f, a[None], tuple(int(i == d) for i in range(3)))
                                                 for d, (f, a) in enumerate(zip(FIELDS[1:], B))]:
        g = 4 if case["call"] == "loop" else 0
        a = np.pad(a, [(0, 0)] + [(g, g + p) for p in plus], mode="wrap")
        out[f + "_00"] = np.moveaxis(a, 0, -1)
    return out


class _PeriodicBox:
    """Finite-volume constrained-transport MHD on the periodic map
    x = xi + a sin 2 pi eta (and cyclic); vectors are arrays of shape
    (3, ni, nj, nk), index 0 of a face or edge axis at the cell's low side."""

    def __init__(self, spec, amp=0.05):
        self.c = physics.constants(spec.params)
        n = spec.blocks[0].ncell
        # nodes -1 .. n + 1 of the map, so that all of a cell's neighbours' nodes are there
        x = np.meshgrid(*[np.arange(-1, m + 3) / m for m in n], indexing="ij")
        P = np.stack([x[d] + amp * np.sin(2.0 * np.pi * x[(d + 1) % 3]) for d in range(3)])
        self.n = n

        def at(A, di, dj, dk):
            return A[:, 1 + di:1 + di + n[0], 1 + dj:1 + dj + n[1], 1 + dk:1 + dk + n[2]]

        def step(d, s):
            v = [0, 0, 0]
            v[d] = s
            return v

        def add(*vs):
            return [sum(q) for q in zip(*vs)]

        def cross(a, b):
            return np.cross(a, b, axis=0)

        def norm(a):
            return np.sqrt((a * a).sum(0))

        centre = sum(P[:, i:P.shape[1] - 1 + i, j:P.shape[2] - 1 + j, k:P.shape[3] - 1 + k]
                     for i in (0, 1) for j in (0, 1) for k in (0, 1)) / 8.0  # of the cell above each node
        xc = at(centre, 0, 0, 0)
        o = [0, 0, 0]
        self.S, face_c, self.beta, self.alpha, edge = [], [], [], [], []
        for d in range(3):
            a, b = step((d + 1) % 3, 1), step((d + 2) % 3, 1)
            p0, pa, pb, pab = (at(P, *v) for v in (o, a, b, add(a, b)))
            self.S.append(0.5 * (cross(pa - p0, pb - p0) + cross(pb - pab, pa - pab)))
            face_c.append((p0 + pa + pb + pab) / 4.0)
            self.beta.append(norm(xc - at(centre, *step(d, -1))) / norm(self.S[d]))
            a, b = step((d + 1) % 3, -1), step((d + 2) % 3, -1)
            c00, c10, c01, c11 = (at(centre, *v) for v in (add(a, b), b, a, o))
            dual = 0.5 * (cross(c10 - c00, c01 - c00) + cross(c01 - c11, c10 - c11))
            edge.append(at(P, *step(d, 1)) - p0)
            self.alpha.append(norm(edge[d]) / norm(dual))
        # the six outward faces and twelve edges of a cell, with the least-squares maps
        # from face fluxes to B and from edge circulations to J
        faces, dist, vol = [], [], 0.0
        for d in range(3):
            for side in (0, 1):
                S, f = self.S[d], face_c[d]
                if side:
                    S = np.roll(S, -1, 1 + d)
                    a, b = step((d + 1) % 3, 1), step((d + 2) % 3, 1)
                    h = step(d, 1)
                    f = sum(at(P, *add(h, v)) for v in (o, a, b, add(a, b))) / 4.0
                S = S if side else -S
                vol = vol + (S * (f - xc)).sum(0) / 3.0
                faces.append(S)
                dist.append(norm(f - xc))
        self.vol = vol
        self.edge_rolls = [[(a, b) for b in (0, 1) for a in (0, 1)] for _ in range(3)]
        edges = [self._corner(edge[d], d, a, b) for d in range(3) for a, b in self.edge_rolls[d]]
        self.WB = self._least_squares(faces, [1.0 / q for q in dist])
        self.WJ = self._least_squares(edges, [np.ones(n)] * 12)

    @staticmethod
    def _corner(a, d, s1, s2):
        """an edge array of direction d at the cell's corner (s1, s2) of the other two axes"""
        axes = [a.ndim - 3 + (d + 1) % 3, a.ndim - 3 + (d + 2) % 3]
        return np.roll(a, (-s1, -s2), axes)

    @staticmethod
    def _least_squares(S, mu):
        S, mu = np.stack(S), np.stack(mu)
        M = np.einsum("fxijk,fyijk,fijk->ijkxy", S, S, mu)
        return np.einsum("ijkxy,fyijk,fijk->fxijk", np.linalg.inv(M), S, mu)

    def fields(self, U, B):
        """cell B, edge and cell J, velocity and pressure"""
        flux = []
        for d in range(3):
            flux += [-B[d], np.roll(B[d], -1, d)]
        Bc = np.einsum("fxijk,fijk->xijk", self.WB, np.stack(flux))
        h = [self.beta[d] * B[d] for d in range(3)]
        J = []
        for d in range(3):
            p, q = (d + 1) % 3, (d + 2) % 3  # circulation of the dual face around the edge
            J.append((np.roll(h[p], 1, q) - h[p] + h[q] - np.roll(h[q], 1, p)) * self.alpha[d])
        Jc = np.einsum("fxijk,fijk->xijk", self.WJ,
                       np.stack([self._corner(J[d], d, a, b) for d in range(3) for a, b in self.edge_rolls[d]]))
        rho = np.maximum(U[0], 1e-12)
        V = U[1:4] / rho
        p = np.maximum((self.c["gamma"] - 1.0) * np.maximum(U[4] - 0.5 * rho * (V * V).sum(0), 0.0), 1e-12)
        return Bc, Jc, V, p

    def time_step(self, U, B):
        c, g = self.c, self.c["gamma"]
        Bc = self.fields(U, B)[0]
        rho = np.maximum(U[0], 1e-2)
        V = U[1:4] / rho
        cs2 = g * (g - 1.0) * (U[4] - 0.5 * rho * (V * V).sum(0)) / rho
        va2 = c["inver_MA2"] * (Bc * Bc).sum(0) / rho
        total = 0.0
        for d in range(3):
            for S in (self.S[d], np.roll(self.S[d], -1, 1 + d)):
                A = np.sqrt((S * S).sum(0))
                un, bn = (V * S).sum(0) / A, (Bc * S).sum(0) / A
                t = cs2 + va2
                root = np.sqrt(np.maximum(t * t - 4.0 * cs2 * c["inver_MA2"] * bn * bn / rho, 0.0))
                total = total + (np.abs(un) + np.sqrt(0.5 * (t + root))) * A
        return float((c["cfl"] * self.vol / total).min())

    def euler(self, U, B, dt):
        c, g = self.c, self.c["gamma"]
        Bc, Jc, V, p = self.fields(U, B)
        rho = U[0]
        E = p / (g - 1.0) + 0.5 * rho * (V * V).sum(0)
        Q = np.concatenate([rho[None], rho * V, E[None]])
        cs = np.sqrt(g * p / rho)
        rhs = np.zeros_like(U)
        for d in range(3):
            S = self.S[d]
            A = np.sqrt((S * S).sum(0))

            def one(R):
                q, v, pr, s = (np.roll(a, 1, a.ndim - 3 + d) if R == 0 else a for a in (Q, V, p, cs))
                un = (S * v).sum(0)
                f = q * un
                f[1:4] += S * pr
                f[4] += un * pr
                return q, f, np.abs(un) + s * A

            (qL, fL, rL), (qR, fR, rR) = one(0), one(1)
            F = 0.5 * (fL + fR) - 0.5 * np.maximum(rL, rR) * (qR - qL)
            rhs -= (np.roll(F, -1, 1 + d) - F) / self.vol
        nt = rho / c["M_H"] * c["M_ref"]
        fc = c["momentum_hall_coeff"] * nt / np.sqrt(nt * nt + c["ne_hall_floor"] ** 2)
        jxb = np.cross(Jc, Bc, axis=0)
        rhs[1:4] += fc * jxb
        rhs[4] += fc * (jxb * V).sum(0)
        # contravariant velocities, face EMF (Rusanov on both transverse fluxes), edge EMF
        W = [(0.5 * (self.S[d] + np.roll(self.S[d], -1, 1 + d)) * V).sum(0) / self.vol for d in range(3)]
        Bm = [0.5 * (B[d] + np.roll(B[d], -1, d)) for d in range(3)]

        def transport(f, b):
            """flux of component b through the faces of direction f"""
            L = lambda a: np.roll(a, 1, f)  # noqa: E731
            GL, GR = L(W[f]) * L(Bm[b]) - L(W[b]) * B[f], W[f] * Bm[b] - W[b] * B[f]
            r = np.maximum(np.abs(L(W[f])), np.abs(W[f]))
            return 0.5 * (GL + GR) - 0.5 * r * (Bm[b] - L(Bm[b]))

        Ee = []
        for d in range(3):
            p1, q1 = (d + 1) % 3, (d + 2) % 3
            e1, e2 = -transport(p1, q1), transport(q1, p1)  # on the faces normal to p1 and to q1
            mean = 0.25 * (e1 + np.roll(e1, 1, q1) + e2 + np.roll(e2, 1, p1))

            def peak(a):
                a = np.maximum(np.abs(a), np.abs(np.roll(a, 1, p1)))
                return np.maximum(a, np.roll(a, 1, q1))

            Ee.append(mean + 0.25 * (peak(W[p1]) * (B[q1] - np.roll(B[q1], 1, p1))
                                     - peak(W[q1]) * (B[p1] - np.roll(B[p1], 1, q1))))
        Bn = []
        for d in range(3):
            p1, q1 = (d + 1) % 3, (d + 2) % 3
            curl = Ee[p1] - np.roll(Ee[p1], -1, q1) + np.roll(Ee[q1], -1, p1) - Ee[q1]
            Bn.append(B[d] - dt * curl)
        return U + dt * rhs, Bn
