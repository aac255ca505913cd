"""The solver's work as its users have it done, as cases that can be timed.

A case is one call sequence of a program that holds a solver (or a batch of
them) and has new inputs for it: a power map solved to steady state, a sweep of
power maps, a backward-Euler run, a batch of uneven stacks, or the one-call
form that also builds and frees the solver. Sizes and stacks are those of the
benchmark's workloads, the tests and the reference's grid-convergence table
(64 x 64 to 1024 x 1024 columns, 7 to 20 planes).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-thermal_gb300"))
import cthermal as ct  # noqa: E402

PRECISION = {"fp64": ct.Precision.MG_FP64, "fp32": ct.Precision.MG_FP32, "flex": ct.Precision.MG_FP32_FLEX,
             "dw": ct.Precision.MG_FP32_FLEX_DW}
DIE = 10e-3  # m, the die's x extent
H_TOP = 2e4  # W/(m^2 K), the heat sink
TSV_K, TSV_RHO_C = 400.0, 3.45e6  # copper
# name, thickness (m), k (W/(m K)), rho c (J/(m^3 K))
SI = ("Si", 50e-6, 130.0, 1.66e6)
BOND = ("bond", 10e-6, 2.0, 1.70e6)
TIM = ("TIM", 25e-6, 5.0, 2.00e6)
CU = ("Cu", 1e-3, 400.0, 3.45e6)
TOL_STEADY, TOL_STEP, MAXIT = 1e-10, 1e-9, 1000
DT0, GROWTH, DT_MAX = 1e-5, 1.1, 0.05  # the transient driver's step sizes


def listed():
    return [
        # an interactive floorplan tool's coarse preview: one map in, one field out, latency is all
        dict(name="steady_64", kind="steady", io="host", nx=64, ny=64, tiers=2, si=2, tsv=False, precision="flex", maps=1),
        # a script's one call: solver built, solved and freed (the coarsest grid of the convergence table)
        dict(name="oneshot_200", kind="oneshot", nx=200, ny=200, tiers=2, si=2, tsv=False, precision="flex"),
        # a three-tier stack with TSV arrays on an off-grid die: odd sizes, partial tiles
        dict(name="steady_237x181_tsv", kind="steady", io="host", nx=237, ny=181, tiers=3, si=2, tsv=True, precision="flex", maps=1),
        # the plain double-precision solve that other answers are checked with
        dict(name="steady_400_fp64", kind="steady", io="device", nx=400, ny=400, tiers=2, si=2, tsv=False, precision="fp64", maps=1),
        # the reference's default build (float V-cycle, Fletcher-Reeves) on an odd grid
        dict(name="steady_501x333_fp32", kind="steady", io="device", nx=501, ny=333, tiers=2, si=2, tsv=False, precision="fp32", maps=1),
        # the headline: the 12.5 um grid, power map and field on the device
        dict(name="steady_800", kind="steady", io="device", nx=800, ny=800, tiers=2, si=2, tsv=False, precision="flex", maps=1),
        # the same end to end: a sweep of host power maps with queued copies
        dict(name="sweep_800", kind="steady", io="queued", nx=800, ny=800, tiers=2, si=2, tsv=False, precision="flex", maps=3),
        # the largest single stack: four tiers, TSV blocks in the bond layers
        dict(name="four_tier_1024", kind="steady", io="device", nx=1024, ny=1024, tiers=4, si=2, tsv=True, precision="flex", maps=1),
        # the double-word outer iteration
        dict(name="steady_640_dw", kind="steady", io="device", nx=640, ny=640, tiers=2, si=2, tsv=False, precision="dw", maps=1),
        # backward Euler from a cold stack: queued steps, warm starts, few iterations each
        dict(name="transient_400", kind="transient", nx=400, ny=400, tiers=2, si=2, tsv=False, precision="flex", steps=12),
        # a floorplan sweep: uneven stacks solved together
        dict(name="batch_48", kind="batch", count=48, lo=64, hi=512, mix=4, precision="flex"),
        # many stacks stepped together, blocks switching on and off (the batch's default precision)
        dict(name="batch_transient_16", kind="batch_transient", count=16, nx=256, ny=256, tiers=2, si=2, steps=6, precision="dw"),
    ]


def draw(rng):
    """One more case of the listed ranges."""
    def logsize(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["steady", "steady", "steady", "steady", "oneshot", "transient", "batch", "batch_transient"])
    c = dict(kind=kind, tiers=rng.randint(1, 4), si=rng.choice([1, 2, 2, 3]), tsv=rng.random() < 0.3,
             precision=rng.choice(["flex", "flex", "flex", "fp32", "fp64", "dw"]))
    if kind == "steady":
        c["io"] = rng.choice(["host", "device", "queued"])
        c["maps"] = rng.randint(2, 3) if c["io"] == "queued" else 1
        hi = 1024 if c["precision"] != "fp64" and c["maps"] == 1 else 640
        c["nx"] = logsize(48, hi)
        c["ny"] = max(48, min(hi, int(c["nx"] * rng.uniform(0.6, 1.6))))
    elif kind == "oneshot":
        c["nx"], c["ny"] = logsize(48, 400), logsize(48, 400)
    elif kind == "transient":
        c["nx"], c["ny"], c["steps"] = logsize(64, 600), logsize(64, 600), rng.randint(4, 12)
        c["precision"] = rng.choice(["flex", "flex", "fp64", "dw"])
    elif kind == "batch":
        c = dict(kind=kind, count=rng.randint(6, 40), lo=rng.choice([32, 64]), hi=rng.choice([256, 384, 512]),
                 mix=rng.randint(5, 10**6), precision=rng.choice(["flex", "dw"]))
    else:
        c["nx"], c["ny"] = logsize(96, 320), logsize(96, 320)
        c["count"], c["steps"], c["tsv"] = rng.randint(4, 16), rng.randint(3, 6), False
        c["precision"] = rng.choice(["flex", "dw"])
    return c


# ---- inputs --------------------------------------------------------------------

class Stack:
    """Layers, grid, floorplan and TSV regions of one stack."""

    def __init__(self, nx, ny, tiers, si, tsv, rng, cu=4):
        self.nx, self.ny = nx, ny
        self.layers = []  # (spec, planes, active)
        for t in range(tiers):
            self.layers.append((SI, si, True))
            if t + 1 < tiers:
                self.layers.append((BOND, 1, False))
        self.layers += [(TIM, 1, False), (CU, cu, False)]
        self.dx = DIE / nx
        self.Lx, self.Ly = DIE, self.dx * ny
        self.plane_layer = [k for k, (_, n, _) in enumerate(self.layers) for _ in range(n)]
        self.nz = len(self.plane_layer)
        self.cells = nx * ny * self.nz
        self.tsvs = []  # (layer, i0, j0, cells x, cells y, fraction)
        if tsv:
            for k, (spec, _, _) in enumerate(self.layers):
                if spec is BOND or (tiers == 1 and spec is TIM):
                    for _ in range(24):
                        w, h = int(rng.integers(4, 17)), int(rng.integers(4, 17))
                        self.tsvs.append((k, int(rng.integers(0, nx - w)), int(rng.integers(0, ny - h)), w, h,
                                          float(rng.choice([0.1, 0.25, 1.0]))))

    def power(self, rng, blocks=12, on=None):
        """A power map (nz, ny, nx) in W: 25 W per 10 x 10 mm Si tier, a third
        of it uniform and the rest in rectangular blocks of log-normal density."""
        P = np.zeros((self.nz, self.ny, self.nx))
        watts = 25.0 * self.Ly / DIE
        for k, (_, n, active) in enumerate(self.layers):
            if not active:
                continue
            plane = np.zeros((self.ny, self.nx))
            for b in range(blocks):
                w, h = (max(1, int(s * rng.uniform(0.05, 0.3))) for s in (self.nx, self.ny))
                i, j = int(rng.integers(0, self.nx - w + 1)), int(rng.integers(0, self.ny - h + 1))
                dens = math.exp(0.6 * rng.standard_normal())
                if on is None or on[b % len(on)]:
                    plane[j:j + h, i:i + w] += dens
            total = plane.sum()
            if total > 0:
                plane *= 2 / 3 * watts / total
            plane += watts / 3 / plane.size
            for l in range(self.nz):
                if self.plane_layer[l] == k:
                    P[l] = plane / n
        return P

    def spec(self):
        cs = ct.CaseSpec(layers=[ct.Layer(s[0], s[1], s[2], s[3], n, a) for s, n, a in self.layers],
                         Lx=self.Lx, Ly=self.Ly, h_top=H_TOP, h_bot=0.0)
        cs.tsvs = [ct.TsvRegion(k, i * self.dx, j * self.dx, w * self.dx, h * self.dx, f)
                   for k, i, j, w, h, f in self.tsvs]
        return cs

    def model(self, P):
        m = ct.build_case_model(self.spec(), self.nx, self.ny)
        m.P[:] = P.reshape(-1)
        return m


def _stack(case, rng):
    return Stack(case["nx"], case["ny"], case["tiers"], case["si"], case.get("tsv", False), rng)


def _batch_stacks(case):
    """Uneven stacks: sides a multiple of 32 columns apart, 6 to 16 planes. The
    case says which (`mix`); the power maps are the inputs."""
    rng, out = np.random.default_rng(case["mix"]), []
    for _ in range(case["count"]):
        nx, ny = (int(rng.choice(np.arange(case["lo"], case["hi"] + 1, 32))) for _ in range(2))
        planes = int(rng.integers(6, 17))
        si = int(rng.integers(1, 3))
        tiers = max(1, min(4, (planes - 1) // (si + 1)))
        cu = max(1, planes - (tiers * (si + 1) - 1) - 1)
        out.append(Stack(nx, ny, tiers, si, False, rng, cu=cu))
    return out


def _dts(case):
    return [min(DT0 * GROWTH ** k, DT_MAX) for k in range(case["steps"])]


def _switching(case, rng):
    """For each instance and step, whether its blocks switch before the step
    (every instance once before the first) and the step's dt (restarted then)."""
    changed = [[s == 0 or rng.random() < 0.2 for s in range(case["steps"])] for _ in range(case["count"])]
    dts = np.zeros((case["steps"], case["count"]))
    for i in range(case["count"]):
        dt = DT0
        for s in range(case["steps"]):
            if changed[i][s]:
                dt = DT0
            dts[s, i] = dt
            dt = min(dt * GROWTH, DT_MAX)
    return changed, dts


def _inputs(case, seed):
    """Everything that the seed decides, on the host."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "batch":
        stacks = _batch_stacks(case)
        return dict(stacks=stacks, P=[s.power(rng) for s in stacks])
    s = _stack(case, rng)
    if kind == "batch_transient":
        changed, dts = _switching(case, rng)
        maps = [[s.power(rng, 9, rng.random(9) < 0.5) if c else None for c in row] for row in changed]
        return dict(stack=s, dts=dts, maps=maps)
    return dict(stack=s, P=[s.power(rng) for _ in range(case.get("maps", 1))])


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _pinned_copy(a):
    p = _pinned(a.size)
    p[:] = a.reshape(-1)
    return p


def prepare(case, seed):
    kind, prec = case["kind"], PRECISION[case["precision"]]
    inp = _inputs(case, seed)
    st = dict(case=case)
    if kind == "batch":
        stacks = inp["stacks"]
        st["batch"] = ct.GpuBatch.from_specs([s.spec() for s in stacks], [s.nx for s in stacks],
                                             [s.ny for s in stacks], precision=prec)
        st["P"] = [torch.from_numpy(p.reshape(-1)).cuda() for p in inp["P"]]
        st["T"] = _pinned(sum(s.cells for s in stacks))
        st["at"] = np.cumsum([0] + [s.cells for s in stacks])
        return st
    s = inp["stack"]
    if kind == "batch_transient":
        n = case["count"]
        st["batch"] = ct.GpuBatch.from_specs([s.spec()] * n, [s.nx] * n, [s.ny] * n, precision=prec)
        st["maps"] = [[None if p is None else _pinned_copy(p) for p in row] for row in inp["maps"]]
        st["dts"] = inp["dts"]
        st["T"] = _pinned(n * s.cells)
        st["at"] = np.arange(n + 1) * s.cells
        return st
    if kind == "oneshot":
        st["model"] = s.model(inp["P"][0])
        return st
    st["solver"] = ct.GpuPcg.from_spec(s.spec(), s.nx, s.ny, precision=prec)
    if kind == "transient":
        st["P"] = torch.from_numpy(inp["P"][0].reshape(-1)).cuda()
    elif case["io"] == "device":
        st["P"] = [torch.from_numpy(p.reshape(-1)).cuda() for p in inp["P"]]
    else:
        st["P"] = [_pinned_copy(p) for p in inp["P"]]
        st["T"] = [_pinned(s.cells) for _ in inp["P"]]
    return st


# ---- passes --------------------------------------------------------------------

class _DeviceArray:
    """A solver's device field as an array that torch reads in place; it holds
    the solver, so that the memory lives as long as a tensor over it does."""

    def __init__(self, solver):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": (solver.n,), "typestr": "<f8", "data": (solver.device_x(), False),
                                         "strides": None, "version": 2}


def _field(solver):
    return torch.as_tensor(_DeviceArray(solver), device="cuda")


def run(state):
    return {"steady": _run_steady, "oneshot": _run_oneshot, "transient": _run_transient, "batch": _run_batch,
            "batch_transient": _run_batch_transient}[state["case"]["kind"]](state)


def _run_steady(st):
    s, io = st["solver"], st["case"]["io"]
    if io == "queued":
        for P, T in zip(st["P"], st["T"]):
            s.set_power_async(P)
            s.set_x_zero()
            s.set_rhs_steady()
            s.solve_async(TOL_STEADY, MAXIT)
            s.get_x_async(T)
        s.copies_wait()
        return {"T": list(st["T"]), "iters": s.solve_wait().iters}
    if io == "host":
        s.set_power(st["P"][0])
    else:
        s.set_power_device(st["P"][0].data_ptr())
    s.set_x_zero()
    s.set_rhs_steady()
    iters = s.solve(TOL_STEADY, MAXIT).iters
    return {"T": [s.get_x(st["T"][0]) if io == "host" else _field(s)], "iters": iters}


def _run_oneshot(st):
    r = ct.gpu_pcg(st["model"], TOL_STEADY, MAXIT, precision=PRECISION[st["case"]["precision"]])
    return {"T": [r.T], "iters": r.iters}


def _run_transient(st):
    s, dts = st["solver"], _dts(st["case"])
    s.set_power_device(st["P"].data_ptr())
    s.set_x_zero()
    for k, dt in enumerate(dts):
        s.set_dt(dt)
        s.set_rhs_transient()
        s.solve_async(TOL_STEP, MAXIT)
        s.step_record_async(dt, k)
    recs, stats = s.step_records(0, len(dts))
    return {"T": _field(s), "records": np.array([(r.T_max, r.q_out, r.q_stored) for r in recs]),
            "iters": np.array([x.iters for x in stats])}


def _run_batch(st):
    b, at = st["batch"], st["at"]
    for i, P in enumerate(st["P"]):
        b.set_power_device(i, P.data_ptr())
    b.set_x_zero()
    b.set_rhs_steady()
    stats = b.solve(TOL_STEADY, MAXIT)
    for i in range(len(b)):
        b.get_x(i, st["T"][at[i]:at[i + 1]])
    return {"T": st["T"], "iters": np.array([x.iters for x in stats])}


def _run_batch_transient(st):
    b, at, dts = st["batch"], st["at"], st["dts"]
    b.set_x_zero()
    recs, iters = [], []
    for k in range(len(dts)):
        for i, row in enumerate(st["maps"]):
            if row[k] is not None:
                b.set_power(i, row[k])
        iters.append([x.iters for x in b.step_transient(dts[k], TOL_STEP, MAXIT)])
        recs.append(b.step_records(dts[k]))
    for i in range(len(b)):
        b.get_x(i, st["T"][at[i]:at[i + 1]])
    return {"T": st["T"], "records": np.array(recs), "iters": np.array(iters)}


# ---- what a pass cannot do without -----------------------------------------------

def work(case):
    """Bytes: the power maps, the operator (three faces and a capacity of four
    bytes a cell) and the fields, once each. Flops: about 120 a cell and PCG
    iteration (operator 14, vectors 10, V-cycle 4/3 of four line-solve sweeps
    and a restriction), with the iterations the method takes (13 from zero, 4 a
    warm-started step)."""
    if case["kind"] == "batch":
        side = (case["lo"] + case["hi"]) / 2
        cells, solves, iters = case["count"] * side * side * 11, 1, 13
    else:
        cells = case["nx"] * case["ny"] * (case["tiers"] * (case["si"] + 1) + 4)
        solves, iters = case.get("maps", 1), 13
        if "steps" in case:
            solves, iters = case["steps"], 4
        cells *= case.get("count", 1)
    fields = solves if "steps" not in case else 1
    return {"bytes": cells * (16.0 + 16.0 * fields), "flops": 120.0 * cells * iters * solves}


# ---- the same answers in 64 bits ---------------------------------------------------

class _Operator:
    """The stack's conductances (double formulas, stored in float as the model
    keeps them), and a solve in double: flexible PCG on (A + C/dt), with the
    plane averages' operator inverted in cosine modes as the preconditioner."""

    def __init__(self, s):
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        nx, ny, nz, d = s.nx, s.ny, s.nz, s.dx
        f = torch.zeros((nz, ny, nx), dtype=torch.float64, device=dev)
        for k, i, j, w, h, frac in s.tsvs:
            for l in range(nz):
                if s.plane_layer[l] == k:
                    f[l, j:j + h, i:i + w] = torch.clamp(f[l, j:j + h, i:i + w] + frac, max=1.0)

        def per_plane(v):
            return torch.tensor(v, dtype=torch.float64, device=dev).view(nz, 1, 1)

        lay = [s.layers[k] for k in s.plane_layer]
        k0, rc = per_plane([x[0][2] for x in lay]), per_plane([x[0][3] for x in lay])
        dz = per_plane([x[0][1] / x[1] for x in lay])
        kxy = k0 * ((1 + f) * TSV_K + (1 - f) * k0) / ((1 - f) * TSV_K + (1 + f) * k0)
        kz = f * TSV_K + (1 - f) * k0
        dy = s.Ly / ny
        A = d * dy

        def stored(t):
            return t.float().double()

        self.gE = stored(dy * dz / (d / (2 * kxy[:, :, :-1]) + d / (2 * kxy[:, :, 1:])))
        self.gN = stored(d * dz / (dy / (2 * kxy[:, :-1]) + dy / (2 * kxy[:, 1:])))
        half = dz / (2 * kz)
        r_up = half.clone()
        r_up[:-1] += half[1:]
        r_up[-1] += 1.0 / H_TOP
        self.gU = stored(A / r_up)
        self.cap = stored((f * TSV_RHO_C + (1 - f) * rc) * A * dz)
        self.face = self.gU.clone()
        self.face[1:] += self.gU[:-1]
        self.face[:, :, :-1] += self.gE
        self.face[:, :, 1:] += self.gE
        self.face[:, :-1] += self.gN
        self.face[:, 1:] += self.gN

        def cosines(n):
            k, i = torch.arange(n, dtype=torch.float64, device=dev), torch.arange(n, dtype=torch.float64, device=dev)
            c = torch.cos(math.pi * k.view(-1, 1) * (i + 0.5) / n) * math.sqrt(2.0 / n)
            c[0] /= math.sqrt(2.0)
            return c.float(), (2 - 2 * torch.cos(math.pi * k / n))

        self.cx, lx = cosines(nx)
        self.cy, ly = cosines(ny)
        mean = lambda t: t.mean(dim=(1, 2)).view(nz, 1, 1)  # noqa: E731
        self.modes = mean(self.gE) * lx.view(1, 1, nx) + mean(self.gN) * ly.view(1, ny, 1)
        self.gu, self.capm = mean(self.gU), mean(self.cap)
        self.nz, self.dev = nz, dev

    def apply(self, x, inv_dt):
        y = (self.face + inv_dt * self.cap) * x
        y[:, :, :-1] -= self.gE * x[:, :, 1:]
        y[:, :, 1:] -= self.gE * x[:, :, :-1]
        y[:, :-1] -= self.gN * x[:, 1:]
        y[:, 1:] -= self.gN * x[:, :-1]
        y[:-1] -= self.gU[:-1] * x[1:]
        y[1:] -= self.gU[:-1] * x[:-1]
        return y

    def modes_solve(self, r, inv_dt):
        scale = float(r.abs().max()) or 1.0
        v = self.cy @ ((r / scale).float() @ self.cx.T)
        diag = self.modes + self.gu + inv_dt * self.capm
        diag[1:] += self.gu[:-1]
        cp, x = [], []
        for l in range(self.nz):
            low = self.gu[l - 1] if l else 0.0
            den = diag[l] + (low * cp[-1] if l else 0.0)
            cp.append(-self.gu[l] / den)
            x.append((v[l] + (low * x[-1] if l else 0.0)) / den)
        for l in range(self.nz - 2, -1, -1):
            x[l] = x[l] - cp[l] * x[l + 1]
        return (self.cy.T @ (torch.stack(x).float() @ self.cx)).double() * scale

    def solve(self, b, inv_dt=0.0):
        x = torch.zeros_like(b)
        bb = float(b.norm())
        for _ in range(6):
            r = b - self.apply(x, inv_dt)
            r0 = float(r.norm())
            if r0 <= 1e-14 * bb:
                break
            p = ap = None
            for _ in range(200):
                z = self.modes_solve(r, inv_dt)
                p = z if p is None else z - (z * ap).sum() / (p * ap).sum() * p
                ap = self.apply(p, inv_dt)
                alpha = (p * r).sum() / (p * ap).sum()
                x += alpha * p
                r -= alpha * ap
                if float(r.norm()) < 1e-9 * r0:
                    break
        return x

    def record(self, x, old, dt):
        return [float(x.max()), float((self.gU[-1] * x[-1]).sum()), float((self.cap * (x - old)).sum()) / dt]


def exact(case, seed):
    inp = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        T = []
        for s, P in zip(inp["stacks"], inp["P"]):
            op = _Operator(s)
            T.append(op.solve(torch.from_numpy(P).to(op.dev)).cpu().numpy().reshape(-1))
        return {"T": np.concatenate(T), "iters": None}
    op = _Operator(inp["stack"])
    zero = torch.zeros_like(op.cap)
    if kind == "batch_transient":
        T, recs = [], np.zeros(inp["dts"].shape + (3,))
        for i, row in enumerate(inp["maps"]):
            x = zero
            for k, P in enumerate(row):
                power = torch.from_numpy(P).to(op.dev) if P is not None else power
                dt, old = float(inp["dts"][k, i]), x
                x = op.solve(power + op.cap / dt * old, 1.0 / dt)
                recs[k, i] = op.record(x, old, dt)
            T.append(x.cpu().numpy().reshape(-1))
        return {"T": np.concatenate(T), "records": recs, "iters": None}
    maps = [torch.from_numpy(P).to(op.dev) for P in inp["P"]]
    if kind == "transient":
        x, recs = zero, []
        for dt in _dts(case):
            old = x
            x = op.solve(maps[0] + op.cap / dt * old, 1.0 / dt)
            recs.append(op.record(x, old, dt))
        return {"T": x.reshape(-1), "records": np.array(recs), "iters": None}
    return {"T": [op.solve(P).reshape(-1).cpu().numpy() for P in maps], "iters": None}
