"""The measured work of the solver, through its public entry points.

A case is one thing that a program using this package does over and over:

* `step`: one physical step (`Solver.step`, a fixed number of inner
  iterations; 10 is the default and the count of the 64^3 workload) and the
  read-back of the new level into the program's pinned buffer
  (`Solver.q_into`), as a host loop that writes or analyses every level does.
  Flat channel, wavy-wall channel (3-D metrics) or the open configuration
  (inflow / outflow, sponges, heated wall, buoyancy); FP64 or mixed
  precision; LU-SGS or DP-LUR; with the previous level or the network as
  initial guess (then from one common point of a run, as guesses are
  compared); optionally with the running statistics of each step;
* `train`: Adam steps of the network on stored levels, and its weights;
* `filter`: the filter sensor of a level, host arrays in and out.

`exact` is the same work in plain 64-bit torch, written from the equations.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cgli_fu_flow_b200 import channel as C

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def listed() -> list[dict]:
    def step(name, nx, ny, nz, grid="flat", precision="fp64", inner="lusgs", predictor=0, stats=False, iters=10):
        return dict(name=name, kind="step", nx=nx, ny=ny, nz=nz, grid=grid, precision=precision, inner=inner,
                    predictor=predictor, stats=stats, iters=iters)

    return [
        # the smallest channel of the tests: launches and latency
        step("step_8x12x8", 8, 12, 8),
        # the plain-method workload: 64^3, ten inner iterations a step
        step("step_64x64x64", 64, 64, 64),
        # the scale workload and benchmark, the largest state here
        step("step_256x192x192", 256, 192, 192),
        # no dimension a multiple of a tile, a warp or a vector
        step("step_ragged_91x53x75", 91, 53, 75),
        # mixed precision on the profiling grid of the channel
        step("mixed_160x128x128", 160, 128, 128, precision="mixed"),
        # mixed precision on the wavy-wall grid (half the 256x256x128 workload per direction)
        step("wavy_mixed_128x128x64", 128, 128, 64, grid="wavy", precision="mixed"),
        # the same grid in FP64 at the size of a parameter study
        step("wavy_64x64x32", 64, 64, 32, grid="wavy"),
        # the open production configuration with its per-step statistics
        step("open_stats_128x96x96", 128, 96, 96, grid="open", stats=True),
        # the alternative inner solver
        step("dplur_128x96x96", 128, 96, 96, inner="dplur"),
        # the network as initial guess, step after step from one common point
        # of a run (how guesses are compared)
        step("learned_64x64x64", 64, 64, 64, precision="mixed", predictor=2),
        # training it on stored levels
        dict(name="train_64x64x64", kind="train", nx=64, ny=64, nz=64, iters=4),
        # the filter sensor of one level
        dict(name="filter_96x72x72", kind="filter", nx=96, ny=72, nz=72),
    ]


def draw(rng) -> dict:
    """One more case: cells spread over their logarithm from the smallest to
    the largest listed, the three directions within a factor of about two of
    each other, odd sizes as often as even ones."""
    kind = rng.choice(["flat"] * 4 + ["mixed"] * 3 + ["wavy"] * 2 + ["open"] * 2 + ["dplur", "learned", "train", "filter"])
    largest = {"flat": 256 * 192 * 192, "mixed": 192 * 160 * 160}.get(kind, 128 * 112 * 112)
    n = math.exp(rng.uniform(math.log(8 * 12 * 8), math.log(largest))) ** (1 / 3)
    if kind == "wavy":   # the wall's two waves need some cells
        n = max(n, 30 + 4 * rng.random())
    nx, ny, nz = (max(least, round(n * rng.uniform(lo, hi)))
                  for least, lo, hi in ((8, 0.9, 1.3), (12, 0.75, 1.05), (8, 0.7, 1.05)))
    if kind in ("learned", "train"):   # the network's own grid rule
        ny, nz = max(12, ny // 4 * 4), max(32, nz // 32 * 32)
    if kind in ("train", "filter"):
        c = dict(kind=kind, nx=nx, ny=ny, nz=nz)
        return dict(c, iters=rng.randint(1, 6)) if kind == "train" else c
    return dict(kind="step", nx=nx, ny=ny, nz=nz, grid=kind if kind in ("wavy", "open") else "flat",
                precision="mixed" if kind in ("mixed", "learned") or (kind == "wavy" and rng.random() < 0.5) else "fp64",
                inner="dplur" if kind == "dplur" else "lusgs", predictor=2 if kind == "learned" else 0,
                stats=rng.random() < 0.3, iters=rng.randint(7, 10) if n > 24 else 10)


def _channel(case: dict) -> C.Channel:
    dims = case["nx"], case["ny"], case["nz"]
    grid = case.get("grid", "flat")
    if grid == "wavy":
        return C.Channel(*dims, wavy=True, wave=C.WAVY["c4"])
    if grid == "open":   # the sponges' share of the slab and the wall temperature of the o2 workload
        nin, nout = C.OPEN["o2"]
        o2 = C.WORKLOADS["o2"][0]
        return C.Channel(*dims, x_open=True, nx_inlet=max(1, case["nx"] * nin // o2),
                         nx_outlet=max(1, case["nx"] * nout // o2), buoyancy=True, twall_lo=343.0592)
    return C.Channel(*dims)


def _noise(ch: C.Channel, seed: int, fields: int) -> torch.Tensor:
    """Uniform on [-1, 1), zero mean over each wall-parallel plane."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    r = 2 * torch.rand((fields, ch.nx, ch.ny, ch.nz), generator=g, dtype=torch.float32).to(DEVICE).double() - 1
    return r - r.mean(dim=(1, 3), keepdim=True)


def _field(ch: C.Channel, seed: int) -> torch.Tensor:
    """Conserved variables (5, nx, ny, nz): the laminar profile with velocity
    perturbations of 10 % of the bulk velocity, uniform density and pressure."""
    y = torch.from_numpy(ch.cell_y()).to(DEVICE)
    vel = 0.1 * ch.u_b * _noise(ch, seed, 3)
    lam = 1.5 * ch.u_b * (1 - (y / ch.h - 1) ** 2)
    vel[0] += lam[None, :, None]
    if ch.wavy:
        vel[1] += (lam[None, :] * torch.from_numpy(ch.line_slope()).to(DEVICE))[:, :, None]
    rho = torch.full_like(vel[0], ch.rho0)
    energy = C.P0 / (C.GAMMA - 1) + 0.5 * rho * (vel * vel).sum(0)
    return torch.cat([rho[None], rho * vel, energy[None]])


def _scales(ch: C.Channel):
    """Input and output scales of the network for a run of this channel: the
    bulk quantities' spread, a step's change of about one part in nx of it."""
    ru = ch.rho0 * ch.u_b
    mean = np.array([ch.rho0, 0.9 * ru, 0, 0, C.P0 / (C.GAMMA - 1)])
    std = np.array([0.01 * ch.rho0, 0.5 * ru, 0.05 * ru, 0.05 * ru, 0.5 * ru * ch.u_b])
    return mean, std, std / ch.nx, std / ch.nx / 4, std / ch.nx / 20


def _theta(seed: int) -> np.ndarray:
    """Network weights (He-uniform hidden layers, a small output layer)."""
    g = np.random.default_rng(seed + 7)
    parts = []
    for ci, co in zip((15, 32, 32, 32, 32), (32, 32, 32, 32, 5)):
        lim = math.sqrt((6.0 if co == 32 else 0.3) / (27 * ci))
        parts += [g.uniform(-lim, lim, 27 * co * ci), g.uniform(-0.05, 0.05, co)]
    return np.concatenate(parts).astype(np.float32)


def _levels(ch: C.Channel, seed: int) -> list[np.ndarray]:
    """Consecutive levels of a smoothly changing flow, for training."""
    q, r = _field(ch, seed), 0.1 * _noise(ch, seed + 3, 5)
    amp = torch.tensor([0.01 * ch.rho0] + [ch.rho0 * ch.u_b] * 3 + [0.01 * C.P0], dtype=torch.float64, device=DEVICE)
    out = []
    for k in range(6):
        d = amp[:, None, None, None] * (math.sin(0.3 * k) * r + 0.05 * math.cos(k) * r.roll(1, 1))
        out.append((q + d).float().cpu().numpy())
    return out


def prepare(case: dict, seed: int) -> dict:
    from cgli_fu_flow_b200.cnn import Network, scales_from_levels
    from cgli_fu_flow_b200.solver import FP64, MIXED, Solver
    ch = _channel(case)
    if case["kind"] == "train":
        net = Network(ch.nx, ch.ny, ch.nz)
        net.set_params(_theta(seed))
        levels = _levels(ch, seed)
        net.set_scales(*scales_from_levels(levels))
        net.reserve_levels(len(levels))
        for q in levels:
            net.push_level_host(q)
        return dict(case=case, net=net)
    sol = Solver(ch, MIXED if case.get("precision") == "mixed" else FP64)
    sol.init(_field(ch, seed).cpu().numpy())
    if case["kind"] == "filter":
        return dict(case=case, sol=sol, y=ch.y_point())
    sol.set_inner_solver(case["inner"])
    state = dict(case=case, sol=sol)
    if case["predictor"] == 2:
        net = Network(ch.nx, ch.ny, ch.nz)
        net.set_params(_theta(seed))
        net.set_scales(*_scales(ch))
        sol.set_learned_guess(net)
        sol.set_predictor(2)
        state["net"] = net
        for _ in range(2):   # two levels of history: the network's inputs
            sol.step(case["iters"])
        state["point"] = Solver(ch, MIXED)
        state["point"].copy_state_from(sol)
    out = torch.empty((5,) + ch.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    state["host"] = out.numpy()
    state["q"] = out[:, 3:ch.nx + 3, 2:ch.ny + 2, 2:ch.nz + 2]
    return state


def run(state: dict):
    case = state["case"]
    if case["kind"] == "train":
        loss = state["net"].train(case["iters"], 1e-3, 1, 0, 3)
        return {"loss": np.float32(loss), "theta": state["net"].get_params()}
    sol = state["sol"]
    if case["kind"] == "filter":
        return sol.filter(state["y"], 0.3, 0.1, 0.01)
    if "point" in state:
        sol.copy_state_from(state["point"])
    sol.step(case["iters"])
    out = {"q": state["q"]}
    if case["stats"]:
        sol.accumulate_statistics()
        out["stats"] = sol.statistics()[0]
    sol.q_into(state["host"])
    return out


def work(case: dict) -> dict:
    cells = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "train":
        # forward, input gradient and weight gradient of the five layers; the
        # weights and the four levels of a pair
        conv = 2 * 27 * (15 * 32 + 3 * 32 * 32 + 32 * 5)
        return {"bytes": case["iters"] * cells * 4 * 5 * 4, "flops": case["iters"] * cells * 3 * conv}
    if case["kind"] == "filter":
        # four variables of U_, Y_point and J in, three face arrays out; two
        # scales of six levels, about 14 operations a variable and level
        return {"bytes": cells * 8 * (4 + 2 + 3), "flops": cells * 2 * 6 * 4 * 14}
    # the three levels of the step read and written once; the operations of
    # an inner iteration: three Roe fluxes, the viscous terms, the residual,
    # the implicit passes and the update
    flops = cells * case["iters"] * 2 * (968 + 330 + 260 + 4 * 88 + 62)
    if case["predictor"] == 2:
        flops += cells * 2 * 27 * (15 * 32 + 3 * 32 * 32 + 32 * 5)
    return {"bytes": cells * 8 * 5 * (3 + 3), "flops": flops}


# --------------------------------------------------------------- exact values
def exact(case: dict, seed: int):
    ch = _channel(case)
    if ch.cells > 3_000_000:   # more than about 20 s in plain torch
        return None
    with torch.no_grad():
        if case["kind"] == "train":
            return _exact_train(case, ch, seed)
        slab = _Slab(ch, _field(ch, seed))
        if case["kind"] == "filter":
            return [t.cpu().numpy() for t in _exact_filter(ch, slab, 0.3, 0.1, 0.01)]
        correct = None
        if case["predictor"] == 2:
            layers = _layers(torch.from_numpy(_theta(seed)).to(DEVICE).double())
            scales = [torch.from_numpy(s).to(DEVICE)[:, None, None, None] for s in _scales(ch)]
            correct = lambda q0, q1, q2: _correction(layers, scales, q0, q1, q2)   # noqa: E731
            for order in (0, 1):
                slab.step(case["iters"], case["inner"], order)
        slab.step(case["iters"], case["inner"], 2 if correct else 0, correct)
        out = {"q": slab.U_[:, 3:ch.nx + 3, 2:ch.ny + 2, 2:ch.nz + 2]}
        if case["stats"]:
            out["stats"] = slab.statistics()
        return out


class _Slab:
    """The solver's step on one slab in plain torch, arrays in the layout
    [nx+6][ny+4][nz+4] (three x ghosts, two y and z ghosts)."""
    K, R, CV = 1.4, 287.0, 717.5

    def __init__(self, ch: C.Channel, q: torch.Tensor):
        self.ch = ch
        self.X, self.Y, self.Z = ch.shape
        self.ie, self.jn, self.kn = ch.nx + 2, ch.ny + 1, ch.nz + 1
        self.d = (ch.dxi, ch.det, ch.dzt)
        f64 = dict(dtype=torch.float64, device=DEVICE)
        i, j = torch.arange(self.X, **f64), torch.arange(self.Y, **f64)
        self.cell = self._metric((i - 2.5) * ch.dxi, (j - 1.5) * ch.det)
        for m in self.cell:   # wall ghost rows repeat the wall cells
            m[:, 1], m[:, self.jn + 1] = m[:, 2], m[:, self.jn]
        # the faces between cell n and n + 1 of each direction
        fy = self._metric((i - 2.5) * ch.dxi, (j - 1.0) * ch.det)
        for m, c in zip(fy, self.cell):
            # (the wall faces take the ghost cell's metric, one plane back)
            m[1:, 1], m[1:, self.jn] = c[:-1, 1], c[:-1, self.jn]
        self.face = (self._metric((i - 2.0) * ch.dxi, (j - 1.5) * ch.det), fy, self.cell)
        self.J = self.cell[0][:, :, None]
        self.force, self.integral = ch.force_lam, 0.0
        quiet = torch.tensor([101300 / 298.0592 / self.R, 0, 0, 0, 101300 / (self.K - 1)], **f64)
        lo, hi = (2, self.ie + 2) if ch.x_open else (3, self.ie + 1)
        self.U = torch.zeros((5,) + ch.shape, **f64)
        self.U[:, lo:hi] = quiet[:, None, None, None] / self.J[lo:hi]
        self.inner = (slice(None), slice(3, self.ie + 1), slice(2, self.jn + 1), slice(2, self.kn + 1))
        self.U[self.inner] = q / self.J[3:self.ie + 1, 2:self.jn + 1]
        self.Uq, self.Uqq, self.U_ = self.U.clone(), self.U.clone(), self.U.clone()
        self._planes()

    def _metric(self, x, eta):
        """(J, eta_x, eta_y) at the given positions; xi_x = zeta_z = 1, the rest 0."""
        ch, g = self.ch, C.STRETCH
        kx = 4 * math.pi / (ch.nx * ch.dxi)
        s = g * (1 - 2 * eta)
        y0 = 0.5 * ch.high * (1 - torch.tanh(s) / math.tanh(g))
        y0p = ch.high * g / math.tanh(g) / torch.cosh(s) ** 2
        yw, ywp = ch.amplitude * torch.sin(kx * x)[:, None], ch.amplitude * kx * torch.cos(kx * x)[:, None]
        y_eta = (ch.high - yw) * y0p / ch.high
        return [1 / y_eta, -ywp * (1 - y0 / ch.high) / y_eta, 1 / y_eta]

    def _planes(self):
        """Interior cells sorted by hyperplane i + j + k, and each one's six
        neighbours in that order; then the x halo (ny nz entries), then a zero."""
        nx, ny, nz = self.ch.nx, self.ch.ny, self.ch.nz
        n, halo = nx * ny * nz, ny * nz
        c = torch.arange(n, device=DEVICE)
        i, j, k = c // halo, c // nz % ny, c % nz
        self.order = torch.argsort(i + j + k, stable=True)
        self.count = torch.bincount(i + j + k).tolist()
        place = torch.empty_like(c)
        place[self.order] = c
        hx, zero = n + j * nz + k, torch.full_like(c, n + halo)

        def at(ok, shift, other):
            return torch.where(ok, place[(c + shift).clamp(0, n - 1)], other)[self.order]

        self.low = [at(i > 0, -halo, hx), at(j > 0, -nz, zero), at(k > 0, -1, zero)]
        self.high = [at(i < nx - 1, halo, hx), at(j < ny - 1, nz, zero), at(k < nz - 1, 1, zero)]

    def prim(self, q, J):
        u = q[1:4] / q[0]
        rho, VV = q[0] * J, (u * u).sum(0)
        P = (q[4] * J - 0.5 * rho * VV) * (self.K - 1)
        return rho, u, VV, P

    # ---------------------------------------------------- halos and walls
    def boundaries(self):
        ch, q, ie, jn, kn = self.ch, self.U_, self.ie, self.jn, self.kn
        if not ch.x_open:
            q[:, ie + 1:ie + 4], q[:, 0:3] = q[:, 3:6].clone(), q[:, ie - 2:ie + 1].clone()
        for js, jg, T in ((2, 1, ch.twall_lo), (jn, jn + 1, ch.twall_hi)):
            sl = slice(3, ie + 1), js, slice(2, kn + 1)
            c, J = q[(slice(None),) + sl], self.J[3:ie + 1, js]
            rho, u, VV, P = self.prim(c, J)
            rw = P / self.R / T
            wall = torch.stack([rw, *(-rw * u), P / (self.K - 1) + 0.5 * rw * VV]) / J
            i = torch.arange(3, ie + 1, device=DEVICE)
            heated = ((i > ch.nx_inlet + 2) & (i < ch.nx - ch.nx_outlet + 3))[:, None]
            q[:, 3:ie + 1, jg, 2:kn + 1] = torch.where(heated, wall, c)
        if ch.x_open:
            self.open_end(2, 3, False)
            self.open_end(ie + 1, ie, True)
        pl = slice(2, ie + 2) if ch.x_open else slice(None)
        q[:, pl, :, 1], q[:, pl, :, kn + 1] = q[:, pl, :, kn].clone(), q[:, pl, :, 2].clone()

    def open_end(self, ig, ic, outlet):
        """One pseudo-time step (dt / 200) of the characteristic relations
        M (Gamma + 3 dtau / (2 dt) M)^-1 (amplitudes + time derivative)."""
        ch, K = self.ch, self.K
        dt, dtau = ch.dt, ch.dt / 200
        sl = slice(None), slice(2, self.jn + 1), slice(2, self.kn + 1)
        q, qi = self.U_[:, ig][sl], self.U_[:, ic][sl]
        Jg, Ji = self.J[ig, 2:self.jn + 1], self.J[ic, 2:self.jn + 1]
        ri, ui, _, Pi = self.prim(qi, Ji)
        rho, u, VV, P = self.prim(q, Jg)
        T, C2, U = P / rho, K * P / rho, u[0]
        H = 0.5 * VV + C2 / (K - 1)
        beta = torch.clamp(VV / C2, min=C.PRECOND_EPS)
        s = 1 / (K * T * (2 * dt + 3 * dtau) * (2 * dt + 3 * beta * dtau))
        t3 = H - H * K - VV + K * (T + VV)
        a4 = -4 * (K - 1) * (beta - 1) * dt * dt * s
        b3 = 4 * t3 * (beta - 1) * dt * dt * s
        m = torch.zeros((5, 5) + U.shape, dtype=torch.float64, device=DEVICE)
        m[0, 0] = 2 * dt * (2 * ((K - 1) * (H - VV) + t3 * beta) * dt + 3 * K * T * beta * dtau) * s
        m[0, 4] = -a4
        m[4, 0] = H * b3
        m[4, 4] = 2 * dt * (2 * H * (K - 1) * (beta - 1) * dt + K * T * (2 * dt + 3 * beta * dtau)) * s
        for a in range(3):
            m[0, 1 + a], m[1 + a, 0] = u[a] * a4, u[a] * b3
            m[1 + a, 4], m[4, 1 + a] = -u[a] * a4, H * u[a] * a4
            for b in range(3):
                m[1 + a, 1 + b] = u[a] * u[b] * a4
            m[1 + a, 1 + a] = 2 * dt * (2 * K * (T - u[a] ** 2 * (beta - 1)) * dt + 2 * u[a] ** 2 * (beta - 1) * dt
                                        + 3 * K * T * beta * dtau) * s
        Up, Cp = 0.5 * (beta + 1) * U, 0.5 * torch.sqrt(U * U * (beta - 1) ** 2 + 4 * beta * C2)
        sg = -1 if outlet else 1
        dp, du, dT = sg * (Pi - P) / ch.dxi, sg * (ui - u) / ch.dxi, sg * (Pi / ri - T) / ch.dxi
        if outlet:
            L4 = (Up + Cp) * (dp - rho * (Up - Cp - U) * du[0])
            L5, leaving = L4 * (Up + Cp - U) / (Up - Cp - U), U > 0
        else:
            L5 = (Up - Cp) * (dp - rho * (Up + Cp - U) * du[0])
            L4, leaving = L5 * (Up - Cp - U) / (Up + Cp - U), U <= 0
        zero = torch.zeros_like(U)
        L1 = torch.where(leaving, U * (dT + dp * (1 - K) / K / rho), zero)
        L2, L3 = torch.where(leaving, U * du[2], zero), torch.where(leaving, -U * du[1], zero)
        k0 = 0.5 / Cp * (L4 * (Up + Cp - U) - L5 * (Up - Cp - U))
        amp = torch.stack([k0, 0.5 / (rho * Cp) * (L4 - L5), -L3, L2, L1 + (K - 1) / K * k0 / rho])
        amp = amp / Jg + (3 * q - 4 * self.U[:, ig][sl] + self.Uq[:, ig][sl]) / (2 * dt)
        self.U_[:, ig, 2:self.jn + 1, 2:self.kn + 1] = q - dtau * torch.einsum("abjk,bjk->ajk", m, amp)

    # ------------------------------------------------------------- fluxes
    def _faces(self, axis, first, last):
        """Interpolated left and right states of the faces n = first..last
        between cell n and n + 1 along `axis` (all interior cells across)."""
        keep = [slice(3, self.ie + 1), slice(2, self.jn + 1), slice(2, self.kn + 1)]

        def cut(lo, hi):
            sl = list(keep)
            sl[axis] = slice(lo, hi + 1)
            return self.U_[(slice(None),) + tuple(sl)], (1 / self.J.expand(self.U_.shape[1:]))[tuple(sl)]

        def side(lo, hi, offs, coef):
            if hi < lo:
                return None
            s = [(cut(lo + o, hi + o), c) for o, c in zip(offs, coef)]
            return sum(c * u for (u, _), c in s) / sum(c * w for (_, w), c in s)

        five = ((-2, -1, 0, 1, 2), (2, -13, 47, 27, -3)), ((-1, 0, 1, 2, 3), (-3, 27, 47, -13, 2))
        three = ((-1, 0, 1), (-1, 5, 2)), ((0, 1, 2), (2, 5, -1))
        two = (0, 1), (1, 1)
        if axis == 0 and not self.ch.x_open:
            return side(first, last, *five[0]), side(first, last, *five[1])
        f, e = first, last
        if axis == 1:
            left = [(f, f + 1, two), (f + 2, f + 2, three[0]), (f + 3, e - 2, five[0]), (e - 1, e - 1, three[0]),
                    (e, e, ((0, -1), (1, 1)))]
            right = [(f, f, ((1, 2), (1, 1))), (f + 1, f + 1, three[1]), (f + 2, e - 3, five[1]),
                     (e - 2, e - 2, three[1]), (e - 1, e - 1, ((1, 0), (1, 1))), (e, e, two)]
        else:
            left = [(f, f, two), (f + 1, f + 1, three[0]), (f + 2, e - 1, five[0]), (e, e, three[0])]
            right = [(f, f, three[1]), (f + 1, e - 2, five[1]), (e - 1, e - 1, three[1]), (e, e, two)]
        join = [[s for s in (side(lo, hi, *st) for lo, hi, st in seg) if s is not None] for seg in (left, right)]
        return torch.cat(join[0], axis + 1), torch.cat(join[1], axis + 1)

    def _cut_face(self, axis, first, last):
        """(J, normal vector components, the three metric vectors) of those faces."""
        sl = [slice(3, self.ie + 1), slice(2, self.jn + 1)]
        if axis < 2:
            sl[axis] = slice(first, last + 1)
        J, ex, ey = (m[tuple(sl)][:, :, None] for m in self.face[axis])
        one, zero = torch.ones_like(J), torch.zeros_like(J)
        return J, ((one, zero, zero), (ex, ey, zero), (zero, zero, one))

    def flux(self, axis):
        first, last = (2, 1, 1)[axis], (self.ie, self.jn, self.kn)[axis]
        L, R = self._faces(axis, first, last)
        J, dirs = self._cut_face(axis, first, last)
        m, K = dirs[axis], self.K
        sq = torch.sqrt(sum(a * a for a in m))

        def state(q):
            rho, u = q[0], q[1:4] / q[0]
            VV = (u * u).sum(0)
            P = (q[4] - 0.5 * rho * VV) * (K - 1)
            return rho, u, sum(a * b for a, b in zip(m, u)), VV, P, 0.5 * VV + K * P / rho / (K - 1)

        rl, ul, Ul, Vl, Pl, Hl = state(L)
        rr, ur, Ur, Vr, Pr, Hr = state(R)
        wl, wr = torch.sqrt(rl) / (torch.sqrt(rl) + torch.sqrt(rr)), torch.sqrt(rr) / (torch.sqrt(rl) + torch.sqrt(rr))
        rho, u, U, H = torch.sqrt(rl * rr), wl * ul + wr * ur, wl * Ul + wr * Ur, wl * Hl + wr * Hr
        VV = (u * u).sum(0)
        Cs = (H - 0.5 * VV) * (K - 1)
        th = VV / Cs
        beta, Un = torch.clamp(th, min=C.PRECOND_EPS), U / sq
        dP, dU = Pr - Pl, (Ur - Ul) / sq
        S = 0.5 * torch.sqrt(4 * beta * Cs + (Un * (1 - beta)) ** 2)
        Up, Cp = 0.5 * (1 + th) * Un, 0.5 * torch.sqrt(4 * Cs * th + (Un * (1 - th)) ** 2)
        t3 = 0.25 * (1 - beta) * (1 + beta) * Un * Un / S
        delU = (S - t3 - beta * Un.abs()) * dP / (rho * beta * Cs) + Up / S * dU
        delP = Up / S * dP + (Cp - Un.abs() + 0.5 * (1 - th) * Un * Up / S) * rho * dU
        jump = torch.stack([rr - rl, *(rr * ur - rl * ul), (Pr - Pl) / (K - 1) + 0.5 * (rr * Vr - rl * Vl)])
        one = torch.ones_like(rho)
        diss = Un.abs() * jump + delU * rho * torch.stack([one, *u, H]) + delP * torch.stack(
            [0 * one, *(one * a / sq for a in m), Un])
        conv = torch.stack([rl * Ul + rr * Ur, *(rl * ul[a] * Ul + rr * ur[a] * Ur + m[a] * (Pl + Pr) for a in range(3)),
                            Ul * (3.5 * Pl + 0.5 * rl * Vl) + Ur * (3.5 * Pr + 0.5 * rr * Vr)])
        F = 0.5 * (conv - diss * sq) / J
        if axis == 1:   # walls: pressure and the normal dissipation only
            for w in (0, -1):
                pp, Jw = (Pl + Pr)[:, w], J[:, w]
                F[:, :, w] = 0
                F[2, :, w] = 0.5 * (m[1][:, w] * pp - diss[2][:, w]) / Jw
                if self.ch.wavy:
                    F[1, :, w] = 0.5 * m[0][:, w] * pp / Jw
        return F.diff(dim=axis + 1) / self.d[axis]

    def viscous(self):
        """Divergence of the viscous fluxes (momentum and energy)."""
        J = self.J
        rho = self.U_[0]
        u = self.U_[1:4] / rho
        P = (self.U_[4] - 0.5 * rho * (u * u).sum(0)) * (self.K - 1) * J
        w = torch.cat([u, (P / (rho * self.R) / J)[None]])
        total = 0
        for axis in range(3):
            lo = [3, 2, 2]
            hi = [self.ie, self.jn, self.kn]
            hi[axis] += 1

            def at(n=0, t=None, s=0):
                sl = []
                for a in range(3):
                    o = (n if a == axis else 0) + (s if a == t else 0)
                    sl.append(slice(lo[a] + o, hi[a] + 1 + o))
                return w[(slice(None),) + tuple(sl)]

            Jf, dirs = self._cut_face(axis, lo[axis] - 1, hi[axis] - 1)
            n = dirs[axis]
            c, b = at(), at(-1)
            mean = 0.5 * (c + b)
            out = [0, 0, 0, 0]
            for t in range(3):
                if t == axis:
                    f = lambda g: (g(c) - g(b)) / self.d[axis]   # noqa: E731
                else:
                    p, pb, q, qb = at(0, t, 1), at(-1, t, 1), at(0, t, -1), at(-1, t, -1)
                    f = lambda g: 0.25 * (g(p) + g(pb) - g(q) - g(qb)) / self.d[t]   # noqa: E731
                nt = sum(a * d for a, d in zip(n, dirs[t]))
                for i in range(3):
                    for j in range(3):
                        cf = n[j] * dirs[t][i] - (2 / 3) * n[i] * dirs[t][j] + (nt if i == j else 0)
                        if not torch.any(cf != 0):
                            continue
                        du = f(lambda g, j=j: g[j])
                        out[i] = out[i] + cf * du
                        if i == j:
                            out[3] = out[3] + 0.5 * cf * f(lambda g, j=j: g[j] ** 2)
                        elif t != axis:
                            out[3] = out[3] + cf * mean[i] * du
                        elif i < j:
                            out[3] = out[3] + cf * f(lambda g, i=i, j=j: g[i] * g[j])
                out[3] = out[3] + self.CV * self.K * nt * f(lambda g: g[3]) / C.PR
            T = mean[3]
            mu = C.MU0 * (T / 298.0592) ** 1.5 * (298.0592 + 110) / (T + 110)
            total = total + torch.stack([mu * o / Jf for o in out]).diff(dim=axis + 1) / self.d[axis]
        return total

    # --------------------------------------------------- residual and update
    def residual(self, dplur):
        """Gamma^-1 of the residual on the interior cells, (5, nx, ny, nz)."""
        ch, K = self.ch, self.K
        J = self.J[3:self.ie + 1, 2:self.jn + 1]
        rho, u, VV, P = self.prim(self.U_[self.inner], J)
        Rk = -(3 * self.U_[self.inner] - 4 * self.U[self.inner] + self.Uq[self.inner]) / (2 * ch.dt)
        for axis in range(3):
            Rk = Rk - self.flux(axis)
        Rk[1:] += self.viscous()
        f = -(rho - 1.1842) * 9.81 if ch.buoyancy and not dplur else self.force
        Rk[1] += f / J
        Rk[4] += f * u[0] / J
        if ch.x_open and not dplur:
            Rk += self.sponge(rho, u, VV, P) / J
        T, Cs = P / rho, K * P / rho
        H, beta = 0.5 * VV + Cs / (K - 1), torch.clamp(VV / Cs, min=C.PRECOND_EPS)
        ur = (u * Rk[1:4]).sum(0)
        dH = -(H * (K - 1) + VV - K * (T + VV)) * beta
        d51 = (K - 1) * (VV + K * T * beta + (K - 1) * VV * beta + H * (beta - 1 - K * beta)) / (rho * K)
        MR = torch.stack([dH * Rk[0] - (K - 1) * beta * (ur - Rk[4]), *((Rk[1:4] - u * Rk[0]) / rho),
                          d51 * Rk[0] - (K - 1) * (1 + (K - 1) * beta) / (rho * K) * (ur - Rk[4])])
        return MR, rho, u, beta, Cs, P

    def sponge(self, rho, u, VV, P):
        ch, K, nx = self.ch, self.K, self.ch.nx
        i = torch.arange(3, self.ie + 1, dtype=torch.float64, device=DEVICE)[:, None, None]
        outlet = i >= max(3, nx - ch.nx_outlet + 2)
        inlet = ~outlet & (i <= ch.nx_inlet + 2)
        out = outlet.double()
        jk = slice(2, self.jn + 2), slice(2, self.kn + 2)
        up = (self.U_[1, 3] / self.U_[0, 3])[jk] * ch.det / self.cell[2][3][2:self.jn + 2, None] * ch.dzt
        target = up.sum() / (ch.high * ch.dzt * ch.nz)
        Cs = K * P / rho
        beta = torch.clamp(VV / Cs, min=C.PRECOND_EPS)
        Cpl = 0.5 * torch.sqrt((u[0] * (beta - 1)) ** 2 + 4 * beta * Cs)
        ramp = torch.where(outlet, (i - 0.5 - (nx + 1 - ch.nx_outlet)) / ch.nx_outlet,
                           torch.full_like(rho, (ch.nx_inlet - 0.5) / ch.nx_inlet)) ** 3
        Us = torch.where(outlet | inlet, ramp * Cpl, torch.zeros_like(rho))
        Sig = (0.035 + 1.215 * out) * Us / ch.high
        Q = self.U_ * self.J
        c = Q[self.inner]
        back = Q[:, 2:self.ie, 2:self.jn + 1, 2:self.kn + 1]
        far = torch.zeros_like(c)
        far[0], far[4] = 1.1842, 253250.0
        far[1] = out * 1.1842 * target
        far[4] += out * 0.5 * 1.1842 * target * target
        return -Us * (c - back) / ch.dxi - Sig * (c - far)

    def operators(self, rho, u, beta, Cs, P):
        """The split Jacobians A+ and A- of the three directions over their
        spacing, (cells, 15, 5) each, and the diagonal, sorted by hyperplane."""
        ch, K = self.ch, self.K
        _, ex, ey = (m[3:self.ie + 1, 2:self.jn + 1][:, :, None] for m in self.cell)
        one, zero = torch.ones_like(ex), torch.zeros_like(ex)
        dirs = ((one, zero, zero), (ex, ey, zero), (zero, zero, one))
        n = ch.cells
        low, high = (torch.zeros((n, 15, 5), dtype=torch.float64, device=DEVICE) for _ in range(2))
        lam = 0
        T = P / rho
        for a, m in enumerate(dirs):
            U = sum(x * y for x, y in zip(m, u))
            l = 0.5 * ((beta + 1) * U.abs() + torch.sqrt((U * (beta - 1)) ** 2 + 4 * beta * Cs * sum(x * x for x in m)))
            lam = lam + l / self.d[a]
            for A, s in ((low, 1), (high, -1)):
                B = A[:, 5 * a:5 * a + 5]

                def put(r, c, v):
                    B[:, r, c] = (0.5 * v).expand(rho.shape).reshape(-1)[self.order] / self.d[a]

                put(0, 0, beta * U + s * l)
                put(4, 0, U * (K - 1) * (beta - 1) / rho / K)
                put(4, 4, U + s * l)
                for v in range(3):
                    put(0, 1 + v, P * K * beta * m[v])
                    put(1 + v, 0, m[v] / rho)
                    put(1 + v, 1 + v, U + s * l)
                    put(4, 1 + v, beta * T * (K - 1) * m[v])
        a1, a2 = 2 * ch.dt / (3 * beta + 2 * lam * ch.dt), 2 * ch.dt / (3 + 2 * lam * ch.dt)
        d51 = -6 * (K - 1) * (beta - 1) * ch.dt / (K * rho) * a1 * a2 / (4 * ch.dt * ch.dt)
        diag = [x.reshape(-1)[self.order][:, None] for x in (a1, a2, d51)]
        return low, high, diag

    def iterate(self, solver):
        ch = self.ch
        self.boundaries()
        MR, rho, u, beta, Cs, P = self.residual(solver == "dplur")
        MR = MR.reshape(5, -1).t()[self.order]
        low, high, (a1, a2, d51) = self.operators(rho, u, beta, Cs, P)
        n, halo = ch.cells, ch.ny * ch.nz
        grid = lambda v: v[torch.argsort(self.order)].reshape(ch.nx, halo, -1)   # noqa: E731

        def diag(r, s=slice(None)):
            return torch.cat([a1[s] * r[:, :1], a2[s] * r[:, 1:4], d51[s] * r[:, :1] + a2[s] * r[:, 4:]], 1)

        def products(A, v, s=slice(None)):
            return torch.bmm(A[s], v[:, :, None])[:, :, 0]

        def halo_products(A, v, plane):
            """The x product of the periodic image of `plane`."""
            if ch.x_open:
                return torch.zeros((halo, 5), dtype=torch.float64, device=DEVICE)
            sl = grid(torch.arange(n, device=DEVICE)[:, None])[plane, :, 0]
            return products(A, v[sl], sl)[:, :5]

        dq = diag(MR)
        if solver == "dplur":
            for _ in range(4):
                s = 0
                for A, nb, plane, sign in ((low, self.low, -1, -1), (high, self.high, 0, 1)):
                    o = torch.zeros((n + halo + 1, 15), dtype=torch.float64, device=DEVICE)
                    o[:n], o[n:n + halo, :5] = products(A, dq), halo_products(A, dq, plane)
                    s = s + sign * sum(o[nb[a], 5 * a:5 * a + 5] for a in range(3))
                dq = diag(MR - s)
        else:
            ends = []
            start = [0]
            for c in self.count:
                start.append(start[-1] + c)
            for _ in range(2):
                first = dq
                for A, nb, plane, back in ((low, self.low, -1, False), (high, self.high, 0, True)):
                    o = torch.zeros((n + halo + 1, 15), dtype=torch.float64, device=DEVICE)
                    o[n:n + halo, :5] = halo_products(A, first, plane)
                    new = torch.empty_like(dq)
                    for p in reversed(range(len(self.count))) if back else range(len(self.count)):
                        s = slice(start[p], start[p + 1])
                        L = o[nb[0][s], :5] + o[nb[1][s], 5:10] + o[nb[2][s], 10:]
                        v = ends[s] - diag(L, s) if back else diag(MR[s] + L, s)
                        new[s] = v
                        o[s] = products(A, v, s)
                    ends = new
                dq = ends
        J = self.J[3:self.ie + 1, 2:self.jn + 1]
        dq = grid(dq).reshape(ch.nx, ch.ny, ch.nz, 5).permute(3, 0, 1, 2) * J
        Pn, un, Tn = P + dq[0], u + dq[1:4], P / rho + dq[4]
        rn = Pn / Tn
        self.U_[self.inner] = torch.stack([rn, *(rn * un), Pn / (self.K - 1) + 0.5 * rn * (un * un).sum(0)]) / J

    def step(self, iters, solver, order=0, correct=None):
        s, J = self.inner, self.J[3:self.ie + 1, 2:self.jn + 1]
        q0, q1, q2 = self.U[s], self.Uq[s], self.Uqq[s]
        if order:
            self.U_[s] = 2 * q0 - q1 if order == 1 else 3 * q0 - 3 * q1 + q2
        if correct:
            self.U_[s] += correct(q0 * J, q1 * J, q2 * J) / J
        for _ in range(iters):
            self.iterate(solver)
        pl = slice(2, self.ie + 2)
        self.Uqq[:, pl], self.Uq[:, pl], self.U[:, pl] = self.Uq[:, pl], self.U[:, pl].clone(), self.U_[:, pl]
        ch = self.ch
        bulk = self.U_[s][1].sum() / (1 / self.J[3, 2:self.jn + 1]).sum() / ch.nx / ch.nz
        e = ch.rho0 * ch.u_b - float(bulk)
        self.integral += e
        self.force = ch.force_lam + (0.5 * e + 0.05 * self.integral) / ch.dt

    def statistics(self):
        J = self.J[3:self.ie + 1, 2:self.jn + 1]
        rho, u, VV, P = self.prim(self.U_[self.inner], J)
        T = P / (rho * self.R)
        U, V, W = u
        rows = [x.sum(2) for x in (U, V, W, T, U * U, V * V, W * W, T * T, U * V, U * T, V * T)]
        k = 150 - 2
        rows += [x[:, :, k] if self.ch.nz > k else torch.zeros_like(rows[0]) for x in (U, T)]
        return torch.stack(rows)


def _layers(theta: torch.Tensor):
    """The network's weights (cout, cin, 3, 3, 3) and biases, layer by layer."""
    out, o = [], 0
    for ci, co in zip((15, 32, 32, 32, 32), (32, 32, 32, 32, 5)):
        n = 27 * ci * co
        out.append((theta[o:o + n].reshape(3, 3, 3, co, ci).permute(3, 4, 0, 1, 2), theta[o + n:o + n + co]))
        o += n + co
    return out


def _network(layers, x: torch.Tensor) -> torch.Tensor:
    x = x[None]
    for l, (w, b) in enumerate(layers):
        x = torch.nn.functional.pad(x, (1, 1, 0, 0, 1, 1), mode="circular")
        x = torch.nn.functional.conv3d(torch.nn.functional.pad(x, (0, 0, 1, 1, 0, 0)), w, b)
        x = torch.nn.functional.gelu(x) if l + 1 < len(layers) else x
    return x[0]


def _inputs(scales, q0, q1, q2):
    mean, std, d1, d2, _ = scales
    return torch.cat([(q0 - mean) / std, (q0 - q1) / d1, (q0 - 2 * q1 + q2) / d2])


def _correction(layers, scales, q0, q1, q2):
    return _network(layers, _inputs(scales, q0, q1, q2)) * scales[4]


def _exact_train(case, ch, seed):
    """Adam on the mean squared error of the scaled correction, the pairs
    drawn with the documented splitmix64 stream of the seed (1)."""
    from cgli_fu_flow_b200.cnn import scales_from_levels
    levels = _levels(ch, seed)
    scales = [torch.from_numpy(np.asarray(s)).to(DEVICE).double()[:, None, None, None] for s in scales_from_levels(levels)]
    q = [torch.from_numpy(x).to(DEVICE).double() for x in levels]
    theta = torch.from_numpy(_theta(seed)).to(DEVICE).double()
    m, v, losses, st, mask = torch.zeros_like(theta), torch.zeros_like(theta), [], 1, (1 << 64) - 1
    for k in range(1, case["iters"] + 1):
        st = (st + 0x9E3779B97F4A7C15) & mask
        r = ((st ^ (st >> 30)) * 0xBF58476D1CE4E5B9) & mask
        r = ((r ^ (r >> 27)) * 0x94D049BB133111EB) & mask
        p = (r ^ (r >> 31)) % 3
        with torch.enable_grad():
            t = theta.clone().requires_grad_(True)
            want = (q[p + 3] - (3 * q[p + 2] - 3 * q[p + 1] + q[p])) / scales[4]
            loss = ((_network(_layers(t), _inputs(scales, q[p + 2], q[p + 1], q[p])) - want) ** 2).mean()
            loss.backward()
        g = t.grad
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        theta = theta - 1e-3 * (m / (1 - 0.9 ** k)) / (torch.sqrt(v / (1 - 0.999 ** k)) + 1e-8)
        losses.append(float(loss))
    return {"loss": np.float64(np.mean(losses)), "theta": theta}


def _exact_filter(ch, slab, crit, e_high, e_low):
    """Six filter levels of the density and the momenta at two scales, the
    energy of the velocity's high-pass part, and its ratio on every face."""
    U, J = slab.U_[:4], slab.J.expand(slab.U_.shape[1:])
    Y = torch.from_numpy(ch.y_point()).to(DEVICE)
    g, ny, nz = ch.nx + 2, ch.ny + 1, ch.nz + 1
    jj, kk = slice(2, ny + 1), slice(2, nz + 1)
    energy = []
    for two in (False, True):
        mid, out = (2.0, 0.25) if two else (6.0, 0.125)
        prev, acc = U, 0
        for lev, hp in enumerate((6.0, -15.0, 20.0, -15.0, 6.0, -1.0)):
            a, b = ((1, g + 2), (2, g + 1), (3, g))[lev % 3]
            I = slice(a, b + 1)
            Gx, Gy, L = U.clone(), U.clone(), U.clone()
            Gx[:, I, jj, kk] = out * (prev[:, a - 1:b, jj, kk] + mid * prev[:, I, jj, kk] + prev[:, a + 1:b + 2, jj, kk])
            yp, yc, ym = (Y[I, s, kk] for s in (slice(3, ny + 2), jj, slice(1, ny)))
            wp, wm = (yp - yc) / (yp - ym), (yc - ym) / (yp - ym)
            r = [Gx[:, I, s, kk] * J[I, s, kk] for s in (slice(1, ny), jj, slice(3, ny + 2))]
            Gy[:, I, jj, kk] = (0.5 * (wp * r[0] + r[1] + wm * r[2]) if two else
                                0.125 * (2 * wp * r[0] + 6 * r[1] + 2 * wm * r[2])) / J[I, jj, kk]
            L[:, I, jj, kk] = out * (Gy[:, I, jj, 1:nz] + mid * Gy[:, I, jj, kk] + Gy[:, I, jj, 3:nz + 2])
            if lev == 2:
                L[:, g + 1:g + 4], L[:, 0:3] = L[:, 3:6].clone(), L[:, g - 2:g + 1].clone()
            acc = acc + hp * L[:, 3:g + 1, jj, kk]
            prev = L
        u = U[:, 3:g + 1, jj, kk]
        E = torch.zeros_like(J)
        E[3:g + 1, jj, kk] = ((u[1:] / u[0] - acc[1:] / acc[0]) ** 2).sum(0)
        E[:, 1], E[:, ny + 1] = E[:, 2], E[:, ny]
        E[:, :, 1], E[:, :, nz + 1] = E[:, :, 2], E[:, :, nz]
        E[2], E[g + 1] = E[g], E[3]
        energy.append(E)
    eps = []
    for axis in range(3):
        lo = [(3, 2, 2), (3, 1, 2), (3, 2, 1)][axis] if axis else (2, 2, 2)
        a = tuple(slice(l, h + 1) for l, h in zip(lo, (g, ny, nz)))
        b = tuple(slice(s.start + (t == axis), s.stop + (t == axis)) for t, s in enumerate(a))
        ratio = (energy[0][a] + energy[0][b]) / (energy[1][a] + energy[1][b])
        ep = torch.zeros_like(J)
        # arrays are indexed by the lower cell along the axis, one less across
        at = tuple(slice(s.start - (t != axis), s.stop - (t != axis)) for t, s in enumerate(a))
        high = (ratio >= crit).double()
        ep[at] = high * e_high + (1 - high) * e_low
        eps.append(ep)
    return eps
