"""The work a user of this framework has it do, as cases that can be timed and
compared: time marches of one grid (fast and exact precision, the run loop and
the per-step driver), batches of uneven steady solves, and the surrogate's
inference and training iteration.

Kinds of case:

``march``     the coaxial channel (``workloads.channel_config``): initial planes
              from pinned host memory, ``GpuSolver.run`` for a number of steps
              with adaptive dt, the 10 physical planes back in pinned memory
              (a restart, a stretch of the march, a snapshot).
``thruster``  the same for the short-cathode thruster with the axis of symmetry
              (three inner-wall segments, the last one AxisLF), the relative
              change checked every 100 steps as the driver loop does.
``driver``    the per-step drop-in loop: ``Advance(dt)``, ``ComputeDt`` back on
              the host, for a number of steps, then the snapshot.
``batch``     many solves of uneven grids in one ``BatchSolver.run`` on an
              autotuned plan.
``predict``   the surrogate's forward pass on a batch of parameter draws.
``train``     one training iteration of the surrogate (forward, loss, backward,
              Adam) through the captured graph.

``exact`` evaluates the same schemes in plain torch in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__

mpd = __graft_entry__.load_package()

GAMMA = 5.0 / 3.0
R1, R2 = 0.2, 0.8                 # electrode radii of the channel
SWEEP_GRIDS = ((100, 40), (200, 80), (400, 160), (800, 320))
PLANES = ("rho", "v_z", "v_r", "v_phi", "e", "p", "P", "H_z", "H_r", "H_phi")


def listed():
    return [
        # The smallest grid of the parameter sweep: launches and chains count.
        dict(name="march_100x40", kind="march", L=100, M=40, steps=1000, every=0),
        # The validation channel, 1000 steps, judged by the residual as a
        # steady solve is.
        dict(name="march_200x80", kind="march", L=200, M=80, steps=1000, every=50),
        # An odd, ragged grid (no multiple of a strip, a tile or a vector).
        dict(name="march_611x247", kind="march", L=611, M=247, steps=1000, every=50),
        # The grid the framework's throughput is quoted on.
        dict(name="march_1600x640", kind="march", L=1600, M=640, steps=1000, every=0),
        # The large grid of the serving mix.
        dict(name="march_4096x1600", kind="march", L=4096, M=1600, steps=300, every=0),
        # The thruster at its default resolution, in the default precision.
        dict(name="thruster_800x400", kind="thruster", L=800, M=400, steps=500, precision="fast"),
        # The same where the reference's bits are wanted.
        dict(name="thruster_exact_800x400", kind="thruster", L=800, M=400, steps=200,
             precision="exact"),
        # The host-driven loop of a program that steps the solver itself.
        dict(name="driver_400x160", kind="driver", L=400, M=160, steps=300),
        # The parameter sweep: uneven solves of all four grids at once.
        dict(name="batch_sweep", kind="batch", n=32, smallest=0, largest=3, steps=500),
        # Many solves of the smallest grid, as the surrogate's training data are made.
        dict(name="batch_small", kind="batch", n=96, smallest=0, largest=0, steps=500),
        # Inference on the grid the surrogate is trained on.
        dict(name="predict_400x160", kind="predict", H=400, W=161, batch=16),
        # One iteration of its bootstrap training on the coarse grid.
        dict(name="train_100x40", kind="train", H=100, W=41, batch=16),
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("march", "march", "march", "thruster", "thruster", "driver", "batch",
                       "predict", "train"))
    if kind == "march":
        L = _between(rng, 48, 4096)
        M = min(1600, max(16, int(L * rng.uniform(0.25, 0.6))))
        every = rng.choice((0, 50))
        return dict(kind=kind, L=L, M=M, steps=_between(rng, 150, 300 if L > 2000 else 1000),
                    every=every)
    if kind == "thruster":
        L = _between(rng, 100, 1000)
        M = max(24, int(L * rng.uniform(0.3, 0.6)))
        precision = rng.choice(("fast", "fast", "exact"))
        return dict(kind=kind, L=L, M=M, steps=200, precision=precision)
    if kind == "driver":
        L = _between(rng, 64, 1600)
        return dict(kind=kind, L=L, M=max(16, int(L * rng.uniform(0.3, 0.5))),
                    steps=_between(rng, 50, 300))
    if kind == "batch":
        lo = rng.randrange(4)
        hi = rng.randrange(lo, 4)
        return dict(kind=kind, n=_between(rng, 4, 96 if hi < 2 else 24), smallest=lo, largest=hi,
                    steps=_between(rng, 100, 500))
    H = _between(rng, 50, 400 if kind == "predict" else 200)
    return dict(kind=kind, H=H, W=int(H * 0.4) + rng.randrange(2),
                batch=rng.choice((1, 4, 16)) if kind == "predict" else 16)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _channel_draw(rng):
    """A point of the sweep box."""
    return dict(amp=float(rng.uniform(0.5, 2.0)),
                beta=float(math.exp(rng.uniform(math.log(0.05), math.log(1.0)))),
                vz=float(rng.uniform(0.05, 0.3)), a=float(rng.uniform(0.0, 0.2)))


def _channel_params(case, seed):
    return _channel_draw(np.random.default_rng([seed, case["L"], case["M"]]))


def _batch_params(case, seed):
    rng = np.random.default_rng([seed, case["n"], case["smallest"], case["largest"]])
    grids = SWEEP_GRIDS[case["smallest"]:case["largest"] + 1]
    out = []
    for i in range(case["n"]):
        L, M = grids[i % len(grids)]
        out.append(dict(_channel_draw(rng), L=L, M=M))
    return out


def _thruster_params(case, seed):
    rng = np.random.default_rng([seed, case["L"], case["M"], 7])
    L = case["L"]
    hi1, hi2 = int(235 * L / 800), int(263 * L / 800)
    return dict(beta=float(0.01 * rng.uniform(0.8, 1.25)), Hz0=float(0.25 * rng.uniform(0.8, 1.25)),
                rho=float(0.1 * rng.uniform(0.8, 1.25)), vz=float(0.1 * rng.uniform(0.8, 1.25)),
                hi1=hi1, hi2=hi2)


def _thruster_config(case, p):
    return mpd.SimConfig.from_yaml(f"""
physics: {{gamma: 1.67, beta: {p['beta']!r}, H_z0: {p['Hz0']!r}}}
time: {{T: 6, dt: 1.0e-7}}
adaptive_dt: {{enabled: true, cfl_number: 0.45, growth_factor: 1.10, dt_min: 1.0e-10, dt_max: 5.0e-5}}
grid: {{L_max: {case['L']}, M_max: {case['M']}}}
convergence: {{threshold: 1.0e-30, check_frequency: 100}}
geometry:
  type: short_cathode_cosine
  params: {{z_center: 0.31, transition_half_width: 0.02, r_inner_before: 0.200,
            r_inner_after: 0.005, r_outer: 0.800}}
initial_conditions:
  rho: {p['rho']!r}
  v_z: {p['vz']!r}
  v_r: 0.1
  v_phi: 0.0
  H_z: H_z0
  H_r: "H_z * r_z"
  H_phi: "(1 - 0.9 * z) * r_0 / r"
  e: "beta / (2 * (gamma - 1))"
boundary_conditions:
  l_lo:
    - {{rho: neumann, v_z: {{dirichlet: 0.0}}, v_r: neumann, v_phi: neumann, e: neumann,
       H_z: "H_z0", H_r: {{dirichlet: 0.0}}, H_phi: "r_0 / r"}}
  l_hi:
    - {{rho: neumann, v_z: neumann, v_r: neumann, v_phi: neumann, e: neumann, H_z: neumann,
       H_r: neumann, H_phi: neumann}}
  m_hi:
    - {{rho: neumann, v_z: neumann, v_r: "v_z * r_z", v_phi: neumann, e: neumann,
       H_z: neumann, H_r: "H_z * r_z", H_phi: neumann}}
  m_lo:
    - {{range: [0, {p['hi1']}], rho: neumann, v_z: neumann, v_r: "v_z_nb * r_z_nb",
       v_phi: neumann, e: neumann, H_z: neumann, H_r: "H_z_nb * r_z_nb", H_phi: neumann}}
    - {{range: [{p['hi1'] + 1}, {p['hi2']}], rho: {{dirichlet: {p['rho']!r}}},
       v_z: neumann, v_r: neumann, v_phi: {{dirichlet: 0.0}}, e: "beta / (2 * (gamma - 1))",
       H_z: neumann, H_r: "H_z_nb * r_z_nb", H_phi: neumann}}
    - {{range: [{p['hi2'] + 1}, -1], rho: axis_lf, v_z: axis_lf, v_r: {{dirichlet: 0.0}},
       v_phi: {{dirichlet: 0.0}}, e: axis_lf, H_z: axis_lf, H_r: {{dirichlet: 0.0}},
       H_phi: {{dirichlet: 0.0}}}}
""")


def _pinned(L, M, *n):
    return torch.empty((*n, 10, L + 2, M + 3), dtype=torch.float64, pin_memory=True)


def _solver(cfg, precision, out=None):
    """A solver, its initial planes in pinned host memory and a snapshot buffer."""
    s = mpd.build_case(cfg, precision=precision)
    planes = _pinned(cfg.L_max, cfg.M_max)
    out = _pinned(cfg.L_max, cfg.M_max) if out is None else out
    s.snapshot_async(planes)
    s.snapshot_wait()
    return dict(s=s, cfg=cfg, planes=planes.numpy(), out=out)


def _features(H, W, batch, seed):
    """The surrogate's input (batch x H W x 6, float32): the scaled parameters
    of each draw, and the point's r and z."""
    rng = np.random.default_rng([seed, H, W, batch, 3])
    x = np.empty((batch, H, W, 6))
    z = np.arange(H) / H
    y = np.arange(W) / (W - 1)
    for b in range(batch):
        p = _channel_draw(rng)
        x[b, :, :, 0] = 2 * (p["amp"] - 0.5) / 1.5 - 1
        x[b, :, :, 1] = 2 * (math.log(p["beta"]) - math.log(0.05)) / -math.log(0.05) - 1
        x[b, :, :, 2] = 2 * (p["vz"] - 0.05) / 0.25 - 1
        x[b, :, :, 3] = 2 * p["a"] / 0.2 - 1
        outer = R2 - p["a"] * np.sin(np.pi * z)
        r = (1 - y)[None, :] * R1 + y[None, :] * outer[:, None]
        x[b, :, :, 4] = 2 * (r - 0.5) / 0.6
        x[b, :, :, 5] = (2 * z - 1)[:, None]
    return torch.from_numpy(x.reshape(batch, H * W, 6).astype(np.float32))


def _targets(x, seed):
    """Normalised fields to train on: smooth functions of the input."""
    g = torch.Generator().manual_seed(seed % (1 << 31))
    A = torch.randn(6, 8, generator=g)
    b = torch.randn(8, generator=g)
    return torch.sin(x @ A + b)


def _weights(seed):
    """The network's parameters (width 64, 8 modes per axis, 4 layers)."""
    rng = np.random.default_rng([seed, 11])
    C, Q, hid = 64, 256, 128
    out = {"W_in": rng.standard_normal((6, C)) / math.sqrt(6), "b_in": np.zeros(C)}
    for l in range(4):
        out[f"W{l}"] = rng.standard_normal((C, C)) / math.sqrt(C)
        out[f"b{l}"] = 0.1 * rng.standard_normal(C)
        out[f"R{l}"] = rng.standard_normal((Q, C, C), dtype=np.float32) * (0.5 / math.sqrt(C))
    out["W_p1"] = rng.standard_normal((C, hid)) / math.sqrt(C)
    out["b_p1"] = 0.1 * rng.standard_normal(hid)
    out["W_p2"] = rng.standard_normal((hid, 8)) / math.sqrt(hid)
    out["b_p2"] = np.zeros(8)
    return {k: v.astype(np.float32) for k, v in out.items()}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("march", "driver"):
        p = _channel_params(case, seed)
        st = _solver(mpd.workloads.channel_config(L=case["L"], M=case["M"], **p), "fast")
    elif kind == "thruster":
        st = _solver(_thruster_config(case, _thruster_params(case, seed)), case["precision"])
    elif kind == "batch":
        params = _batch_params(case, seed)
        cfgs = [mpd.workloads.channel_config(**p) for p in params]
        # one snapshot buffer per grid, a solve's planes in its own slot
        outs, parts = {}, []
        for L, M in dict.fromkeys((c.L_max, c.M_max) for c in cfgs):
            n = sum((c.L_max, c.M_max) == (L, M) for c in cfgs)
            outs[f"{L}x{M}"] = _pinned(L, M, n)
        slot = {k: iter(v) for k, v in outs.items()}
        for c in cfgs:
            parts.append(_solver(c, "fast", next(slot[f"{c.L_max}x{c.M_max}"])))
        batch = mpd.BatchSolver([q["s"] for q in parts])
        # the plan for solves that all take the same number of steps
        tuner = mpd.Autotuner(batch.capacity, steps=50)
        plan = tuner.plan(cfgs, max_steps=case["steps"], estimate=lambda c, n: n)
        st = dict(parts=parts, batch=batch, plan=plan, outs=outs)
    else:
        H, W, B = case["H"], case["W"], case["batch"]
        net = mpd.surrogate.SpectralOperator(H, W, B, params=_weights(seed))
        x = _features(H, W, B, seed)
        st = dict(net=net, x=x.reshape(-1, 6).cuda())
        net.x.copy_(st["x"])
        if kind == "train":
            st["y"] = _targets(x, seed).reshape(-1, 8).cuda()
            net.target.copy_(st["y"])
            net.capture()
    st["case"] = case
    return st


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def _numbers(r):
    return np.array([r.t, r.dt, r.residual, r.change, r.max_wave_speed])


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("march", "thruster"):
        s = st["s"]
        s.set_physical(st["planes"])
        r = s.run(T=1e300, max_steps=case["steps"], residual_every=case.get("every") or None)
        s.snapshot_async(st["out"])
        s.snapshot_wait()
        return dict(planes=st["out"], numbers=_numbers(r), steps=r.steps)
    if kind == "driver":
        s, cfg = st["s"], st["cfg"]
        s.set_physical(st["planes"])
        dt = cfg.dt
        for _ in range(case["steps"]):
            s.Advance(dt)
            dt = s.ComputeDt(dt)
        s.snapshot_async(st["out"])
        s.snapshot_wait()
        return dict(planes=st["out"], dt=np.array([dt]))
    if kind == "batch":
        for q in st["parts"]:
            q["s"].set_physical(q["planes"])
        res = st["batch"].run(st["plan"], max_steps=case["steps"], residual_every=50)
        for q in st["parts"]:
            q["s"].snapshot_async(q["out"])
        for q in st["parts"]:
            q["s"].snapshot_wait()
        return dict(planes=st["outs"],
                    numbers=np.stack([_numbers(r) for r in res.runs]),
                    steps=np.array([r.steps for r in res.runs]))
    net = st["net"]
    if kind == "predict":
        net.x.copy_(st["x"])
        return net.forward()
    net.x.copy_(st["x"])
    net.target.copy_(st["y"])
    net.train_step(lr=1e-3)
    return dict(loss=net.loss, grad=net.grad, weights=net.flat, out=net.out)


def work(case):
    kind = case["kind"]
    if kind in ("march", "thruster", "driver"):
        cells = case["L"] * (case["M"] + 1)
        moved = 2 * 10 * 8 * (case["L"] + 2) * (case["M"] + 3)
        # 8 conserved values read and written a step, ~190 operations on 64-bit values
        return dict(bytes=128.0 * cells * case["steps"] + moved, flops=190.0 * cells * case["steps"])
    if kind == "batch":
        grids = SWEEP_GRIDS[case["smallest"]:case["largest"] + 1]
        cells = sum(grids[i % len(grids)][0] * (grids[i % len(grids)][1] + 1)
                    for i in range(case["n"]))
        return dict(bytes=(128.0 * case["steps"] + 160.0) * cells,
                    flops=190.0 * cells * case["steps"])
    P, B, C, Q, hid = case["H"] * case["W"], case["batch"], 64, 256, 128
    rows = P * B
    layer = 2.0 * rows * C * C + 2 * 2.0 * rows * C * Q + 2.0 * B * Q * C * C
    fwd = 2.0 * rows * 6 * C + 4 * layer + 2.0 * rows * C * hid + 2.0 * rows * hid * 8
    nparam = 6 * C + 4 * (C * C + Q * C * C) + C * hid + hid * 8
    # per layer the activation in and out; input, output; bases and weights once
    moved = 4.0 * (rows * (6 + 8 + C * 2 * 5 + hid * 2) + 2 * P * Q + nparam)
    if kind == "predict":
        return dict(bytes=moved, flops=fwd)
    return dict(bytes=3 * moved + 4.0 * 7 * nparam, flops=3 * fwd)


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _March:
    """The Lax-Friedrichs march of a stack of same-shaped grids, arrays
    (solves, rows l = 1..L, columns m = 1..M+1), plain 64-bit torch."""

    def __init__(self, L, M, gamma, rin, rout, drin, drout, prims, bc):
        self.L, self.M, self.g = L, M, gamma
        y = (torch.arange(M + 1, dtype=torch.float64) / M).to(rin.device)
        self.r = (1 - y) * rin[:, :, None] + y * rout[:, :, None]
        self.rz = (1 - y) * drin[:, :, None] + y * drout[:, :, None]
        self.dr = ((rout - rin) / M)[:, :, None]
        self.dz, self.dy = 1.0 / L, 1.0 / M
        self.bc = bc
        self.old = prims            # rho, v_z, v_r, v_phi, e, H_z, H_r, H_phi
        self.U = self.conserved(prims, self.r)
        n = self.U[0].shape[0]
        self.t = torch.zeros(n, dtype=torch.float64, device=rin.device)
        self.residual = self.change = None
        self.speed = None

    @staticmethod
    def conserved(q, r):
        rho, vz, vr, vp, e, Hz, Hr, Hp = q
        m = rho * r
        return [m, m * vz, m * vr, m * vp, m * e, Hp, Hz * r, Hr * r]

    @staticmethod
    def prims(U, r):
        i = 1 / U[0]
        return [U[0] / r, U[1] * i, U[2] * i, U[3] * i, U[4] * i, U[6] / r, U[7] / r, U[5]]

    def pressures(self, q):
        p = (self.g - 1) * q[0] * q[4]
        return p, p + 0.5 * (q[5] ** 2 + q[6] ** 2 + q[7] ** 2)

    def step(self, dt):
        """One step with dt per solve, shape (solves,)."""
        U, q, r = self.U, self.old, self.r
        rho, vz, vr, vp, e, Hz, Hr, Hp = q
        p, P = self.pressures(q)
        d = dt[:, None, None]
        kz = d / (2 * self.dz)
        kr = d / (2 * self.dr[:, 1:-1])
        N, S = (slice(None), slice(2, None), slice(1, -1)), (slice(None), slice(None, -2), slice(1, -1))
        E, W = (slice(None), slice(1, -1), slice(2, None)), (slice(None), slice(1, -1), slice(None, -2))
        C = (slice(None), slice(1, -1), slice(1, -1))
        Gz = [None, (Hz * Hz - P) * r, Hz * Hr * r, Hp * Hz * r, None, Hz * vp, None, Hz * vr * r]
        Gr = [None, Hz * Hr * r, (Hr * Hr - P) * r, Hp * Hr * r, None, Hr * vp, Hr * vz * r, None]
        new = []
        for k in range(8):
            u = U[k]
            o = 0.25 * (u[N] + u[S] + u[E] + u[W])
            if k != 6:
                f = -u * vz if Gz[k] is None else Gz[k] - u * vz
                o = o + kz * (f[N] - f[S])
            if k != 7:
                f = -u * vr if Gr[k] is None else Gr[k] - u * vr
                o = o + kr * (f[E] - f[W])
            new.append(o)
        new[2] = new[2] + d * (rho * vp * vp + P - Hp * Hp)[C]
        new[3] = new[3] + d * (-rho * vr * vp + Hp * Hr)[C]
        a, b = vz * r, vr * r
        new[4] = new[4] - p[C] * (kz * (a[N] - a[S]) + kr * (b[E] - b[W]))
        n = [torch.empty_like(x) for x in U]
        for k in range(8):
            n[k][C] = new[k]
        self.faces(n, self.prims(new, r[C]), dt)
        num = torch.stack([(n[k] - U[k]).abs().amax(dim=(1, 2)) for k in range(8)])
        den = torch.stack([U[k].abs().amax(dim=(1, 2)) for k in range(8)])
        self.residual = (num / den.clamp_min(1e-300)).amax(0)
        self.U = n
        self.old = self.prims(n, r)
        q = self.old
        cs = torch.sqrt(self.g * (self.g - 1) * q[4])
        ca = torch.sqrt((q[5] ** 2 + q[6] ** 2 + q[7] ** 2) / q[0])
        self.speed = (torch.sqrt(q[1] ** 2 + q[2] ** 2) + cs + ca).amax(dim=(1, 2))
        self.t = self.t + dt

    def faces(self, n, c, dt):
        """L_LO, M_HI, M_LO, L_HI in that order; c: new primitives of the
        interior cells (row i, column j of c is row i + 1, column j + 1)."""
        old = self.old
        # L_LO: interior columns see the new row 2, the wall columns the old one
        nb = [torch.cat([o[:, 1, :1], x[:, 0, :], o[:, 1, -1:]], dim=1) for o, x in zip(old, c)]
        first = self.bc["l_lo"](self, nb)
        hi_nb = [torch.cat([f[:, -2:-1], x[:, :, -1]], dim=1) for f, x in zip(first, c)]
        m_hi = self.bc["m_hi"](self, hi_nb)                       # rows 1..L-1
        lo_nb = [x[:, :, 0] for x in c]
        m_lo, axis = self.bc["m_lo"](self, lo_nb, dt)             # rows 2..L-1
        last = [torch.cat([a[:, -1:], x[:, -1, :], b[:, -1:]], dim=1)
                for a, x, b in zip(m_lo, c, m_hi)]
        r = self.r

        def put(where, q):
            for k, u in enumerate(self.conserved(q, r[where])):
                n[k][where] = u

        put((slice(None), 0), first)
        put((slice(None), slice(0, -1), -1), m_hi)
        put((slice(None), slice(1, -1), 0), m_lo)
        for k, (row, u) in axis.items():
            n[k][:, row:self.L - 1, 0] = u
        put((slice(None), -1), self.bc["l_hi"](self, last))

    def run(self, steps, dt0, cfl, dt_min, dt_max, check=0):
        dx = min(self.dz, self.dy)
        dt = torch.full_like(self.t, dt0)
        prev = [x.clone() for x in self.seven()]
        for i in range(steps):
            self.step(dt)
            dt = torch.minimum(dt * 1.1, cfl * dx / (self.speed + 1e-10)).clamp(dt_min, dt_max)
            if check and (i + 1) % check == 0:
                now = self.seven()
                num = sum(((x - y) ** 2).sum(dim=(1, 2)) for x, y in zip(now, prev))
                den = sum((x ** 2).sum(dim=(1, 2)) for x in now)
                self.change = torch.sqrt(num) / torch.sqrt(den)
                prev = [x.clone() for x in now]
        self.dt = dt
        return self

    def seven(self):
        q = self.old
        return [q[0], q[1], q[2], q[3], q[5], q[6], q[7]]

    def planes(self):
        """(solves, 10, L + 2, M + 3) with zero ghost cells."""
        q = self.old
        p, P = self.pressures(q)
        x = torch.stack([q[0], q[1], q[2], q[3], q[4], p, P, q[5], q[6], q[7]], dim=1)
        return torch.nn.functional.pad(x, (1, 1, 1, 1))

    def numbers(self):
        """(solves, 5): t, next dt, residual, relative change, wave speed."""
        change = self.change if self.change is not None else torch.zeros_like(self.t)
        return torch.stack([self.t, self.dt, self.residual, change, self.speed], dim=1)


def _exact_channel(L, M, params, steps):
    """March of the solves in params (amp, beta, vz, a each) on one grid."""
    dev = _device()
    col = {k: torch.tensor([p[k] for p in params], dtype=torch.float64, device=dev)[:, None]
           for k in ("amp", "beta", "vz", "a")}
    z = (torch.arange(L, dtype=torch.float64) / L).to(dev)[None, :]
    one = torch.ones_like(col["a"])
    rin, rout = R1 * one * torch.ones_like(z), R2 - col["a"] * torch.sin(math.pi * z)
    drin, drout = torch.zeros_like(rin), -col["a"] * math.pi * torch.cos(math.pi * z)
    e0 = col["beta"] / (2 * (GAMMA - 1))
    y = (torch.arange(M + 1, dtype=torch.float64) / M).to(dev)
    r = (1 - y) * rin[:, :, None] + y * rout[:, :, None]
    zero = torch.zeros_like(r)
    q = [zero + 1, zero + col["vz"][:, :, None], zero, zero, zero + e0[:, :, None], zero, zero,
         (col["amp"] * 0.2)[:, :, None] / r]

    def l_lo(m, nb):
        o = torch.zeros_like(nb[0])
        return [o + 1, o + col["vz"], o, o, o + e0, nb[5], nb[6], col["amp"] * 0.2 / m.r[:, 0]]

    def wall(nb, rz):
        return [nb[0], nb[1], nb[1] * rz, nb[3], nb[4], nb[5], nb[5] * rz, nb[7]]

    bc = dict(l_lo=l_lo, l_hi=lambda m, nb: nb,
              m_hi=lambda m, nb: wall(nb, m.rz[:, :-1, -1]),
              m_lo=lambda m, nb, dt: (wall(nb, m.rz[:, 1:-1, 0]), {}))
    return _March(L, M, GAMMA, rin, rout, drin, drout, q, bc).run(steps, 1e-5, 0.4, 1e-12, 1.0)


def _exact_thruster(case, p):
    dev = _device()
    L, M, g = case["L"], case["M"], 1.67
    zc, hw, before, after, outer = 0.31, 0.02, 0.200, 0.005, 0.800
    z = (torch.arange(L, dtype=torch.float64) / L)[None, :]
    xi = (z - (zc - hw)) / (2 * hw)
    rin = torch.where(z < zc - hw, before, torch.where(
        z < zc + hw, before + (after - before) * 0.5 * (1 - torch.cos(math.pi * xi)), after))
    drin = torch.where((z < zc - hw) | (z >= zc + hw), 0.0,
                       (after - before) * 0.5 * math.pi * torch.sin(math.pi * xi) / (2 * hw))
    rin, drin, z = rin.to(dev), drin.to(dev), z.to(dev)
    rout, drout = torch.full_like(rin, outer), torch.zeros_like(rin)
    r0 = (before + outer) / 2
    y = (torch.arange(M + 1, dtype=torch.float64) / M).to(dev)
    r = (1 - y) * rin[:, :, None] + y * rout[:, :, None]
    rz = (1 - y) * drin[:, :, None] + y * drout[:, :, None]
    zero = torch.zeros_like(r)
    e0 = p["beta"] / (2 * (g - 1))
    Hz = zero + p["Hz0"]
    q = [zero + p["rho"], zero + p["vz"], zero + 0.1, zero, zero + e0, Hz, Hz * rz,
         (1 - 0.9 * z[:, :, None]) * r0 / r]
    # rows of the M_LO segments, as indices of rows 2..L-1
    b1, b2 = p["hi1"], p["hi2"]      # last index of the first / second segment, exclusive

    def l_lo(m, nb):
        o = torch.zeros_like(nb[0])
        return [nb[0], o, nb[2], nb[3], nb[4], o + p["Hz0"], o, r0 / m.r[:, 0]]

    def m_hi(m, nb):
        rz_ = m.rz[:, :-1, -1]
        return [nb[0], nb[1], nb[1] * rz_, nb[3], nb[4], nb[5], nb[5] * rz_, nb[7]]

    def m_lo(m, nb, dt):
        old = [x[:, :, 0] for x in m.old]              # rows 1..L of the wall column
        kept = [x[:, 1:-1] for x in old]               # rows 2..L-1
        rznb = m.rz[:, 1:-1, 1]
        o = torch.zeros_like(nb[0])
        s1 = [nb[0], nb[1], nb[1] * rznb, nb[3], nb[4], nb[5], nb[5] * rznb, nb[7]]
        s2 = [o + p["rho"], nb[1], nb[2], o, o + e0, nb[5], nb[5] * rznb, nb[7]]
        s3 = [kept[0], kept[1], o, o, kept[4], kept[5], o, o]
        out = [torch.cat([a[:, :b1], b[:, b1:b2], c[:, b2:]], dim=1) for a, b, c in zip(s1, s2, s3)]
        # the axis rows' half-stencil update: row index i of rows 2..L-1 is
        # index i + 1 of rows 1..L
        i0 = b2
        U = m.U
        P = m.pressures(m.old)[1][:, :, 0]
        pg = m.pressures(m.old)[0][:, :, 0]
        n_rows = m.L - 2
        c, no, so = slice(i0 + 1, n_rows + 1), slice(i0 + 2, n_rows + 2), slice(i0, n_rows)
        d = dt[:, None]
        dr = m.dr[:, c, 0]
        vzc, vzn = old[1][:, c], old[1][:, no]
        Hzc, Hzn = old[5][:, c], old[5][:, no]
        vzs, Hzs = old[1][:, so].clone(), old[5][:, so].clone()
        vzs[:, 0], Hzs[:, 0] = out[1][:, i0 - 1], out[5][:, i0 - 1]   # the segment before it
        vr_e, Hz_e, Hr_e, vz_e = (nb[k][:, i0:] for k in (2, 5, 6, 1))
        rc, rn, rs, re = m.r[:, c, 0], m.r[:, no, 0], m.r[:, so, 0], m.r[:, c, 1]
        fix = {}

        def parts(k):
            u = U[k]
            return (u[:, c, 0] / rc, u[:, no, 0] / rn, u[:, so, 0] / rs, u[:, c, 1] / re)

        for k in (0, 1, 4, 6):
            uc, un, us, ue = parts(k)
            mean = 0.25 * (un + us + ue + uc)
            along = -(un * vzn - us * vzs) / (2 * m.dz)
            across = -(ue * vr_e) / dr                # v_r of the axis cell is 0
            if k == 0:
                across = -(ue * vr_e - uc * vr_e) / dr
                s = along + across
            elif k == 1:
                s = ((Hzn * Hzn - P[:, no]) - (Hzs * Hzs - P[:, so])) / (2 * m.dz) \
                    + Hz_e * Hr_e / dr + along + across
            elif k == 4:
                s = -pg[:, c] * ((vzn - vzs) / (2 * m.dz) + vr_e / dr) + along + across
            else:
                s = Hr_e * vz_e / dr + across
            fix[k] = (i0 + 1, (mean + d * s) * rc)
        return out, fix

    bc = dict(l_lo=l_lo, l_hi=lambda m, nb: nb, m_hi=m_hi, m_lo=m_lo)
    return _March(L, M, g, rin, rout, drin, drout, q, bc).run(case["steps"], 1e-7, 0.45, 1e-10,
                                                            5e-5, check=100)


def _basis(n):
    x = (torch.arange(n, dtype=torch.float64) + 0.5) / n
    rows = [torch.cos(2 * math.pi * k * x) for k in range(8)]
    rows += [torch.sin(2 * math.pi * k * x) for k in range(1, 9)]
    return torch.stack(rows)


def _network(x, w, H, W):
    """The spectral operator on x (batch, H W, 6), 64 bits."""
    bz, by = _basis(H).to(x.device), _basis(W).to(x.device)
    B = x.shape[0]
    gelu = torch.nn.functional.gelu
    tanh = dict(approximate="tanh")
    h = x @ w["W_in"] + w["b_in"]
    for l in range(4):
        grid = h.reshape(B, H, W, -1)
        v = torch.einsum("ah,bw,nhwc->nabc", bz, by, grid).reshape(B, 256, -1) / (H * W)
        u = torch.einsum("nqc,qcd->nqd", v, w[f"R{l}"]).reshape(B, 16, 16, -1)
        s = torch.einsum("ah,bw,nabc->nhwc", bz, by, u).reshape(B, H * W, -1)
        h = h @ w[f"W{l}"] + w[f"b{l}"] + s
        if l < 3:
            h = gelu(h, **tanh)
    h = gelu(h @ w["W_p1"] + w["b_p1"], **tanh)
    return h @ w["W_p2"] + w["b_p2"]


def exact(case, seed):
    kind = case["kind"]
    if kind == "march":
        m = _exact_channel(case["L"], case["M"], [_channel_params(case, seed)], case["steps"])
        return dict(planes=m.planes()[0], numbers=m.numbers()[0].cpu().numpy(), steps=None)
    if kind == "driver":
        m = _exact_channel(case["L"], case["M"], [_channel_params(case, seed)], case["steps"])
        return dict(planes=m.planes()[0], dt=m.dt.cpu().numpy())
    if kind == "thruster":
        m = _exact_thruster(case, _thruster_params(case, seed))
        return dict(planes=m.planes()[0], numbers=m.numbers()[0].cpu().numpy(), steps=None)
    if kind == "batch":
        params = _batch_params(case, seed)
        numbers, planes = [None] * len(params), {}
        for L, M in SWEEP_GRIDS:
            idx = [i for i, p in enumerate(params) if (p["L"], p["M"]) == (L, M)]
            if not idx:
                continue
            m = _exact_channel(L, M, [params[i] for i in idx], case["steps"])
            planes[f"{L}x{M}"] = m.planes()
            for i, row in zip(idx, m.numbers().cpu().numpy()):
                numbers[i] = row
        return dict(planes=planes, numbers=np.stack(numbers), steps=None)
    H, W, B = case["H"], case["W"], case["batch"]
    dev = _device()
    w = {k: torch.from_numpy(v).to(dev, torch.float64) for k, v in _weights(seed).items()}
    x = _features(H, W, B, seed)
    xd = x.to(dev, torch.float64)
    if kind == "predict":
        with torch.no_grad():
            return _network(xd, w, H, W).reshape(-1, 8)
    for v in w.values():
        v.requires_grad_(True)
    y = _network(xd, w, H, W)
    loss = ((y - _targets(x, seed).to(dev, torch.float64)) ** 2).mean()
    loss.backward()
    order = ["W_in", "b_in"] + [n for l in range(4) for n in (f"W{l}", f"b{l}", f"R{l}")] + \
        ["W_p1", "b_p1", "W_p2", "b_p2"]
    grad = torch.cat([w[k].grad.reshape(-1) for k in order])
    flat = torch.cat([w[k].detach().reshape(-1) for k in order])
    # Adam's first step: both bias-corrected moments are the gradient's own
    new = flat - 1e-3 * grad / (grad.abs() + 1e-8)
    return dict(loss=loss.detach().reshape(1), grad=grad, weights=new, out=y.detach().reshape(-1, 8))
