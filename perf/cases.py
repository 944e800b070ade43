"""Timed cases of the framework: what a flow solver that runs on it does between two looks at its fields.

A pass advances the flow a stretch of time steps through the public binding (`chapsim.gpu`, which calls the C ABI one
to one) and brings the fields to pinned host buffers, as a run does between two dumps. The state evolves from pass to
pass, as a run's does. Kinds:

  channel   periodic channel, `advance(steps)`: one graph replay per step. FP64 contexts let `autotune` choose the
            kernel variants; mixed-precision ones pin the choice (`tune`), as a program does whose results have to be
            reproducible bit by bit.
  driver    periodic channel, called as the unchanged Fortran time loop calls it: CFL and dt, three substeps, the x-z
            means and their time average every step, the monitor line at the end of the stretch; default variants.
  stream    independent field sets stepped once each through the asynchronous transfer calls.
  ensemble  several uneven channels advanced together.
  explicit  main domain with explicit viscous terms and non-uniform properties.
  heated    main domain with Crank-Nicolson viscous terms and the energy equation; properties by the table search or
            by the learned model.
  open      main domain with inflow and outflow, fed by a periodic channel.

Grids are those of the benchmark, the configurations and the tests, and others between them: every length is one of the
seven that the library takes.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chapsim1.0_b200"))

from chapsim import gpu, thermo  # noqa: E402
from chapsim.mesh import channel_setup, xinout_setup  # noqa: E402

DTMIN, CFLGV, STR2 = 1e-6, 0.5, 2.0
LENGTHS = (32, 64, 96, 128, 192, 256, 384)
MIXED_TUNE = 64 | 256 | 1024 | 2048  # scan y-solve, 16-line z tiles, line pairs in the z and y sweeps
PLANE = 8                            # fused plane transforms


def listed():
    return [
        # the smallest grid, driven call by call with the statistics on: launches and latency
        {"name": "driver_32", "kind": "driver", "L": 32, "M": 32, "N": 32, "steps": 10},
        # the small validation channel, a stretch of steps at once
        {"name": "channel_64", "kind": "channel", "L": 64, "M": 64, "N": 64, "steps": 50, "precision": "fp64", "tune": -1},
        # the Re_tau 180 channel in both precisions
        {"name": "channel_128", "kind": "channel", "L": 128, "M": 128, "N": 128, "steps": 30, "precision": "fp64",
         "tune": -1},
        {"name": "channel_128_mixed", "kind": "channel", "L": 128, "M": 128, "N": 128, "steps": 30,
         "precision": "mixed", "tune": MIXED_TUNE | PLANE},
        # a grid of three different lengths, two of them no power of two
        {"name": "channel_192x256x96", "kind": "channel", "L": 192, "M": 256, "N": 96, "steps": 15,
         "precision": "fp64", "tune": -1},
        # the Re_tau 395 channel: the headline workload, in both precisions
        {"name": "channel_384", "kind": "channel", "L": 384, "M": 256, "N": 384, "steps": 10, "precision": "fp64",
         "tune": -1},
        {"name": "channel_384_mixed", "kind": "channel", "L": 384, "M": 256, "N": 384, "steps": 10,
         "precision": "mixed", "tune": MIXED_TUNE},
        # field sets streamed through host memory, one step each
        {"name": "stream_192", "kind": "stream", "L": 192, "M": 128, "N": 192, "steps": 4},
        # uneven channels of a parameter study, advanced together
        {"name": "ensemble_6", "kind": "ensemble", "members": "64x64x64 96x64x128 128x128x64 96x96x96 192x64x96 192x128x192",
         "steps": 10},
        # the heated main domain in FP64 with the table search, and in mixed precision with the learned model
        {"name": "heated_256", "kind": "heated", "L": 256, "M": 192, "N": 128, "steps": 10, "precision": "fp64",
         "learned": False},
        {"name": "heated_128_learned", "kind": "heated", "L": 128, "M": 96, "N": 128, "steps": 10,
         "precision": "mixed", "learned": True},
        # a developing flow: a periodic channel feeds a main domain twice its length; explicit viscous terms
        {"name": "open_256", "kind": "open", "LT": 128, "L": 256, "M": 128, "N": 128, "steps": 10},
    ]


def draw(rng):
    kind = rng.choice(["channel"] * 6 + ["driver", "stream", "ensemble", "explicit", "heated", "heated", "open"])
    most = {"channel": 384 * 256 * 384, "driver": 1 << 21, "stream": 1 << 23, "ensemble": 1 << 21, "explicit": 1 << 23,
            "heated": 1 << 23, "open": 1 << 22}[kind]

    def grid(most):
        want = math.exp(rng.uniform(math.log(32.0 ** 3), math.log(float(most))))
        every = [(l, m, n) for l in LENGTHS for m in LENGTHS for n in LENGTHS
                 if 0.5 * want <= l * m * n <= min(2.0 * want, most) and max(l, m, n) <= 6 * min(l, m, n)]
        return rng.choice(every or [(32, 32, 32)])

    L, M, N = grid(most)
    steps = max(4, min(40, int(6e7 / (L * M * N))))
    c = {"kind": kind, "L": L, "M": M, "N": N, "steps": steps}
    if kind == "channel":
        c["precision"] = rng.choice(["fp64", "fp64", "mixed"])
        plane = PLANE if 64 <= min(L, N) and max(L, N) <= 192 else 0
        c["tune"] = -1 if c["precision"] == "fp64" else MIXED_TUNE | plane
    elif kind == "stream":
        c["steps"] = 4
    elif kind == "ensemble":
        c = {"kind": kind, "steps": steps, "members": " ".join("%dx%dx%d" % grid(most) for _ in range(rng.randint(2, 6)))}
    elif kind == "heated":
        c["precision"], c["learned"] = rng.choice([("fp64", False), ("fp64", True), ("mixed", False), ("mixed", True)])
        c["steps"] = min(steps, 10)
    elif kind == "open":
        c["LT"], c["steps"] = rng.choice([64, 96, 128]), min(steps, 10)
    return c


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _members(case):
    if case["kind"] == "ensemble":
        return [tuple(int(v) for v in m.split("x")) for m in case["members"].split()]
    return [(case.get("LT", case["L"]), case["M"], case["N"])]


def _flow_parameters(L, M, N):
    """Domain and Reynolds number of the benchmark's channels: (HX, HZ, REN, DT0)."""
    if L * M * N > 1 << 23:
        return 2 * math.pi, math.pi, 6875.0, 0.05
    return 4 * math.pi, 4 * math.pi / 3, 2800.0, 0.05


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _start_field(L, M, N, seed):
    """Perturbed Poiseuille flow of unit bulk velocity, before its projection: Q (3, N, M + 2, L), made from the seed."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(int(seed))
    Q = torch.zeros((3, N, M + 2, L), dtype=torch.float64, device=dev)
    Q[:, :, 1:M + 1] = 0.1 * (2.0 * torch.rand((3, N, M, L), generator=g, dtype=torch.float64, device=dev) - 1.0)
    Q[1, :, 1] = 0.0
    Q[:, :, 1:M + 1] -= Q[:, :, 1:M + 1].mean(dim=(1, 3), keepdim=True)
    y = torch.tanh(STR2 * (torch.arange(M + 1, dtype=torch.float64, device=dev) / M - 0.5)) / math.tanh(0.5 * STR2)
    u = 1.5 * (1.0 - (0.5 * (y[1:] + y[:-1])) ** 2)
    Q[0, :, 1:M + 1] += (u * 2.0 / (u * (y[1:] - y[:-1])).sum())[None, :, None]
    return Q


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _p(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _channel(L, M, N, seed, precision="fp64"):
    """A periodic-channel context with the seed's projected start field."""
    HX, HZ, REN, DT0 = _flow_parameters(L, M, N)
    ch = gpu.ChannelTG(channel_setup(L, M, N, HX, HZ, STR2, REN), precision=precision)
    ch.upload(_start_field(L, M, N, seed).cpu().numpy(), np.zeros(ch.field_shape()))
    ch.set_dt(DT0)
    ch.SOLVERRK3_MOM_tg(0)
    return ch


def _buffers(ch, n=1):
    s = ch.field_shape()
    return [(_pinned(3, *s), _pinned(*s)) for _ in range(n)]


def _last_layer(table, x_lo, x_hi, off, scale, seed=11):
    """Weights of the 1-64-64-6 property model: seeded hidden layers, the output layer fitted to the table."""
    r = np.random.default_rng(seed)
    w1, b1 = r.uniform(-6.0, 6.0, 64), r.uniform(-4.0, 4.0, 64)
    w2, b2 = r.uniform(-0.35, 0.35, (64, 64)), r.uniform(-0.5, 0.5, 64)
    li = table.lists
    keep = (li["DH"] >= x_lo) & (li["DH"] <= x_hi)
    x = 2.0 * (li["DH"][keep] - x_lo) / (x_hi - x_lo) - 1.0
    h = np.tanh(np.tanh(x[:, None] * w1 + b1) @ w2.T + b2)
    # the reference's assignment: the density takes the viscosity's spline, and so on round
    y = np.stack([li[n][keep] for n in ("H", "T", "M", "K", "D", "CP")], axis=1)
    A = np.concatenate([h, np.ones((h.shape[0], 1))], axis=1)
    w = np.linalg.solve(A.T @ A + 1e-4 * np.eye(65), A.T @ ((y - off) / scale))
    return np.concatenate([w1, b1, w2.reshape(-1), b2, w[:64].T.reshape(-1), w[64]]).astype(np.float32)


def _heated(case, seed):
    L, M, N = case["L"], case["M"], case["N"]
    HX, HZ, REN, _ = _flow_parameters(L, M, N)
    dt, qw = 1e-3, 0.5
    rows, T0 = thermo.synthetic_table()
    table = thermo.SplineTable.from_rows(rows, T0)
    ch = gpu.ChannelIO(channel_setup(L, M, N, HX, HZ, STR2, REN), ivisscheme=gpu.VIS_IMPLICIT, precision=case["precision"])
    ones = np.ones(ch.field_shape())
    ch.upload_io(_start_field(L, M, N, seed).cpu().numpy(), np.zeros(ch.field_shape()), ones, ones, ones)
    ch.set_dt(dt)
    DH = np.zeros(ch.field_shape())
    DH[:, 1:M + 1] = 1e-3 * np.random.default_rng(seed).uniform(-1.0, 1.0, (N, M, L))
    ch.thermal_init(table, DH, qw, qw, 1.0 / REN / (table.ref["M0"] * table.ref["CP0"] / table.ref["K0"]))
    if case["learned"]:
        dh = table.lists["DH"]
        ch.mlp_init(float(dh[0] + 0.02 * (dh[-1] - dh[0])), float(dh[-1] - 0.02 * (dh[-1] - dh[0])), seed=11)
        _, norm = ch.mlp_params()
        ch.mlp_set_params(_last_layer(table, norm[0], norm[1], norm[2:8], norm[8:14]))
        ch.thermal_use_mlp(True)
    return ch, dt


def _explicit(case, seed):
    """Main domain of non-uniform density and viscosity (the waves' phases from the seed), explicit viscous terms."""
    L, M, N = case["L"], case["M"], case["N"]
    HX, HZ, REN, _ = _flow_parameters(L, M, N)
    ch = gpu.ChannelIO(channel_setup(L, M, N, HX, HZ, STR2, REN), ivisscheme=gpu.VIS_EXPLICIT)
    a, b, c = np.random.default_rng(seed).uniform(0.0, 2 * math.pi, 3)
    k, j, i = np.meshgrid(np.arange(N), np.arange(M + 2), np.arange(L), indexing="ij", sparse=True)
    rho = 1.0 + 0.05 * np.sin(2 * np.pi * i / L + a) * np.cos(2 * np.pi * k / N + b) + 0.02 * np.cos(np.pi * j / M)
    mu0 = 1.0 + 0.1 * np.cos(2 * np.pi * i / L + c) * np.sin(np.pi * j / M) + 0.0 * k
    mu = mu0 * (1.0 + 0.03 * np.sin(2 * np.pi * k / N + a))
    ch.upload_io(_start_field(L, M, N, seed).cpu().numpy(), np.zeros(ch.field_shape()), rho, mu0, mu)
    ch.set_dt(1e-3)
    return ch, 1e-3


def _open(case, seed):
    LT, L, M, N = case["LT"], case["L"], case["M"], case["N"]
    HX, HZ, REN, _ = _flow_parameters(LT, M, N)
    tg = _channel(LT, M, N, seed)
    Q, _PR = tg.download()
    io = gpu.ChannelXinout(xinout_setup(L, M, N, L * HX / LT, HZ, STR2, REN), tg=tg)
    G = np.ascontiguousarray(Q[:, :, :, [(i - 1) % LT for i in range(L + 2)]])
    ones = np.ones(io.field_shape())
    io.upload_io(G, np.zeros(io.field_shape()), ones, ones, ones)
    io.set_dt(0.01)
    return io, tg, 0.01


def prepare(case, seed):
    kind, s = case["kind"], {"case": case, "kind": case["kind"], "steps": case["steps"]}
    if kind in ("channel", "driver", "stream"):
        L, M, N = case["L"], case["M"], case["N"]
        s["ch"] = ch = _channel(L, M, N, seed, case.get("precision", "fp64"))
        s["DT0"], s["REN"] = _flow_parameters(L, M, N)[3], ch.s.REN
        if kind == "channel":
            ch.autotune(case["tune"])
        s["out"] = _buffers(ch, case["steps"] if kind == "stream" else 1)
        if kind == "stream":
            s["in"] = _buffers(ch, case["steps"])
            for k, (q, p) in enumerate(s["in"]):
                q[...], p[...] = _start_field(L, M, N, seed + 7919 * k).cpu().numpy(), 0.0
    elif kind == "ensemble":
        s["ch"] = [_channel(*m, seed + 7919 * k) for k, m in enumerate(_members(case))]
        for ch in s["ch"]:
            ch.autotune()
        s["group"] = gpu.Ensemble(s["ch"])
        s["DT0"] = 0.05
        s["out"] = [_buffers(ch)[0] for ch in s["ch"]]
    elif kind == "open":
        s["ch"], s["tg"], s["DT0"] = _open(case, seed)
        s["tg_out"] = _buffers(s["tg"])[0]
    else:
        s["ch"], s["DT0"] = (_heated if kind == "heated" else _explicit)(case, seed)
    if kind in ("open", "heated", "explicit"):
        f = s["ch"].field_shape()
        s["out"] = (_pinned(3, *f), _pinned(3, *f), _pinned(*f))
        s["thermal"] = [_pinned(*f) for _ in range(7)] if kind == "heated" else []
    return s


# ---- one pass -------------------------------------------------------------------------------------------------------

def run(s):
    kind, ch, n, DT0 = s["kind"], s["ch"], s["steps"], s["DT0"]
    if kind == "channel":
        ch.advance(n, DT0, DTMIN, CFLGV)
        ch.download_async(*s["out"][0])
        ch.io_wait()
        return {"Q": s["out"][0][0], "PR": s["out"][0][1]}
    if kind == "driver":
        for _ in range(n):
            dt, _cfl = ch.step_begin(DT0, DTMIN, CFLGV)
            for NS in (1, 2, 3):
                ch.SOLVERRK3_MOM_tg(NS)
            ch.PP_MEAN_ZX_FLOW_TG()
            ch.PP_MEAN_T_TG()
        mon = ch.PP_MONITOR_TG(s["REN"])
        means, _count = ch.download_pp_means(averaged=True)
        ch.download_async(*s["out"][0])
        ch.io_wait()
        return {"Q": s["out"][0][0], "PR": s["out"][0][1], "dt": dt, "means": means,
                "monitor": np.array([mon[k] for k in gpu.PP_MONITOR])}
    if kind == "stream":
        ch.set_dt(DT0)
        ch.upload_async(*s["in"][0])
        for k in range(n):
            if k + 1 < n:
                ch.upload_async(*s["in"][k + 1])
            ch.advance(1, DT0, DTMIN, CFLGV)
            ch.download_async(*s["out"][k])
        ch.io_wait()
        return {"Q%d" % k: q for k, (q, p) in enumerate(s["out"])} | {"PR%d" % k: p for k, (q, p) in enumerate(s["out"])}
    if kind == "ensemble":
        s["group"].advance(n, DT0, DTMIN, CFLGV)
        for c, (q, p) in zip(ch, s["out"]):
            c.download_async(q, p)
        for c in ch:
            c.io_wait()
        return {"Q%d" % k: q for k, (q, p) in enumerate(s["out"])} | {"PR%d" % k: p for k, (q, p) in enumerate(s["out"])}
    ch.advance(n, DT0, DTMIN, CFLGV)
    G, Q, PR = s["out"]
    ch._check(ch.lib.chapsim_download_io_fields(ch.h, _p(G), _p(Q), _p(PR)))
    got = {"G": G, "Q": Q, "PR": PR}
    if kind == "heated":
        ch._check(ch.lib.chapsim_download_thermal_fields(ch.h, *[_p(a) for a in s["thermal"]]))
        got |= dict(zip(("DH", "H", "T", "D", "M", "K", "CP"), s["thermal"]))
    if kind == "open":
        s["tg"].download_async(*s["tg_out"])
        s["tg"].io_wait()
        got |= {"TQ": s["tg_out"][0], "TPR": s["tg_out"][1]}
    return got


def work(case):
    """Each substep reads the fields that it starts from and writes those that it leaves, once; the operations are those
    of the stencils, the line solves and the transforms per point."""
    word = 4 if case.get("precision") == "mixed" else 8
    pts = sum(l * m * n for l, m, n in _members(case))
    fft = 2.5 * 2 * math.log2(max(64, pts ** (2 / 3)))  # forward and inverse, x and z, real data
    bytes_, flops = pts * word * 14, pts * (260 + fft)  # Q, PR, CONVH0 in and out
    if case["kind"] in ("open", "explicit", "heated"):
        own = case["L"] * case["M"] * case["N"]
        flow = (24 if case["kind"] == "open" else 22)  # G, Q, PR, EXPLT0 in and out, and the properties
        heat = 18 if case["kind"] == "heated" else 0    # DH and its old right-hand side in and out, the properties out
        bytes_ = (bytes_ if case["kind"] == "open" else 0) + own * (word * flow + 8 * heat)
        flops = (flops if case["kind"] == "open" else 0) + own * (500 + fft + (300 if heat else 0))
    return {"bytes": 3.0 * case["steps"] * bytes_, "flops": 3.0 * case["steps"] * flops}


# ---- the periodic channel's step in plain torch, 64 bits ------------------------------------------------------------

class _Exact:
    """The fractional-step RK3 of the periodic channel on dense operators: spectral solves in x and z, inverse matrices
    in y. Fields are (N, rows, L)."""

    def __init__(self, L, M, N):
        self.L, self.M, self.N = L, M, N
        HX, HZ, REN, self.DT0 = _flow_parameters(L, M, N)
        dev = self.dev = _device()
        self.nu = 1.0 / REN
        self.dxi, self.dzi = L / HX, N / HZ
        y = np.tanh(STR2 * (np.arange(M + 1) / M - 0.5)) / math.tanh(0.5 * STR2)  # faces
        yc = 0.5 * (y[1:] + y[:-1])                                               # centres
        fi = 1.0 / (y[1:] - y[:-1])                                               # rows 1..M
        ci = np.concatenate([[2.0 / (y[1] - y[0])], 2.0 / (y[2:] - y[:-2]), [2.0 / (y[M] - y[M - 1])]])  # faces 1..M+1
        wff = np.concatenate([[0.0], (y[1:M] - yc[:-1]) / (yc[1:] - yc[:-1]), [1.0]])
        self.vol = 2.0 * L * N
        row = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)[None, :, None]  # noqa: E731
        self.fi, self.ci, self.wf, self.wb = row(fi), row(ci), row(wff), row(1.0 - wff)
        # second y derivative of u and w (one-sided at the walls), of v, and of the pressure
        lo, up = fi * ci[:-1], fi * ci[1:]
        a = np.diag(-(lo + up)) + np.diag(lo[1:], -1) + np.diag(up[:-1], 1)
        b = 4.0 / (2.0 / ci[1] + 1.0 / fi[0])
        a[0, 0], a[0, 1] = -b * (ci[1] + 2.0 * fi[0]), b * ci[1]
        b = 4.0 / (2.0 / ci[M - 1] + 1.0 / fi[M - 1])
        a[M - 1, M - 1], a[M - 1, M - 2] = -b * (2.0 * fi[M - 1] + ci[M - 1]), b * ci[M - 1]
        lov, upv = np.concatenate([[0.0], fi[:-1] * ci[1:M]]), np.concatenate([[0.0], fi[1:] * ci[1:M]])
        cv = np.concatenate([[1.0], -(lov + upv)[1:]])
        v = np.diag(cv) + np.diag(lov[1:], -1) + np.diag(upv[:-1], 1)
        self.dyy = [torch.tensor(m, dtype=torch.float64, device=dev) for m in (a, v, a)]
        lo[0], up[-1] = 0.0, 0.0
        self.plo, self.pup, self.pc = lo.tolist(), up.tolist(), (-(lo + up)).tolist()
        kx = 2.0 * (1.0 - np.cos(2 * np.pi * np.arange(L // 2 + 1) / L)) * self.dxi ** 2
        kz = 2.0 * (1.0 - np.cos(2 * np.pi * np.arange(N) / N)) * self.dzi ** 2
        self.kx = torch.tensor(kx, dtype=torch.float64, device=dev)[None, None, :]
        self.kz = torch.tensor(kz, dtype=torch.float64, device=dev)[:, None, None]

    @staticmethod
    def d(a, axis, n):
        """The neighbour n further along a periodic axis."""
        return torch.roll(a, -n, axis)

    def convection(self, Q):
        M, d = self.M, self.d
        (u, v, w), (uP, vP, wP), (uM, vM, wM) = [[q[:, o:o + M] for q in Q] for o in (1, 2, 0)]
        f, b, fP, bP = self.wf[:, :M], self.wb[:, :M], self.wf[:, 1:], self.wb[:, 1:]
        xp, xm, zp, zm = (lambda a: d(a, 2, 1)), (lambda a: d(a, 2, -1)), (lambda a: d(a, 0, 1)), (lambda a: d(a, 0, -1))
        x4, x2, z4, z2, c4 = self.dxi / 4, self.dxi / 2, self.dzi / 4, self.dzi / 2, self.ci[:, :M] / 4
        cx = (((xp(u) + u) ** 2 - (xm(u) + u) ** 2) * x4
              + ((vP + xm(vP)) * (fP * uP + bP * u) - (v + xm(v)) * (f * u + b * uM)) * self.fi / 2
              + ((zp(w) + xm(zp(w))) * (zp(u) + u) - (w + xm(w)) * (u + zm(u))) * z4)
        yu, yw = f * u + b * uM, f * w + b * wM
        cy = ((xp(yu) * (xp(v) + v) - yu * (v + xm(v))) * x2 + ((vP + v) ** 2 - (v + vM) ** 2) * c4
              + (zp(yw) * (zp(v) + v) - yw * (v + zm(v))) * z2)
        cz = ((xp(u + zm(u)) * (xp(w) + w) - (u + zm(u)) * (w + xm(w))) * x4
              + ((vP + zm(vP)) * (fP * wP + bP * w) - (v + zm(v)) * (f * w + b * wM)) * self.fi / 2
              + ((zp(w) + w) ** 2 - (w + zm(w)) ** 2) * z4)
        return -cx, -cy, -cz

    def substep(self, ns):
        M, d = self.M, self.d
        gam = (1.0, 8 / 15, 5 / 12, 3 / 4)[ns]
        rho = (0.0, 0.0, -17 / 60, -5 / 12)[ns]
        al = (gam + rho) * self.dt
        Q, P = self.Q, self.P
        conv = self.convection(Q)
        left, add = None, []
        for c in range(3):
            q, p = Q[c][:, 1:M + 1], P[:, 1:M + 1]
            lap = ((d(q, 2, 1) - 2 * q + d(q, 2, -1)) * self.dxi ** 2 + (d(q, 0, 1) - 2 * q + d(q, 0, -1)) * self.dzi ** 2
                   + self.dyy[c] @ q)
            grad = ((p - d(p, 2, -1)) * self.dxi, (p - P[:, 0:M]) * self.ci[:, :M], (p - d(p, 0, -1)) * self.dzi)[c]
            r = (gam * conv[c] + rho * self.H[c]) * self.dt + al * (self.nu * lap - grad)
            if c == 0:
                r = r - (r / self.fi).sum() / self.vol
            self.H[c] = conv[c]
            F = 0.5 * al * self.nu
            s = torch.fft.rfftn(r, dim=(0, 2)) / ((1 + F * self.kx) * (1 + F * self.kz))
            r = torch.fft.irfftn(s, s=(self.N, self.L), dim=(0, 2))
            if c == 1:
                r[:, 0] = left  # the wall row still holds the u increment of the same substep
            m = torch.eye(M, dtype=torch.float64, device=self.dev) - F * self.dyy[c]
            r = torch.linalg.inv(m) @ r
            if c == 0:
                left = r[:, 0].clone()
            add.append(r)
        for c in range(3):
            first = 1 if c == 1 else 0  # v on the wall face stays
            Q[c][:, 1 + first:M + 1] += add[c][:, first:]
        div = (((d(Q[0], 2, 1) - Q[0]) * self.dxi + (d(Q[2], 0, 1) - Q[2]) * self.dzi)[:, 1:M + 1]
               + (Q[1][:, 2:M + 2] - Q[1][:, 1:M + 1]) * self.fi) / al
        phi = torch.zeros_like(P)
        phi[:, 1:M + 1] = self.poisson(div)
        phi[:, 0], phi[:, M + 1] = phi[:, 1], phi[:, M]
        Q[0][:, 1:M + 1] -= al * self.dxi * (phi - d(phi, 2, -1))[:, 1:M + 1]
        Q[2][:, 1:M + 1] -= al * self.dzi * (phi - d(phi, 0, -1))[:, 1:M + 1]
        Q[1][:, 2:M + 1] -= al * self.ci[:, 1:M] * (phi[:, 2:M + 1] - phi[:, 1:M])
        P[:, 1:M + 1] += phi[:, 1:M + 1] - 0.5 * al * self.nu * div
        P[:, 0], P[:, M + 1] = P[:, 1], P[:, M]

    def poisson(self, div):
        M = self.M
        s = torch.fft.rfftn(div, dim=(0, 2))
        s[0, 0, 0] = 0.0  # the constant mode is fixed by its first row
        k = (self.kx + self.kz)[:, 0]
        h, first = [], torch.ones_like(k)
        first[0, 0] = 0.0
        piv = self.pc[0] - k
        up = self.pup[0] * first
        for j in range(M):
            if j:
                piv = self.pc[j] - k - self.plo[j] * h[-1]
                up = self.pup[j]
                s[:, j] = (s[:, j] - self.plo[j] * s[:, j - 1]) / piv
            else:
                piv[0, 0] = 1.0
                s[:, 0] = s[:, 0] / piv
            h.append(up / piv)
        for j in range(M - 2, -1, -1):
            s[:, j] = s[:, j] - h[j] * s[:, j + 1]
        return torch.fft.irfftn(s, s=(self.N, self.L), dim=(0, 2))

    def step(self):
        M, d, (u, v, w) = self.M, self.d, self.Q
        c = (((u + d(u, 2, 1)).abs() * self.dxi + (w + d(w, 0, 1)).abs() * self.dzi)[:, 1:M + 1]
             + (v[:, 1:M + 1] + v[:, 2:M + 2]).abs() * self.fi)
        self.dt = max(min(self.DT0, 5 * self.dt, CFLGV / (0.5 * float(c.max()))), DTMIN)
        for ns in (1, 2, 3):
            self.substep(ns)

    def start(self, Q, project=True):
        self.Q, self.P, self.dt = Q.clone(), torch.zeros_like(Q[0]), self.DT0
        self.H = [torch.zeros_like(Q[0][:, 1:self.M + 1]) for _ in range(3)]
        if project:
            self.substep(0)
        return self

    def advance(self, n):
        for _ in range(n):
            self.step()
        return self.Q, self.P


def exact(case, seed):
    """Q and PR of the periodic channels after one pass. None for the main domains: their step has no form that plain
    torch would run in seconds (per-point coefficients in every line solve); statistics of the driver are left out."""
    kind = case["kind"]
    if kind in ("heated", "explicit", "open"):
        return None
    if kind == "stream":
        got, (l, m, n) = {}, _members(case)[0]
        e = _Exact(l, m, n)
        dt = e.DT0
        for k in range(case["steps"]):
            e.start(_start_field(l, m, n, seed + 7919 * k), project=False)
            e.dt = dt  # the time step follows on from set to set
            got["Q%d" % k], got["PR%d" % k] = e.advance(1)
            dt = e.dt
        return got
    outs = []
    for k, (l, m, n) in enumerate(_members(case)):
        e = _Exact(l, m, n).start(_start_field(l, m, n, seed + 7919 * k))
        outs.append(e.advance(case["steps"]))
    if kind == "ensemble":
        return {"Q%d" % k: q for k, (q, p) in enumerate(outs)} | {"PR%d" % k: p for k, (q, p) in enumerate(outs)}
    got = {"Q": outs[0][0], "PR": outs[0][1]}
    if kind == "driver":
        got |= {"dt": e.dt, "means": None, "monitor": None}
    return got
