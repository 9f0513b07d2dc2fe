"""The work that the performance of this framework is judged on: the time step
on its grids and precisions, the hydrostatic columns every run starts from, a
batched parameter sweep, the Poisson solve on a caller's own device arrays, and
the Fourier neural operator's forward pass and training step.

A case is a dict of plain values; `prepare` makes its inputs on the GPU from a
seed, `run` is one pass through the public entry points, `work` the bytes and
operations one pass cannot do without, and `exact` the same outputs from plain
torch in 64 bits.

Steps start from a convecting state: a charge profile that falls from the
injector to the collector, modulated by rolls in x and y, and the velocity of
such rolls plus seeded noise, so that every component of every field carries
more than round-off.  A pass advances the state it finds by `steps` time steps
and reads the nine fields back, as a run does between two records; a run keeps
its records at the precision it computes in (FP64 and FP32 runs) or stores its
populations in (16-bit runs).
"""
import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parents[1] / "ehd-convection-3d_b200"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))

import ehd  # noqa: E402
import fno  # noqa: E402
import sweep  # noqa: E402

FIELDS = ("rho", "u", "v", "w", "q", "phi", "ex", "ey", "ez")
RECORD = {"fp64": torch.float64, "fp32": torch.float32, "fp16": torch.float16,
          "bf16": torch.float16, "mixed": torch.float16}
POP_BYTES = {"fp64": (8, 8), "fp32": (4, 4), "fp16": (2, 2), "bf16": (2, 2), "mixed": (2, 4)}


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # the hydrostatic column (1 x 1 x NZ, FP64) that fixes I0 and the start
        # of every run: tens of thousands of steps of a few nodes, until the
        # charge has crossed the gap (runs take 4 to 16 such transits)
        {"name": "column_33", "kind": "column", "count": 1, "nz": 33, "transits": 1.25},
        # the same for the instances of a sweep at once
        {"name": "columns_12x25", "kind": "column", "count": 12, "nz": 25, "transits": 1.25},
        # the 64 x 64 x 33 grid of the 2,000-step comparison with the
        # reference (FP64) and of the neural operator's trajectories (FP32)
        {"name": "step_fp64_64x64x33", "kind": "step", "nx": 64, "ny": 64, "nz": 33,
         "precision": "fp64", "T": 200.0, "steps": 200},
        {"name": "step_fp32_64x64x33", "kind": "step", "nx": 64, "ny": 64, "nz": 33,
         "precision": "fp32", "T": 200.0, "steps": 200},
        # the reference's own default grid, whose runs to saturated Nu_e take
        # a million steps; 122 = 2 x 61 is no size of a power of two
        {"name": "step_fp32_122x122x101", "kind": "step", "nx": 122, "ny": 122, "nz": 101,
         "precision": "fp32", "T": 996.0, "steps": 150},
        # the benchmark's grid in the reference's precision and in FP32
        {"name": "step_fp64_256x256x129", "kind": "step", "nx": 256, "ny": 256, "nz": 129,
         "precision": "fp64", "T": 200.0, "steps": 150},
        {"name": "step_fp32_256x256x129", "kind": "step", "nx": 256, "ny": 256, "nz": 129,
         "precision": "fp32", "T": 200.0, "steps": 300},
        # the fine grid that takes a warm start, in 16-bit storage
        {"name": "step_fp16_512x512x129", "kind": "step", "nx": 512, "ny": 512, "nz": 129,
         "precision": "fp16", "T": 300.0, "steps": 100},
        # a share of the T sweep: uneven grids stepped as one batch
        {"name": "sweep_fp32_24", "kind": "batch", "count": 24, "nz_lo": 24, "nz_hi": 48,
         "precision": "fp32", "steps": 100},
        # the Poisson solve and E field inside another code's step, on its own
        # device arrays
        {"name": "poisson_noalloc_96x96x65", "kind": "noalloc", "nx": 96, "ny": 96, "nz": 65},
        # the warm start's network: prediction and one training step
        {"name": "fno_forward_b4", "kind": "fno", "train": False, "nx": 64, "ny": 64, "nz": 33,
         "batch": 4, "width": 32, "layers": 4, "modes": 12, "hidden": 128},
        {"name": "fno_train_b4", "kind": "fno", "train": True, "nx": 64, "ny": 64, "nz": 33,
         "batch": 4, "width": 32, "layers": 4, "modes": 12, "hidden": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same kinds: steps (three in five of the draws) on
    grids from 16 x 16 x 9 to 512 wide, any width among them, in every
    precision; columns, sweeps, Poisson solves and networks of other sizes."""
    r = rng.random()
    if r < 0.6:
        while True:
            nx = _log_int(rng, 16, 512)
            # planes are square or nearly so in most runs
            ny = nx if rng.random() < 0.5 else min(512, max(16, int(nx * rng.uniform(0.5, 2.0))))
            nz = _log_int(rng, 9, 161)
            if nx * ny * nz <= 9_000_000:
                break
        prec = rng.choice(["fp32", "fp32", "fp64", "mixed", "fp16", "bf16"])
        steps = max(20, min(200, int(2.0e8 / (nx * ny * nz))))
        return {"kind": "step", "nx": nx, "ny": ny, "nz": nz, "precision": prec,
                "T": round(rng.uniform(150.0, 400.0), 1), "steps": steps}
    if r < 0.7:
        if rng.random() < 0.6:
            return {"kind": "column", "count": 1, "nz": _log_int(rng, 9, 65), "transits": 1.25}
        return {"kind": "column", "count": rng.randint(2, 12), "nz": _log_int(rng, 9, 25),
                "transits": 1.25}
    if r < 0.78:
        lo = rng.randint(16, 32)
        return {"kind": "batch", "count": rng.randint(2, 16), "nz_lo": lo,
                "nz_hi": rng.randint(lo, 48), "precision": rng.choice(["fp32", "fp32", "fp64", "mixed"]),
                "steps": rng.randint(30, 100)}
    if r < 0.86:
        smooth = [n for n in range(16, 161) if _smooth(n)]
        while True:
            nx, ny, nz = rng.choice(smooth), rng.choice(smooth), _log_int(rng, 9, 129)
            # the working storage the entry point has
            if ((nx // 2 + 16) * 16 + (nx // 2 + 1) * 24 + 16) * ny * nz < 62_000_000:
                return {"kind": "noalloc", "nx": nx, "ny": ny, "nz": nz}
    nx, ny, nz = (rng.randint(16, 72) for _ in range(3))
    modes = rng.randint(3, min(12, nx // 2 - 1, ny // 2, nz // 2))
    return {"kind": "fno", "train": r >= 0.93, "nx": nx, "ny": ny, "nz": min(nz, 48),
            "batch": rng.randint(1, 4), "width": rng.choice([8, 16, 24, 32]),
            "layers": rng.randint(2, 4), "modes": min(modes, min(nz, 48) // 2),
            "hidden": rng.choice([32, 64, 128])}


def _smooth(n):
    for f in (2, 3, 5):
        while n % f == 0:
            n //= f
    return n == 1


# ---- inputs ------------------------------------------------------------------

# the reference's own magic parameters, M, C and Fe (the sweeps')
LAMBDA_F, LAMBDA_G, M_GROUP, C_GROUP, FE_GROUP = 1.0 / 12.0, 1.0e-6, 10.0, 10.0, 4000.0
RHO0, VOLTAGE, EPS, CFL = 1600.0, 1.0e4, 1.0e-4, 0.01


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _params(nx, ny, nz, T):
    dz = 1.0 / (nz - 1)
    return ehd.params_from_groups(nx, ny, nz, nx * dz, ny * dz, T=T, M=M_GROUP, C=C_GROUP,
                                  Fe=FE_GROUP, lambda_f=LAMBDA_F, lambda_g=LAMBDA_G, cfl=CFL)


def _start(nx, ny, nz, seed):
    """The nine FP64 fields of the convecting start, [z][y][x] tensors."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(int(seed))
    f64 = dict(dtype=torch.float64, device=dev)

    def rnd(*shape):
        return torch.rand(shape, generator=g, **f64)

    z = torch.arange(nz, **f64)[:, None, None] / (nz - 1)
    y = torch.arange(ny, **f64)[None, :, None] / ny * (2 * math.pi)
    x = torch.arange(nx, **f64)[None, None, :] / nx * (2 * math.pi)
    c = rnd(8).tolist()
    px, py, qx, qy = (2 * math.pi * v for v in c[:4])
    amp = 0.1 + 0.1 * c[4]
    ax, ay = 0.5 + c[5], 0.5 + c[6]
    cell = ax * torch.cos(x + px) + ay * torch.cos(y + py) + 0.3 * torch.cos(x + qx) * torch.sin(y + qy)
    up, side = torch.sin(math.pi * z), torch.sin(2 * math.pi * z)
    noise = 2.0 * rnd(3, nz, ny, nx) - 1.0
    inside = torch.ones(nz, 1, 1, **f64)
    inside[0] = 0.0
    inside[-1] = 0.0
    zero = torch.zeros(nz, ny, nx, **f64)
    q0 = C_GROUP * VOLTAGE * EPS
    out = {
        "rho": zero + RHO0,
        "u": (amp * ax * side * torch.sin(x + px) + 1e-3 * noise[0]) * inside,
        "v": (amp * ay * side * torch.sin(y + py) + 1e-3 * noise[1]) * inside,
        "w": (amp * up * cell + 1e-3 * noise[2]) * inside,
        "q": q0 / torch.sqrt(1.0 + 6.0 * z) * (1.0 + 0.15 * up * cell),
        "phi": zero + VOLTAGE * (1.0 - z),
        "ex": zero, "ey": zero, "ez": zero + VOLTAGE,
    }
    return {k: v.contiguous() for k, v in out.items()}


def _ptr(t):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))


def _column_groups(case, seed):
    """T of each column of a case."""
    rng = np.random.default_rng([11, seed])
    return [float(t) for t in rng.uniform(150.0, 400.0, case["count"])]


def _column_steps(case):
    """Steps of `transits` times the charge's transit time Lz^2 / (K V), even."""
    K = math.sqrt(EPS / RHO0) / M_GROUP
    n = int(round(case["transits"] / (K * VOLTAGE) * (case["nz"] - 1) / CFL))
    return n + (n & 1)


def _sweep_instances(case, seed):
    """(nx, ny, nz, T, seed) of each instance of a batch: the sweep's uneven
    grids, nz cells and 2 nz by 2 nz columns (the grids are the case's, the
    groups and starts the seed's)."""
    cells = np.linspace(case["nz_lo"], case["nz_hi"], 4).round().astype(int) // 8 * 8
    cells = [max(8, int(c)) for c in cells]
    rng = np.random.default_rng([12, seed])
    return [(2 * cells[i % 4], 2 * cells[i % 4], cells[i % 4] + 1, float(rng.uniform(100.0, 400.0)),
             int(seed) * 1000 + i) for i in range(case["count"])]


def _fno_config(case):
    m = case["modes"]
    return dict(nx=case["nx"], ny=case["ny"], nz=case["nz"], in_channels=9, out_channels=5,
                width=case["width"], layers=case["layers"], modes=(m, m, m),
                hidden=case["hidden"], max_batch=case["batch"])


def _fno_inputs(case, seed):
    """Network input, target and flat FP32 weights (the initial
    distributions of the product) from a seed, on the device."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(int(seed))
    B, Z, Y, X = case["batch"], case["nz"], case["ny"], case["nx"]
    W, H, modes = case["width"], case["hidden"], 4 * case["modes"] ** 3
    a = torch.randn(B, Z, Y, X, 9, generator=g, device=dev)
    t = torch.randn(B, Z, Y, X, 5, generator=g, device=dev)

    def dense(fan_in, n):
        b = 1.0 / math.sqrt(fan_in)
        return (2.0 * torch.rand(n, generator=g, device=dev) - 1.0) * b

    parts = [dense(9, 9 * W), dense(9, W)]
    for _ in range(case["layers"]):
        parts += [dense(W, W * W), dense(W, W)]
        parts += [torch.rand(modes * W * W, generator=g, device=dev) / (W * W) for _ in range(2)]
    parts += [dense(W, W * H), dense(W, H), dense(H, H * 5), dense(H, 5)]
    return a, t, torch.cat(parts)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "column":
        return {"case": case, "params": [_params(64, 64, case["nz"], T)
                                         for T in _column_groups(case, seed)]}
    if kind == "step":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        insts = [(nx, ny, nz, case["T"], seed)]
        sims = [ehd.Simulation(_params(nx, ny, nz, case["T"]), case["precision"])]
        batch = None
    elif kind == "batch":
        insts = _sweep_instances(case, seed)
        batch = ehd.Batch([_params(nx, ny, nz, T) for nx, ny, nz, T, _ in insts], case["precision"])
        sims = batch.instances
    if kind in ("step", "batch"):
        # pinned FP64 buffers for the field copies, the instances of a batch
        # one after another, and the records at the run's own precision
        total = sum(nx * ny * nz for nx, ny, nz, _, _ in insts)
        host = {k: torch.empty(total, dtype=torch.float64, pin_memory=True) for k in FIELDS}
        prec = RECORD[case["precision"]]
        record = host if prec == torch.float64 else {k: torch.empty(total, dtype=prec) for k in FIELDS}
        spans, at = [], 0
        for sim, (nx, ny, nz, _, s) in zip(sims, insts):
            n = nx * ny * nz
            span = [_ptr(host[k][at:at + n]) for k in FIELDS]
            fields = _start(nx, ny, nz, s)
            for k in FIELDS:
                host[k][at:at + n].copy_(fields[k].reshape(-1))
            ehd._check(ehd.lib().ehd_set_fields(sim.h, *span))
            spans.append(span)
            at += n
        return {"case": case, "sims": sims, "batch": batch, "host": host, "record": record,
                "spans": spans}
    if kind == "noalloc":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        q = _start(nx, ny, nz, seed)["q"]
        out = {k: torch.empty_like(q) for k in ("phi", "ex", "ey", "ez")}
        return {"case": case, "params": _params(nx, ny, nz, 200.0), "q": q, "out": out}
    a, t, w = _fno_inputs(case, seed)
    net = fno.FNO(**_fno_config(case))
    net.set_params(w.cpu().numpy())
    grads = torch.empty(net.nparam, dtype=torch.float32, pin_memory=True)
    return {"case": case, "net": net, "a": a, "t": t, "grads": grads}


# ---- one pass ------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "column":
        p, n = state["params"], _column_steps(case)
        if len(p) == 1:
            cols = [ehd.hydrostatic_profile(p[0], n, "fp64")]
        else:
            cols = sweep.hydrostatic_profiles(ehd, p, [n] * len(p))
        # the velocity, Ex and Ey of the hydrostatic state are zero
        out = {k: np.stack([prof[k] for prof, _ in cols]) for k in ("rho", "q", "phi", "ez")}
        out["i0"] = np.array([i0 for _, i0 in cols])
        return out
    if kind in ("step", "batch"):
        (state["batch"] or state["sims"][0]).step(case["steps"])
        for sim, span in zip(state["sims"], state["spans"]):
            ehd._check(ehd.lib().ehd_get_fields(sim.h, *span))
        if state["record"] is not state["host"]:
            for k in FIELDS:
                state["record"][k].copy_(state["host"][k])
        return state["record"]
    if kind == "noalloc":
        o = state["out"]
        ehd.poisson_noalloc(state["params"], state["q"].data_ptr(), o["phi"].data_ptr(),
                            o["ex"].data_ptr(), o["ey"].data_ptr(), o["ez"].data_ptr())
        return o
    net = state["net"]
    if not case["train"]:
        return {"u": net.forward(state["a"])}
    loss = net.backward(state["a"], state["t"])
    net.adam_step(lr=1e-3)
    ehd._check(fno.lib().ehd_fno_get_grads(
        net.h, ctypes.cast(ctypes.c_void_p(state["grads"].data_ptr()), ctypes.POINTER(ctypes.c_float))))
    return {"loss": np.float32(loss), "grads": state["grads"]}


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    kind = case["kind"]
    if kind in ("column", "step", "batch"):
        steps = _column_steps(case) if kind == "column" else case["steps"]
        if kind == "column":
            nodes, prec = case["count"] * case["nz"], "fp64"
        elif kind == "step":
            nodes, prec = case["nx"] * case["ny"] * case["nz"], case["precision"]
        else:
            nodes = sum(nx * ny * nz for nx, ny, nz, _, _ in _sweep_instances(case, 0))
            prec = case["precision"]
        fb, gb = POP_BYTES[prec]
        real = 8 if prec == "fp64" else 4
        # per node and step: both population sets read and written, the charge
        # written, the potential read; about 650 operations of moments and
        # collisions
        step = 54 * (fb + gb) + 2 * real
        return {"bytes": steps * nodes * step, "flops": steps * nodes * 650}
    if kind == "noalloc":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        n = nx * ny * nz
        return {"bytes": 5 * 8 * n, "flops": n * (5 * math.log2(nx * ny) + 16)}
    B, P = case["batch"], case["nx"] * case["ny"] * case["nz"]
    W, H, L, m = case["width"], case["hidden"], case["layers"], case["modes"]
    rows, modes = B * P, 4 * m ** 3
    spec = 2 * modes * W * W
    params = 9 * W + W + L * (W * W + W + spec) + W * H + H + H * 5 + 5
    # pointwise layers, FFT-sized transforms, mode mixing
    fwd = rows * 2 * (9 * W + L * W * W + W * H + H * 5)
    fwd += L * (rows * W * 2 * 5 * math.log2(P) + B * modes * W * W * 8)
    if not case["train"]:
        return {"bytes": 4 * (rows * 14 + params), "flops": fwd}
    # input, target, weights and both moments read, gradients and the updated
    # three written
    return {"bytes": 4 * (rows * 14 + params * 7), "flops": 3 * fwd}


# ---- the same in 64 bits --------------------------------------------------------

_E = np.array([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1],
               [1, 1, 0], [-1, -1, 0], [1, 0, 1], [-1, 0, -1], [0, 1, 1], [0, -1, -1],
               [1, -1, 0], [-1, 1, 0], [1, 0, -1], [-1, 0, 1], [0, 1, -1], [0, -1, 1],
               [1, 1, 1], [-1, -1, -1], [1, 1, -1], [-1, -1, 1], [1, -1, 1], [-1, 1, -1],
               [-1, 1, 1], [1, -1, -1]], dtype=np.float64)
_W = np.array([8 / 27] + [2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8)


def _exact_poisson(q, nx, ny, nz):
    """phi and E of a charge: FFT in x and y, the discrete sine transform of
    the 3-point operator in z as a matrix."""
    dev = q.device
    dz = 1.0 / (nz - 1)
    n = nz - 2
    kx = torch.arange(nx // 2 + 1, dtype=torch.float64, device=dev) * (2 * math.pi / (nx * dz))
    ky = torch.fft.fftfreq(ny, 1.0 / ny, dtype=torch.float64, device=dev) * (2 * math.pi / (ny * dz))
    j = torch.arange(1, n + 1, dtype=torch.float64, device=dev)
    S = torch.sin(math.pi / (n + 1) * j[:, None] * j[None, :])
    lam = 4.0 * torch.sin(math.pi / (2 * (n + 1)) * j) ** 2
    s = torch.fft.rfft2(-q[1:-1] / EPS) * dz ** 2
    s[0, 0, 0] -= VOLTAGE * nx * ny
    shape = s.shape

    def dst(v):
        return torch.view_as_complex((S @ torch.view_as_real(v).reshape(n, -1)).reshape(*shape, 2))

    s = dst(s) / (lam[:, None, None] + ((ky ** 2)[:, None] + (kx ** 2)[None, :])[None] * dz ** 2)
    phi = torch.zeros(nz, ny, nx, dtype=torch.float64, device=dev)
    phi[1:-1] = torch.fft.irfft2(dst(s) * (-2.0 / (n + 1)), s=(ny, nx))
    phi[0] = VOLTAGE
    ex = (torch.roll(phi, 1, 2) - torch.roll(phi, -1, 2)) * (0.5 / dz)
    ey = (torch.roll(phi, 1, 1) - torch.roll(phi, -1, 1)) * (0.5 / dz)
    ez = torch.empty_like(phi)
    ez[1:-1] = (phi[:-2] - phi[2:]) * (0.5 / dz)
    ez[0] = ez[1]
    ez[-1] = ez[-2]
    return phi, torch.stack([ex, ey, ez])


class _ExactStep:
    """The D3Q27 two-relaxation-time step on [27][z][y][x] populations."""

    def __init__(self, T, fields):
        self.f = fields
        nz, ny, nx = fields["q"].shape
        self.nx, self.ny, self.nz = nx, ny, nz
        dev = fields["q"].device
        dz = 1.0 / (nz - 1)
        self.dt = CFL * dz
        self.cs2 = 1.0 / (3.0 * CFL * CFL)
        self.K = math.sqrt(EPS / RHO0) / M_GROUP
        self.nu = EPS * VOLTAGE / (self.K * T * RHO0)
        self.q0 = C_GROUP * VOLTAGE * EPS
        diff = self.K * VOLTAGE / FE_GROUP
        tf, tg = self.nu / self.cs2 / self.dt, diff / self.cs2 / self.dt
        self.rp, self.rm = 1.0 / (tf + 0.5), 1.0 / (LAMBDA_F / tf + 0.5)
        self.gm, self.gp = 1.0 / (tg + 0.5), 1.0 / (LAMBDA_G / tg + 0.5)
        self.E = torch.tensor(_E, device=dev)
        self.W = torch.tensor(_W, device=dev)
        self.opp = torch.tensor([0] + [d + 1 if d % 2 else d - 1 for d in range(1, 27)], device=dev)
        # where each population comes from, for grids small enough for a table
        self.src = None
        if nx * ny * nz <= 4096:
            at = torch.arange(27 * nx * ny * nz, device=dev).reshape(27, nz, ny, nx)
            self.src = torch.stack([torch.roll(at[d], [int(v) for v in _E[d][::-1]], (0, 1, 2))
                                    for d in range(27)])
        self.rho, self.q, self.phi = fields["rho"], fields["q"], fields["phi"]
        self.u = torch.stack([fields["u"], fields["v"], fields["w"]])
        self.e = torch.stack([fields["ex"], fields["ey"], fields["ez"]])
        self.F = self.equilibrium(self.rho, self.u)
        self.G = self.equilibrium(self.q, self.u + self.K * self.e)

    def along(self, v):
        """e_d . v for every direction"""
        return (self.E @ v.reshape(3, -1)).reshape(27, *v.shape[1:])

    def equilibrium(self, dens, u):
        cu = self.along(u) / (self.cs2 * CFL)
        out = cu * (1.0 + 0.5 * cu)
        out += 1.0 - 0.5 * (u * u).sum(0) / self.cs2
        out *= dens
        out *= self.W[:, None, None, None]
        return out

    def relax(self, f, eq, plus, minus):
        """f - plus (symmetric part of f - eq) - minus (antisymmetric part)"""
        d = f - eq
        do = d[self.opp]
        return f - 0.5 * (plus + minus) * d - 0.5 * (plus - minus) * do

    def momentum(self, f):
        return (self.E.T @ f.reshape(27, -1)).reshape(3, *f.shape[1:])

    def step(self):
        nz = self.nz
        F, G, e = self.F, self.G, self.e
        rho, q = F.sum(0), G.sum(0)
        force = q * e
        mom = self.momentum(F) / CFL + 0.5 * self.dt * force
        u = mom / rho
        u[:, 0] = -mom[:, 1] / rho[0]  # the injector mirrors the plane above it
        u2 = u + self.K * e
        # Guo's force populations, relaxed with both rates
        eF = self.along(force)
        src = self.along(u)
        src *= eF
        src /= CFL * CFL * self.cs2
        src += eF / CFL
        src -= (u * force).sum(0)
        src *= self.W[:, None, None, None] / self.cs2
        so = src[self.opp]
        sp, sm = 1.0 - 0.5 * self.rp, 1.0 - 0.5 * self.rm
        F2 = self.relax(F, self.equilibrium(rho, u), self.rp, self.rm)
        F2 += self.dt * 0.5 * ((sp + sm) * src + (sp - sm) * so)
        del eF, src, so
        # no slip on both electrodes: the populations turn round
        F2[:, 0] = F[self.opp, 0]
        F2[:, -1] = F[self.opp, -1]
        G2 = self.relax(G, self.equilibrium(q, u2), self.gp, self.gm)
        G2[:, -1] = G2[:, -2]  # the collector takes what arrives
        # streaming, periodic; the injector's charge populations from its own
        inj = -G2[self.opp, 0] + 2.0 * self.q0 * self.W[:, None, None]
        if self.src is not None:
            F2, G2 = F2.reshape(-1)[self.src], G2.reshape(-1)[self.src]
        else:
            for d in range(1, 27):
                sh = [int(v) for v in _E[d][::-1]]
                F2[d] = torch.roll(F2[d], sh, (0, 1, 2))
                G2[d] = torch.roll(G2[d], sh, (0, 1, 2))
        G2[:, 0] = inj
        self.F, self.G = F2, G2
        self.rho, self.q, self.u = rho, q, u
        self.phi, self.e = _exact_poisson(q, self.nx, self.ny, nz)

    def fields(self):
        v = (self.rho, *self.u, self.q, self.phi, *self.e)
        return dict(zip(FIELDS, v))


def _exact_column(T, nz, steps):
    """Profile after `steps` steps from rest without charge, and the mean
    current of this and the next step on the 64 x 64 plane."""
    dz = 1.0 / (nz - 1)
    K = math.sqrt(EPS / RHO0) / M_GROUP
    zero = torch.zeros(nz, 1, 1, dtype=torch.float64)
    f = {k: zero.clone() for k in FIELDS}
    f["rho"] += RHO0
    f["phi"] += VOLTAGE * (1.0 - torch.arange(nz, dtype=torch.float64)[:, None, None] * dz)
    s = _ExactStep(T, f)

    def current():
        q = s.q.reshape(-1)
        return float((2.0 * q[-2] - q[-3]) * s.e[2].reshape(-1)[-2]) * K * dz * dz

    for _ in range(steps):
        s.step()
    out = {k: v.reshape(-1).clone() for k, v in s.fields().items()}
    i0 = current()
    s.step()
    return out, 0.5 * (i0 + current()) * 64 * 64


def _exact_fno(case, seed):
    a, t, flat = _fno_inputs(case, seed)
    dev = a.device
    W, H, L, m = case["width"], case["hidden"], case["layers"], case["modes"]
    B, Z, Y, X = case["batch"], case["nz"], case["ny"], case["nx"]
    p = flat.double().requires_grad_(case["train"])
    at = [0]

    def take(*shape):
        n = math.prod(shape)
        at[0] += n
        return p[at[0] - n:at[0]].reshape(*shape)

    def kept(n):
        return torch.tensor([k if k < m else n - 2 * m + k for k in range(2 * m)], device=dev)

    ky, kz = kept(Y), kept(Z)
    gelu = torch.nn.functional.gelu
    v = a.double() @ take(9, W) + take(W)
    for l in range(L):
        Wl, bl = take(W, W), take(W)
        R = torch.complex(take(4 * m ** 3, W, W), take(4 * m ** 3, W, W))
        s = torch.fft.rfft(v, dim=3)[:, :, :, :m]
        s = torch.fft.fft(s, dim=2)[:, :, ky]
        s = torch.fft.fft(s, dim=1)[:, kz]
        o = torch.einsum("koi,bki->bko", R, s.reshape(B, -1, W)).reshape(B, 2 * m, 2 * m, m, W)
        o = torch.fft.ifft(torch.zeros(B, Z, 2 * m, m, W, dtype=o.dtype, device=dev)
                           .index_copy(1, kz, o), dim=1)
        o = torch.fft.ifft(torch.zeros(B, Z, Y, m, W, dtype=o.dtype, device=dev)
                           .index_copy(2, ky, o), dim=2)
        z = v @ Wl + bl + torch.fft.irfft(o, n=X, dim=3)
        v = gelu(z) if l < L - 1 else z
    u = gelu(v @ take(W, H) + take(H)) @ take(H, 5) + take(5)
    if not case["train"]:
        return {"u": u}
    loss = torch.mean((u - t.double()) ** 2)
    loss.backward()
    return {"loss": float(loss.detach()), "grads": p.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind == "column":
        if case["count"] * _column_steps(case) > 25000:  # about 0.6 ms a step
            return None
        cols = [_exact_column(T, case["nz"], _column_steps(case)) for T in _column_groups(case, seed)]
        out = {k: torch.stack([f[k] for f, _ in cols]) for k in ("rho", "q", "phi", "ez")}
        out["i0"] = torch.tensor([i0 for _, i0 in cols], dtype=torch.float64)
        return out
    if kind in ("step", "batch"):
        if kind == "step":
            insts = [(case["nx"], case["ny"], case["nz"], case["T"], seed)]
        else:
            insts = _sweep_instances(case, seed)
        nodes = sum(nx * ny * nz for nx, ny, nz, _, _ in insts)
        # a step takes a few milliseconds of launches and grows with its nodes
        if case["steps"] * (len(insts) * 3e-3 + nodes * 4e-9) > 18.0:
            return None
        parts = {k: [] for k in FIELDS}
        for nx, ny, nz, T, s in insts:
            sim = _ExactStep(T, _start(nx, ny, nz, s))
            for _ in range(case["steps"]):
                sim.step()
            for k, v in sim.fields().items():
                parts[k].append(v.reshape(-1))
        return {k: torch.cat(v) for k, v in parts.items()}
    if kind == "noalloc":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        phi, e = _exact_poisson(_start(nx, ny, nz, seed)["q"], nx, ny, nz)
        return {"phi": phi, "ex": e[0], "ey": e[1], "ez": e[2]}
    return _exact_fno(case, seed)
