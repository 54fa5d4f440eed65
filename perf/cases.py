"""Performance cases of the TWMC trajectory engine: what its users run.

A user builds a `System` (one lattice and its parameters), makes tasks (one
per trajectory) and calls `run`, which returns saved frames, the final
fields or the ensemble moment blocks in host arrays; a parameter sweep uses
an `HBatch` instead, and its learned warm start trains an `MLP`. The
configurations are those of `pincosimulator_gb300/workloads.py`, `bench.py`
and `warmstart.py`, over their real range: chains of 32 sites and a hundred
trajectories up to 64 x 64 lattices with thousands, sides that are no powers
of two, Lieb lattices with a ramped drive, FP64 runs, mixed batches.

Result arrays are page-locked and reused from call to call, as `bench.py`
does. The C ABI hands every field over as complex128 and every moment block
as float64, also those of an FP32 run; the programs here go on with an FP32
run's results on the GPU in the precision they were computed in.
"""
import math

import numpy as np
import torch

from pincosimulator_gb300 import twmc

TWO_PI = 2.0 * math.pi


def listed():
    return [
        # a first look at a short chain: few trajectories, few steps; latency and launches are all of it
        {"name": "chain32_few", "kind": "square", "nx": 1, "ny": 32, "hop": "fft", "integrator": "euler", "prec": 32,
         "disorder": 0.0, "ntraj": 100, "steps": 100, "frames": 1, "out": "final", "dt": 0.005, "U": 0.1,
         "omega": -1.0, "F": 1.5},
        # the reference's own CPU runs: a chain of 64 sites, 1000 trajectories, every frame kept
        {"name": "chain64_frames", "kind": "square", "nx": 1, "ny": 64, "hop": "fft", "integrator": "euler", "prec": 32,
         "disorder": 0.0, "ntraj": 1000, "steps": 100, "frames": 10, "out": "frames", "dt": 0.005, "U": 0.1,
         "omega": -1.0, "F": 1.5},
        # a small lattice on the exponential split step, ensemble moments
        {"name": "square16_split", "kind": "square", "nx": 16, "ny": 16, "hop": "fft", "integrator": "split",
         "prec": 32, "disorder": 0.2, "ntraj": 2500, "steps": 250, "frames": 2, "out": "moments", "dt": 0.002,
         "U": 0.2, "omega": -0.5, "F": 2.0},
        # the warm-start sweep's lattice as a single system with omega disorder, fields and moments
        {"name": "square32_fft", "kind": "square", "nx": 32, "ny": 32, "hop": "fft", "integrator": "euler", "prec": 32,
         "disorder": 0.2, "ntraj": 2000, "steps": 250, "frames": 2, "out": "both", "dt": 0.002, "U": 0.2,
         "omega": -0.5, "F": 2.0},
        # the headline workload (64 x 64, omega disorder, FFT hopping) with half its trajectories: the largest
        {"name": "square64_fft", "kind": "square", "nx": 64, "ny": 64, "hop": "fft", "integrator": "euler", "prec": 32,
         "disorder": 0.2, "ntraj": 8192, "steps": 250, "frames": 1, "out": "moments", "dt": 0.002, "U": 0.2,
         "omega": -0.5, "F": 2.0},
        # the same lattice with the hopping applied in real space
        {"name": "square64_stencil", "kind": "square", "nx": 64, "ny": 64, "hop": "stencil", "integrator": "euler",
         "prec": 32, "disorder": 0.2, "ntraj": 4096, "steps": 250, "frames": 1, "out": "moments", "dt": 0.002,
         "U": 0.2, "omega": -0.5, "F": 2.0},
        # sides that are no powers of two and a ragged number of trajectories: always real space
        {"name": "square50_ragged", "kind": "square", "nx": 50, "ny": 50, "hop": "fft", "integrator": "euler",
         "prec": 32, "disorder": 0.2, "ntraj": 777, "steps": 250, "frames": 2, "out": "both", "dt": 0.002, "U": 0.2,
         "omega": -0.5, "F": 2.0},
        # the largest lattice
        {"name": "square128", "kind": "square", "nx": 128, "ny": 128, "hop": "stencil", "integrator": "euler",
         "prec": 32, "disorder": 0.2, "ntraj": 600, "steps": 250, "frames": 1, "out": "both", "dt": 0.002, "U": 0.2,
         "omega": -0.5, "F": 2.0},
        # the Lieb lattice with U disorder and a drive ramped in a table (TWMCLiebSolver's F(t) runs)
        {"name": "lieb768_ramp", "kind": "lieb", "cells": 256, "pbc": True, "ramp": True, "ntraj": 2048, "steps": 250,
         "frames": 2, "out": "both", "dt": 0.002},
        # FP64 mode, as runs are checked with it
        {"name": "square16_f64", "kind": "square", "nx": 16, "ny": 16, "hop": "fft", "integrator": "euler", "prec": 64,
         "disorder": 0.2, "ntraj": 500, "steps": 100, "frames": 1, "out": "both", "dt": 0.002, "U": 0.2,
         "omega": -0.5, "F": 2.0},
        # a frame of a parameter sweep over mixed lattices, with the step variants that its autotuner keeps
        {"name": "sweep_mixed", "kind": "sweep", "points": 24, "traj_scale": 0.25, "tuned": True},
        # minibatches of the warm start's training on 32 x 32 targets
        {"name": "warm_fit", "kind": "fit", "L": 32, "batch": 128, "minibatches": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fft", "fft", "fft", "stencil", "stencil", "stencil", "lieb", "f64", "sweep", "fit"])
    if kind == "fit":
        return {"kind": "fit", "L": rng.choice([16, 32]), "batch": rng.randint(32, 256),
                "minibatches": rng.randint(4, 12)}
    if kind == "sweep":
        return {"kind": "sweep", "points": rng.randint(8, 32), "traj_scale": round(rng.uniform(0.05, 0.25), 3),
                "tuned": rng.choice([True, False])}
    frames = rng.randint(1, 4)
    steps = _log_int(rng, 50, 500)
    if kind == "lieb":
        cells = _log_int(rng, 8, 400)
        most = min(4096, max(16, 2.0e9 // (3 * cells * frames * steps)))
        return {"kind": "lieb", "cells": cells, "pbc": rng.choice([True, False]), "ramp": rng.choice([True, False]),
                "ntraj": _log_int(rng, 16, most), "steps": steps, "frames": frames,
                "out": rng.choice(["final", "both", "moments"]), "dt": 0.002}
    c = {"kind": "square", "integrator": "euler", "hop": "fft", "prec": 32, "disorder": rng.choice([0.0, 0.2]),
         "U": round(rng.uniform(0.05, 0.5), 3), "omega": round(rng.uniform(-2, 2), 3),
         "F": round(rng.uniform(0, 3), 3), "dt": 0.002}
    if kind == "stencil":
        c["hop"] = "stencil"
        if rng.random() < 0.25:
            nx, ny = 1, _log_int(rng, 10, 4096)
        else:
            nx, ny = _log_int(rng, 4, 128), _log_int(rng, 4, 128)
        most_n = 4e9
    else:
        nx, ny = rng.choice([(1, 32), (1, 64), (1, 128), (1, 256), (1, 512), (1, 1024), (1, 2048), (1, 4096), (16, 16),
                             (32, 32), (64, 64)])
        c["integrator"] = rng.choice(["euler", "euler", "split"])
        most_n = 4e9
        if kind == "f64":
            c["prec"] = 64
            frames, steps, most_n = 1, rng.randint(20, 100), 1.0e8
    most = min(16384, max(16, most_n // (nx * ny * frames * steps)))
    c.update(nx=nx, ny=ny, steps=steps, frames=frames, ntraj=_log_int(rng, 16, most))
    c["out"] = "moments" if nx * ny * c["ntraj"] > 6e6 else rng.choice(["final", "both", "frames"])
    if c["out"] == "frames" and nx * ny * c["ntraj"] * frames > 8e6:
        c["out"] = "final"
    return c


# ---------------------------------------------------------------------------
# single systems
# ---------------------------------------------------------------------------
BLOCKS = 32


def _seed0(seed):
    return (int(seed) * 1000003 + 17) % (1 << 31)


def _lieb_table(case):
    n = 3 * case["cells"]
    times = np.round(np.arange(0, 2 + 1e-9, 0.01), 10)
    vals = np.zeros((len(times), n), dtype=complex)
    vals[:, 1::3] = (2.5 * times / 2.0)[:, None]  # the drive on the B sites ramps up to 2.5, then holds
    return times, vals


def _system(case):
    common = dict(gamma=1.0, dt=case["dt"], frame_steps=case["steps"], beta_init=0.0, beta_init_sigma=0.5,
                  n_moment_blocks=BLOCKS)
    if case["kind"] == "lieb":
        drive = dict(F=0.0, F_t=_lieb_table(case)) if case["ramp"] else dict(F=1.0)
        return twmc.System(lattice=twmc.LATTICE_LIEB, nx=1, ny=case["cells"], pbc=case["pbc"], J_AB=1.0, J_BC=1.0,
                           detuning=0.0, omega=0.0, U=twmc.Noisy(0.27, twmc.DISORDER_UNIFORM, 0.06), **drive, **common)
    omega = twmc.Noisy(case["omega"], twmc.DISORDER_GAUSSIAN, case["disorder"]) if case["disorder"] else case["omega"]
    return twmc.System(nx=case["nx"], ny=case["ny"], J=1.0, omega=omega, U=case["U"], F=case["F"],
                       precision=twmc.PREC_F64 if case["prec"] == 64 else twmc.PREC_F32,
                       hop=twmc.HOP_STENCIL if case["hop"] == "stencil" else twmc.HOP_FFT,
                       integrator=twmc.INTEGRATOR_SPLIT if case["integrator"] == "split" else twmc.INTEGRATOR_EULER,
                       **common)


def _sites(case):
    return 3 * case["cells"] if case["kind"] == "lieb" else case["nx"] * case["ny"]


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _prepare_system(case, seed):
    sysd = _system(case)
    n, t, f = _sites(case), case["ntraj"], case["frames"]
    tasks = sysd.make_tasks(t, t_start=0.0, t_end=f * case["steps"] * case["dt"], seed0=_seed0(seed),
                            id0=1 + int(seed) % 1000, store_initial=False)
    bufs = {}
    if case["out"] in ("final", "both", "frames"):
        bufs["final"] = _pinned((t, n), torch.complex128)
    if case["out"] == "frames":
        bufs["frames"] = _pinned((t, f, n), torch.complex128)
    if case["out"] in ("moments", "both"):
        bufs["moments"] = _pinned((f, BLOCKS, n, 3), torch.float64)
    f64 = case["kind"] == "square" and case["prec"] == 64
    return {"kind": "system", "sys": sysd, "tasks": tasks, "bufs": bufs, "f64": f64}


def _run_system(s):
    b = s["bufs"]
    res = s["sys"].run(s["tasks"], frames="frames" in b, final="final" in b, moments="moments" in b, buffers=b)
    out = {}
    for k in sorted(b):
        v = torch.from_numpy(res[k]).cuda()
        if not s["f64"]:
            v = v.to(torch.float32 if k == "moments" else torch.complex64)
        out[k] = v
    return out


# ---------------------------------------------------------------------------
# sweeps (heterogeneous batches)
# ---------------------------------------------------------------------------
SWEEP_STEPS = 250
# what the batch's autotuner keeps on this card, by lattice
TUNED = {(1, 32): "ell2", (1, 64): "ell2", (1, 128): "ell4", (1, 256): "ell2", (1, 512): "ell4", (1, 1024): "ell4",
         (16, 16): "ell2", (32, 32): "ell4", (64, 64): "rowrun", (128, 128): "cluster_pow2"}


def _sweep_points(case, seed):
    """The lattices and trajectories are the case's, the parameters and seeds the seed's."""
    shape = np.random.default_rng(3)
    par = np.random.default_rng(int(seed))
    kinds = sorted(TUNED)
    pts = []
    for _ in range(case["points"]):
        nx, ny = kinds[shape.integers(len(kinds))]
        nt = int(math.exp(shape.uniform(math.log(512), math.log(4096))) * case["traj_scale"])
        pts.append(dict(nx=nx, ny=ny, U=par.uniform(0.05, 0.5), omega=par.uniform(-2, 2), F=par.uniform(0, 3),
                        dt=0.002, n_traj=max(1, nt), seed0=int(par.integers(1, 2 ** 31)), id0=1))
    return pts


def _prepare_sweep(case, seed):
    pts = _sweep_points(case, seed)
    hb = twmc.HBatch(pts, SWEEP_STEPS, variants=[TUNED[(p["nx"], p["ny"])] for p in pts] if case["tuned"] else None)
    n = hb.total_sites
    return {"kind": "sweep", "hb": hb, "mean": torch.zeros(n, 2, dtype=torch.float64, device="cuda"),
            "abs2": torch.zeros(n, dtype=torch.float64, device="cuda")}


def _run_sweep(s):
    hb = s["hb"]
    hb.run(1)
    hb.field_moments(s["mean"].data_ptr(), s["abs2"].data_ptr())
    blocks = np.concatenate(hb.block_means())  # waits for the batch
    return {"blocks": torch.from_numpy(blocks).to(torch.float32), "mean": s["mean"].to(torch.float32),
            "abs2": s["abs2"].to(torch.float32)}


# ---------------------------------------------------------------------------
# training of the learned warm start
# ---------------------------------------------------------------------------
def _fit_data(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    rows, o = case["batch"] * case["minibatches"], 2 * case["L"] ** 2 + 1
    x = torch.rand(rows, 5, device="cuda", generator=g) * 2 - 1
    mix = torch.randn(5, o, device="cuda", generator=g)
    t = torch.tanh(x @ mix) + 0.05 * torch.randn(rows, o, device="cuda", generator=g)
    w = torch.rand(o, device="cuda", generator=g).clamp_min(1e-4)
    return x, t, w


def _widths(case):
    return [5, 256, 256, 256, 2 * case["L"] ** 2 + 1]


def _fit_params(case, seed):
    """Glorot-uniform weights and zero biases, layer after layer, as the network holds them."""
    rng = np.random.default_rng(int(seed))
    parts = []
    for k, n in zip(_widths(case)[:-1], _widths(case)[1:]):
        a = math.sqrt(6.0 / (k + n))
        parts += [rng.uniform(-a, a, n * k), np.zeros(n)]
    return np.concatenate(parts).astype(np.float32)


def _prepare_fit(case, seed):
    x, t, w = _fit_data(case, seed)
    net = twmc.MLP(_widths(case), case["batch"])
    net.set_params(_fit_params(case, seed))
    return {"kind": "fit", "net": net, "x": x, "t": t, "w": w, "batch": case["batch"],
            "minibatches": case["minibatches"]}


LR = 2e-3


def _run_fit(s):
    net, b = s["net"], s["batch"]
    for j in range(s["minibatches"]):
        net.backward(s["x"][j * b:(j + 1) * b].data_ptr(), s["t"][j * b:(j + 1) * b].data_ptr(), b, s["w"].data_ptr())
        net.adam(LR)
    return {"params": net.get_params(), "grads": net.get_grads(), "loss": np.float32(net.last_loss())}


# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "sweep":
        return _prepare_sweep(case, seed)
    if case["kind"] == "fit":
        return _prepare_fit(case, seed)
    return _prepare_system(case, seed)


def run(state):
    if state["kind"] == "sweep":
        return _run_sweep(state)
    if state["kind"] == "fit":
        return _run_fit(state)
    return _run_system(state)


def work(case):
    if case["kind"] == "fit":
        widths = _widths(case)
        p = sum(a * b + b for a, b in zip(widths[:-1], widths[1:]))
        mm = sum(a * b for a, b in zip(widths[:-1], widths[1:]))
        hidden = mm - widths[0] * widths[1]  # no gradient of the first layer's input
        m, b, o = case["minibatches"], case["batch"], widths[-1]
        return {"bytes": m * (b * (5 + o) * 4 + 7 * p * 4), "flops": m * b * (4 * mm + 2 * hidden)}
    if case["kind"] == "sweep":
        by = fl = 0
        for p in _sweep_points(case, 0):
            n = p["nx"] * p["ny"]
            by += n * p["n_traj"] * 16 + n * (24 + 32 * 24)
            fl += n * p["n_traj"] * SWEEP_STEPS * 34
        return {"bytes": by, "flops": fl}
    n, t, f = _sites(case), case["ntraj"], case["frames"]
    outputs = {"final": t * n * 16, "frames": t * n * 16 * (f + 1), "moments": f * BLOCKS * n * 24,
               "both": t * n * 16 + f * BLOCKS * n * 24}[case["out"]]
    if case["kind"] == "square" and case["hop"] == "fft" and n & (n - 1) == 0:
        per = 10 * math.log2(n) + 26  # two FFTs, the k-space multiply and the local step
    else:
        per = 34                      # four neighbours and the local step
    return {"bytes": outputs + t * 8, "flops": n * t * f * case["steps"] * per}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch: Philox4x32-10 (Salmon et al., SC'11)
# counters per (site pair, step, trajectory), Box-Muller, the Euler-Maruyama
# or split step with the hopping as rolls or a torch FFT
# ---------------------------------------------------------------------------
M32 = 0xFFFFFFFF


def _philox(c, k0, k1):
    c0, c1, c2, c3 = c
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57  # wrap in 64 bits: the two halves are still exact
        c0, c1, c2, c3 = ((p1 >> 32) & M32) ^ c1 ^ k0, p1 & M32, ((p0 >> 32) & M32) ^ c3 ^ k1, p0 & M32
        k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
    return c0, c1, c2, c3


def _normal(a, b):
    r = torch.sqrt(-2.0 * torch.log((a.double() + 0.5) * 2.0 ** -32))
    th = (b.double() + 0.5) * (TWO_PI * 2.0 ** -32) - math.pi
    return torch.complex(r * torch.cos(th), r * torch.sin(th))


class _Noise:
    """Draws of a range of trajectories (seed and id per trajectory) on n sites."""

    def __init__(self, seeds, ids, n):
        self.seeds, self.ids, self.n, self.half = seeds[:, None], ids[:, None], n, (n + 1) // 2
        self.pair = torch.arange(self.half, device="cuda")[None, :].expand(len(seeds), -1)

    def _split(self, w, of):
        return torch.cat([of(w[0], w[1]), of(w[2], w[3])[:, :self.n - self.half]], dim=1)

    def wiener(self, step):
        c = (self.pair, torch.full_like(self.pair, step), self.ids.expand_as(self.pair),
             self.seeds.expand_as(self.pair))
        return self._split(_philox(c, 0x243F6A88, 0x85A308D3), _normal)

    def stream(self, which, of=_normal):
        z = torch.zeros_like(self.pair)
        return self._split(_philox((self.pair, z, torch.full_like(z, which), z), self.seeds, self.ids), of)


def _uniform(a, b):
    return torch.complex(a.double() * 2.0 ** -32, b.double() * 2.0 ** -32)


def _square_hop(b, nx, ny):
    v = b.view(-1, nx, ny)
    h = torch.zeros_like(v)
    if ny > 1:
        h += torch.roll(v, 1, 2) + torch.roll(v, -1, 2)
    if nx > 1:
        h += torch.roll(v, 1, 1) + torch.roll(v, -1, 1)
    return h.view(b.shape)


def _lieb_hop(b, pbc):
    v = b.view(len(b), -1, 3)
    A, B, C = v[..., 0], v[..., 1], v[..., 2]
    cp, bn = torch.roll(C, 1, 1), torch.roll(B, -1, 1)
    if not pbc:
        cp[:, 0] = 0
        bn[:, -1] = 0
    return torch.stack([B, A + C + cp, B + bn], dim=2).view(b.shape)


def _exact_chunk(case, seeds, ids):
    """Yields the field after every frame of a range of trajectories."""
    n, dt = _sites(case), case["dt"]
    noise = _Noise(seeds, ids, n)
    b = 0.5 * noise.stream(1)
    scale = math.sqrt(dt / 4.0)
    lieb = case["kind"] == "lieb"
    om, U, F = 0.0, None, None
    if lieb:
        U = 0.27 + 0.06 * noise.stream(2, _uniform).real
        if not case["ramp"]:
            F = 1.0
    else:
        U, F, om = case["U"], case["F"], case["omega"]
        if case["disorder"]:
            om = om + case["disorder"] * noise.stream(3).real
        nx, ny = case["nx"], case["ny"]
    # Lieb: detuning - E = 0
    lin = (-1j * om if not lieb else 0.0) - 0.5
    iU = 1j * U
    if not lieb and case["integrator"] == "split":
        kx, ky = torch.arange(nx, device="cuda").double(), torch.arange(ny, device="cuda").double()
        ck = (0.0 if nx == 1 else torch.cos(TWO_PI * kx / nx))
        ck = (ck[:, None] if nx > 1 else 0.0) + (torch.cos(TWO_PI * ky / ny)[None, :] if ny > 1 else 0.0)
        factor = torch.exp(-2j * dt * (ck + 0.0 * ky[None, :]))
    t = 0.0
    for step in range(case["frames"] * case["steps"]):
        if lieb:
            drive = torch.zeros(n, dtype=torch.complex128, device="cuda")
            if case["ramp"]:
                drive[1::3] = 2.5 * min(t, 2.0) / 2.0
            else:
                drive += F
            hop = -1j * _lieb_hop(b, case["pbc"])
        else:
            drive = F
            if case["integrator"] == "split":
                b = torch.fft.ifft2(torch.fft.fft2(b.view(-1, nx, ny)) * factor).view(b.shape)
                hop = 0.0
            else:
                hop = -1j * _square_hop(b, nx, ny)
        a = (lin + iU * (b.real * b.real + b.imag * b.imag - 1.0)) * b + hop + 1j * drive
        b = b + dt * a + scale * noise.wiener(step)
        t += dt
        if (step + 1) % case["steps"] == 0:
            yield b


def _exact_system(case, seed):
    n, t, f = _sites(case), case["ntraj"], case["frames"]
    per = max(1, min(t, 4_000_000 // n))
    fields = torch.zeros(t, n, dtype=torch.complex128, device="cuda")
    frames = torch.zeros(t, f, n, dtype=torch.complex128, device="cuda") if case["out"] == "frames" else None
    mom = torch.zeros(f, BLOCKS, n, 3, dtype=torch.float64, device="cuda")
    blocks = min(BLOCKS, t)
    edge = torch.tensor([b * t // blocks for b in range(1, blocks)], device="cuda")
    fft = case["kind"] == "square" and case["hop"] == "fft" and n & (n - 1) == 0
    for lo in range(0, t, per):
        at = torch.arange(lo, min(t, lo + per), device="cuda")
        which = torch.bucketize(at, edge, right=True)
        for k, b in enumerate(_exact_chunk(case, (at + _seed0(seed)) & M32, at + 1 + int(seed) % 1000)):
            p = b.real ** 2 + b.imag ** 2
            mom[k, :, :, 0].index_add_(0, which, p)
            mom[k, :, :, 1].index_add_(0, which, p * p)
            if fft:
                q = torch.fft.fft2(b.view(-1, case["nx"], case["ny"])).reshape(b.shape)
                mom[k, :, :, 2].index_add_(0, which, (q.real ** 2 + q.imag ** 2) / n)
            if frames is not None:
                frames[lo:lo + len(at), k] = b
            fields[lo:lo + len(at)] = b
    out = {}
    if case["out"] in ("final", "both", "frames"):
        out["final"] = fields
    if case["out"] == "frames":
        out["frames"] = frames
    if case["out"] in ("moments", "both"):
        out["moments"] = mom
    return out


def _exact_sweep(case, seed):
    means, abs2s, blocks = [], [], []
    for p in _sweep_points(case, seed):
        n, t = p["nx"] * p["ny"], p["n_traj"]
        c = dict(p, kind="square", integrator="euler", disorder=0.0, frames=1, steps=SWEEP_STEPS, hop="fft")
        nb = min(BLOCKS, t)
        edge = torch.tensor([b * t // nb for b in range(1, nb)], device="cuda", dtype=torch.int64)
        mean = torch.zeros(n, dtype=torch.complex128, device="cuda")
        abs2 = torch.zeros(n, dtype=torch.float64, device="cuda")
        mom = torch.zeros(nb, 3, dtype=torch.float64, device="cuda")
        fft = not case["tuned"] and n <= 4096  # k-space populations come from the FFT variants only
        per = max(1, 4_000_000 // n)
        for lo in range(0, t, per):
            at = torch.arange(lo, min(t, lo + per), device="cuda")
            which = torch.bucketize(at, edge, right=True)
            b, = _exact_chunk(c, (at + p["seed0"]) & M32, at + 1)
            q = b.real ** 2 + b.imag ** 2
            mean += b.sum(0)
            abs2 += q.sum(0)
            cols = [q.mean(1), (q * q).mean(1), q.mean(1) if fft else torch.zeros_like(q[:, 0])]  # Parseval
            mom.index_add_(0, which, torch.stack(cols, dim=1))
        means.append(torch.view_as_real(mean / t))
        abs2s.append(abs2 / t)
        blocks.append(mom)
    return {"blocks": torch.cat(blocks), "mean": torch.cat(means), "abs2": torch.cat(abs2s)}


def _exact_fit(case, seed):
    x, t, w = (v.double() for v in _fit_data(case, seed))
    widths = _widths(case)
    flat = torch.from_numpy(_fit_params(case, seed)).double().cuda()
    pars, off = [], 0
    for k, n in zip(widths[:-1], widths[1:]):
        pars.append(flat[off:off + n * k].view(n, k).clone().requires_grad_(True))
        pars.append(flat[off + n * k:off + n * k + n].clone().requires_grad_(True))
        off += n * k + n
    m = [torch.zeros_like(p) for p in pars]
    v = [torch.zeros_like(p) for p in pars]
    b = case["batch"]
    for j in range(case["minibatches"]):
        a = x[j * b:(j + 1) * b]
        for k in range(4):
            a = a @ pars[2 * k].t() + pars[2 * k + 1]
            if k < 3:
                a = 0.5 * a * (1 + torch.erf(a / math.sqrt(2.0)))
        loss = (w * (a - t[j * b:(j + 1) * b]) ** 2).sum() / a.numel()
        grads = torch.autograd.grad(loss, pars)
        with torch.no_grad():
            for p, q, mm, vv in zip(pars, grads, m, v):
                mm.mul_(0.9).add_(0.1 * q)
                vv.mul_(0.999).add_(0.001 * q * q)
                p -= LR * (mm / (1 - 0.9 ** (j + 1))) / (torch.sqrt(vv / (1 - 0.999 ** (j + 1))) + 1e-8)
    flatten = lambda vs: torch.cat([q.detach().reshape(-1) for q in vs])  # noqa: E731
    return {"params": flatten(pars), "grads": flatten(grads), "loss": loss.detach().reshape(())}


def exact(case, seed):
    if case["kind"] == "fit":
        return _exact_fit(case, seed)
    if case["kind"] == "sweep":
        return _exact_sweep(case, seed)
    return _exact_system(case, seed)
