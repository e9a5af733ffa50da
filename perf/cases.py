"""The work that users of this package have it do, as cases that can be timed
and checked: relaxation steps in both precisions over the range of grids, the
batch, the snapshot of a run, and the warm-start network's training step and
application.

A case is a dict of plain values. `listed` gives the named ones, `draw` more of
the same ranges, `prepare` what a program holds before the call (handle or
network, and seeded inputs on the device), `run` one pass through the public
entry points, `work` the bytes and operations that the pass cannot do without,
and `exact` what it returns in 64-bit torch, without the package's kernels.

The initial states are seeded polycrystals of every field: lattices of the
field's own length in Voronoi grains of random orientation, with a little white
noise. They stand for the bulk of a relaxation, which spends most of its steps
on such states. Fields and energies of a single-precision relaxation come back
in single precision, those of a double-precision one in double.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from pfc_b200 import fno, lib
from pfc_b200 import params as P

SIZES = (128, 256, 384, 512, 768, 1024, 1536, 2048, 4096)
BATCH_SIZES = (256, 384, 512, 768, 1024, 1536)
A0 = 7.2552  # lattice length of the heterostructure's first field
POINT_STEPS = 50 * 2 * 4096 * 4096  # steps x points x fields of the largest listed relaxation


def listed():
    return [
        # Short call on a small grid, the reference's precision: a parameter scan, or a box small
        # enough for one grain; latency and launches count.
        relax("relax_fp64_u1_128", 128, 128, 1, "fp64", 10),
        # The single-component honeycomb configuration (512^2, dx = dy = pi/4, dt = 1) in FP64.
        relax("relax_fp64_u1_512", 512, 512, 1, "fp64", 50),
        # The same in single precision.
        relax("relax_fp32_u1_512", 512, 512, 1, "fp32", 50),
        # The reference's three-field heterostructure demo (512^2, U = 3), in its own precision.
        relax("relax_fp64_u3_512", 512, 512, 3, "fp64", 50),
        # A rectangular box of no special length, with the semi-implicit scheme.
        relax("relax_fp32_u2_1440x900", 1440, 900, 2, "fp32", 50, scheme="semi"),
        # The 2048^2 polycrystal configuration with box optimisation.
        relax("relax_fp32_u1_2048", 2048, 2048, 1, "fp32", 50, optimise=True),
        # The headline heterostructure: 4096^2, two fields, box optimised every 50 steps.
        relax("relax_fp32_u2_4096", 4096, 4096, 2, "fp32", 50, optimise=True),
        # The same grid in the reference's precision, the judge of the single-precision runs.
        relax("relax_fp64_u2_4096", 4096, 4096, 2, "fp64", 10),
        # Independent problems of uneven sizes stepped together (256^2 .. 1536^2, one or two fields).
        {"name": "batch_fp32_24", "kind": "batch", "problems": 24, "pick": 7, "steps": 50},
        # Restart and snapshot of a run: fields uploaded from the host, <f>, f(r) and the fields
        # brought back, as the driver writes them.
        {"name": "snapshot_fp64_u2_1024", "kind": "snapshot", "Nx": 1024, "Ny": 1024, "U": 2, "precision": "fp64"},
        # One training iteration of the warm-start network in its training shape (16 tiles of 512^2).
        {"name": "train_512_b16", "kind": "train", "tile": 512, "batch": 16},
        # The shipped network applied tile by tile to a 4096^2 state.
        {"name": "apply_4096", "kind": "apply", "Nx": 4096, "Ny": 4096, "tile": 512, "batch": 16},
    ]


def relax(name, Nx, Ny, U, precision, steps, scheme="etd1", conserved=True, modes=1, optimise=False):
    d = {"kind": "relax", "Nx": Nx, "Ny": Ny, "U": U, "precision": precision, "steps": steps, "scheme": scheme,
         "conserved": conserved, "modes": modes, "optimise": optimise}
    return dict(d, name=name) if name else d


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def smooth_even(n):
    """The next even number from n on with no factor above 7."""
    n += n % 2
    while True:
        m = n
        for f in (2, 3, 5, 7):
            while m % f == 0:
                m //= f
        if m == 1:
            return n
        n += 2


def draw(rng):
    kind = rng.choices(("relax", "batch", "snapshot", "train", "apply"), (12, 2, 2, 2, 2))[0]
    if kind == "batch":
        return {"kind": kind, "problems": rng.randint(8, 32), "pick": rng.randint(0, 9999), "steps": rng.randint(10, 50)}
    if kind == "train":
        return {"kind": kind, "tile": rng.choice((64, 128, 256, 512)), "batch": rng.randint(1, 16)}
    if kind == "apply":
        return {"kind": kind, "Nx": log_int(rng, 300, 4000), "Ny": log_int(rng, 300, 4000),
                "tile": rng.choice((128, 256, 512)), "batch": rng.randint(4, 16)}
    while True:
        precision, U = rng.choice(("fp32", "fp64")), rng.choice((1, 1, 2, 2, 3, 4))
        if rng.random() < 0.5:
            Nx = Ny = rng.choice(SIZES)
        else:
            Nx, Ny = smooth_even(log_int(rng, 64, 3600)), smooth_even(log_int(rng, 64, 3600))
        if not lib.size_supported_for(Nx, Ny, U, precision):
            continue
        if kind == "snapshot":
            if U * Nx * Ny <= 2 * 1024 * 1024:
                return {"kind": kind, "Nx": Nx, "Ny": Ny, "U": U, "precision": precision}
            continue
        most = POINT_STEPS // (Nx * Ny * U * (4 if precision == "fp64" else 1))
        if most < 10:
            continue
        return relax(None, Nx, Ny, U, precision, min(most, rng.randint(10, 50)), rng.choice(("etd1", "etd1", "semi")),
                     rng.random() < 0.8, rng.choice((1, 2)) if U == 1 else 1, rng.random() < 0.5)


# ----------------------------------------------------------- models and states

def model(U, conserved=True, modes=1):
    """(input-file values, dt, dx, means, amplitudes, lattice lengths) of U fields."""
    if U == 1:
        d = P.honeycomb_1c(-0.25)
        mean, amp, dt, dx, lat = [0.25], [-0.4], 1.0, math.pi / 4, [P.A_TRI]
        if not conserved:
            d["alpha"], d["gamma"], mean, dt = [[-0.15]], [[0.8]], [0.06], 0.5
    else:
        z = lambda: [[0.0] * U for _ in range(U)]  # noqa: E731
        a, b, g, e, m = z(), z(), z(), z(), z()
        for u in range(U):
            a[u][u], b[u][u] = (-1.4, 2.25) if u == 0 else (-0.3, 1.0)
            for v in range(u + 1, U):
                if u == 0:
                    a[u][v], e[u][v] = -0.04, -0.8
                else:
                    a[u][v], b[u][v], g[u][v], m[u][v] = 0.5, 0.02, 0.3, 1.018
        s = [1.0] + [1.04 if U == 2 else 1.018] * (U - 1)
        d = {"lambda": [0.0] * U, "alpha": a, "beta": b, "gamma": g, "delta": [2.25] + [1.0] * (U - 1), "epsilon": e,
             "sigma": 0.2, "inv_nu": [[x] for x in s], "omega": [[1.0]] * U, "phi": [[0.0]] * U, "inv_mu": m}
        mean, amp = [0.3] + [-0.3] * (U - 1), [-0.8] + [0.4] * (U - 1)
        dt, dx, lat = 0.25, 0.7, [A0 * x for x in s]
    if modes == 2:  # the square-lattice style two-mode operator
        d["inv_nu"], d["omega"], d["phi"], dt = [[1.0, math.sqrt(2.0)]], [[1.0, 1.0]], [[0.0, 0.05]], 0.5
    return d, dt, dx, mean, amp, lat


def states(Nx, Ny, dx, mean, amp, lat, seed, grains=6):
    """Seeded polycrystalline fields, (U, Ny, Nx) doubles on the device."""
    rng = random.Random(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.arange(Nx, device="cuda", dtype=torch.float64)[None, :] * dx
    y = torch.arange(Ny, device="cuda", dtype=torch.float64)[:, None] * dx
    W, H = Nx * dx, Ny * dx
    out = torch.empty((len(mean), Ny, Nx), device="cuda", dtype=torch.float64)
    centres = [(rng.random() * W, rng.random() * H, rng.random() * math.pi / 3) for _ in range(grains)]
    best = torch.full((Ny, Nx), math.inf, device="cuda", dtype=torch.float64)
    cs = torch.ones_like(best)
    sn = torch.zeros_like(best)
    for cx, cy, th in centres:
        ddx = torch.remainder(x - cx + 0.5 * W, W) - 0.5 * W
        ddy = torch.remainder(y - cy + 0.5 * H, H) - 0.5 * H
        d2 = ddx * ddx + ddy * ddy
        near = d2 < best
        best = torch.where(near, d2, best)
        cs = torch.where(near, math.cos(th), cs)
        sn = torch.where(near, math.sin(th), sn)
    X, Y = x * cs + y * sn, y * cs - x * sn
    for u in range(len(mean)):
        qx = 2.0 * math.pi / lat[u]
        qy = qx / math.sqrt(3.0)
        out[u] = mean[u] + amp[u] * (torch.cos(qx * X) * torch.cos(qy * Y) + 0.5 * torch.cos(2.0 * qy * Y))
        out[u] += 0.01 * torch.randn((Ny, Nx), device="cuda", dtype=torch.float64, generator=gen)
    return out


def relax_problem(case, seed):
    d, dt, dx, mean, amp, lat = model(case["U"], case.get("conserved", True), case.get("modes", 1))
    p = P.make_params(d, 1.0 if case.get("conserved", True) else 0.0, dt)
    return p, dx, states(case["Nx"], case["Ny"], dx, mean, amp, lat, seed)


def batch_problems(case, seed):
    """[(Params, N, dx, fields)] of a batch: sizes and field counts from `pick`, states from the seed."""
    rng = random.Random(case["pick"])
    out = []
    for i in range(case["problems"]):
        N, U = rng.choice(BATCH_SIZES), rng.choice((1, 2))
        d, dt, dx, mean, amp, lat = model(U)
        out.append((P.make_params(d, 1.0, dt), N, dx, states(N, N, dx, mean, amp, lat, seed * 1000 + i)))
    return out


def network_weights(case, seed):
    if case["kind"] == "apply":
        return fno.load_weights()
    return fno.init_params(seed, out_scale=1.0)


def network_tiles(case, seed):
    """(inputs, targets) of a training step: [batch, 2, tile, tile] FP32 pairs of states."""
    T, B = case["tile"], case["batch"]
    _, _, dx, mean, amp, lat = model(2)
    x = torch.stack([states(T, T, dx, mean, amp, lat, seed * 100 + i, grains=2) for i in range(B)])
    y = torch.stack([states(T, T, dx, mean, amp, lat, seed * 100 + 50 + i, grains=2) for i in range(B)])
    return x.float().contiguous(), y.float().contiguous()


# ------------------------------------------------------------------ the passes

def prepare(case, seed):
    kind = case["kind"]
    if kind == "relax":
        p, dx, f0 = relax_problem(case, seed)
        r = lib.Relaxation(p, case["Nx"], case["Ny"], dx, dx, case["precision"], case["scheme"])
        torch.cuda.synchronize()
        r.upload_device(f0.data_ptr())
        s = {"case": case, "r": r, "d": 1e-4, "fields": torch.empty_like(f0)}
        if case["precision"] == "fp32":
            s["single"] = torch.empty(f0.shape, device="cuda", dtype=torch.float32)
        return s
    if kind == "batch":
        probs = batch_problems(case, seed)
        b = lib.Batch([(p, N, N, dx, dx) for p, N, dx, _ in probs], "fp32", autotune=True)
        torch.cuda.synchronize()
        for q, (_, _, _, f0) in zip(b.problems, probs):
            q.upload_device(f0.data_ptr())
        n = sum(f0.numel() for *_, f0 in probs)
        return {"case": case, "b": b, "fields": torch.empty(n, device="cuda", dtype=torch.float64),
                "single": torch.empty(n, device="cuda", dtype=torch.float32)}
    if kind == "snapshot":
        p, dx, f0 = relax_problem(case, seed)
        r = lib.Relaxation(p, case["Nx"], case["Ny"], dx, dx, case["precision"])
        return {"case": case, "r": r, "host": f0.cpu().numpy()}
    net = fno.Network(case["tile"], case["batch"])
    net.set_params(network_weights(case, seed))
    if kind == "train":
        x, y = network_tiles(case, seed)
        torch.cuda.synchronize()
        return {"case": case, "net": net, "x": x, "y": y}
    _, _, dx, mean, amp, lat = model(2)
    f0 = states(case["Nx"], case["Ny"], dx, mean, amp, lat, seed)
    return {"case": case, "net": net, "x": f0, "out": torch.empty_like(f0)}


def in_single(s, stream):
    """The downloaded fields in the precision they were computed in, ordered on the relaxation's own stream."""
    with torch.cuda.stream(torch.cuda.ExternalStream(stream)):
        s["single"].copy_(s["fields"])
    return s["single"]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "relax":
        r = s["r"]
        r.step(case["steps"])
        if case["optimise"]:
            s["d"] = r.optimize(1, 1, s["d"])
        f, nave = r.evaluate()
        r.download_device(s["fields"].data_ptr())
        box = np.array(r.box())
        if case["precision"] == "fp32":
            return {"fields": in_single(s, r.stream), "f": np.float32(f), "nave": nave, "box": box.astype(np.float32)}
        return {"fields": s["fields"], "f": f, "nave": nave, "box": box}
    if kind == "batch":
        b, at, f = s["b"], 0, []
        b.step(case["steps"])
        for q in b.problems:
            f.append(q.evaluate()[0])
            q.download_device(s["fields"].data_ptr() + 8 * at)
            at += q.U * q.Nx * q.Ny
        return {"fields": in_single(s, b.stream), "f": np.array(f, dtype=np.float32)}
    if kind == "snapshot":
        r = s["r"]
        r.upload(s["host"])
        f, nave, fr = r.evaluate(want_f=True)
        out = r.download()
        if case["precision"] == "fp32":
            return {"f": np.float32(f), "nave": nave, "fr": fr.astype(np.float32), "fields": out.astype(np.float32)}
        return {"f": f, "nave": nave, "fr": fr, "fields": out}
    if kind == "train":
        loss, grad = s["net"].loss_grad(s["x"].data_ptr(), s["y"].data_ptr(), case["batch"], want_grad=True)
        return {"loss": np.float32(loss), "grad": grad}
    s["net"].apply(s["x"].data_ptr(), s["out"].data_ptr(), case["Nx"], case["Ny"],
                   torch.cuda.current_stream().cuda_stream)
    return {"fields": s["out"].float()}


# ------------------------------------------------------------------------ work

def step_work(Nx, Ny, U, precision):
    """One step: the transforms of a grid larger than the chip's memory take two sweeps each way over
    the half spectrum, read and written in each, beside the spectral state, read and written once."""
    half = (Nx // 2 + 1) * Ny * U
    size = 8 if precision == "fp32" else 16
    fft = 2 * 2.5 * Nx * Ny * math.log2(Nx * Ny) * U
    return 6 * size * half, fft + 30.0 * Nx * Ny * U


def network_work(tile, batch, backward):
    """Activations of the four layers: each read and written once (and their gradients, with the saved
    pre-activations, on the way back), beside the tiles; channel products and truncated transforms."""
    C, L, MX, MY = fno.CHANNELS, fno.LAYERS, fno.MODES_X, fno.MODES_Y
    pix = batch * tile * tile
    act = 4.0 * C * pix
    fwd_bytes, fwd_flops = L * 2 * act + 4.0 * 4 * pix, L * (2.0 * C * C + 2.0 * C * 4 * MX) * pix
    if not backward:
        return fwd_bytes, fwd_flops
    return fwd_bytes + L * 4 * act, 3 * fwd_flops


def work(case):
    kind = case["kind"]
    if kind == "relax":
        b, f = step_work(case["Nx"], case["Ny"], case["U"], case["precision"])
        return {"bytes": b * case["steps"], "flops": f * case["steps"]}
    if kind == "batch":
        rng = random.Random(case["pick"])
        b = f = 0.0
        for _ in range(case["problems"]):
            N, U = rng.choice(BATCH_SIZES), rng.choice((1, 2))
            x, y = step_work(N, N, U, "fp32")
            b, f = b + x * case["steps"], f + y * case["steps"]
        return {"bytes": b, "flops": f}
    if kind == "snapshot":
        b, f = step_work(case["Nx"], case["Ny"], case["U"], case["precision"])
        pts = case["Nx"] * case["Ny"]
        return {"bytes": 8.0 * pts * (2 * case["U"] + 1) + 2 * b, "flops": 3 * f}
    if kind == "train":
        b, f = network_work(case["tile"], case["batch"], True)
        return {"bytes": b, "flops": f}
    core = case["tile"] // 2
    tiles = -(-case["Nx"] // core) * -(-case["Ny"] // core)
    b, f = network_work(case["tile"], tiles, False)
    return {"bytes": b + 32.0 * case["Nx"] * case["Ny"], "flops": f}


# -------------------------------------------------------------- 64-bit results

class Exact:
    """The relaxation in 64-bit torch: the state is the real fields, whose spectra are taken anew each step."""

    def __init__(self, p, Nx, Ny, dx, dy, fields, scheme="etd1"):
        self.p, self.U, self.Nx, self.Ny, self.m, self.scheme = p, p.U, Nx, Ny, fields.clone(), scheme
        self.set_box(dx, dy)

    def k2(self, dx, dy):
        kx = torch.arange(self.Nx // 2 + 1, device="cuda", dtype=torch.float64) * (2 * math.pi / (dx * self.Nx))
        j = torch.arange(self.Ny, device="cuda", dtype=torch.float64)
        ky = torch.where(j < self.Ny // 2, j, j - self.Ny) * (2 * math.pi / (dy * self.Ny))
        return ky[:, None] ** 2 + kx[None, :] ** 2

    def operator(self, u, k2):
        v = torch.ones_like(k2)
        for w in range(self.p.W[u]):
            v = v * (self.p.omega[u][w] * (self.p.nu2[u][w] - k2) ** 2 + self.p.phi[u][w])
        return v

    def coupling(self, u, v, k2):
        p = self.p
        return p.beta[u][v] * (p.mu2[u][v] - k2) ** 2 + p.epsilon[u][v] * torch.exp(-k2 / p.sigma ** 2)

    def set_box(self, dx, dy):
        p = self.p
        self.dx, self.dy = dx, dy
        k2 = self.k2(dx, dy)
        o = (-k2 if p.c != 0.0 else torch.full_like(k2, -1.0))
        self.A, self.B = [], []
        for u in range(self.U):
            a = p.alpha[u][u] + p.beta[u][u] * self.operator(u, k2)
            x = o * a * p.dt
            if self.scheme == "semi":
                self.A.append(1.0 / (1.0 - x))
                self.B.append(o * p.dt / (1.0 - x))
            else:
                self.A.append(torch.exp(x))
                self.B.append(torch.where(a == 0.0, o * p.dt, torch.expm1(x) / torch.where(a == 0.0, 1.0, a)))
        self.C = {(u, v): self.coupling(u, v, k2) for u in range(self.U) for v in range(u + 1, self.U)}

    def step(self, n):
        p, m = self.p, self.m
        for _ in range(n):
            nl = []
            for u in range(self.U):
                x = m[u]
                t = p.lambda_[u] + x * x * (p.gamma[u][u] + p.delta[u] * x)
                for v in range(self.U):
                    if v != u:
                        i, j = min(u, v), max(u, v)
                        t = t + p.alpha[i][j] * m[v] + 0.5 * p.gamma[i][j] * (2.0 * x * m[v] + m[v] * m[v])
                nl.append(torch.fft.rfft2(t))
            s = [torch.fft.rfft2(m[u]) for u in range(self.U)]
            for (u, v), c in self.C.items():
                nl[u] += c * s[v]
                nl[v] += c * s[u]
            for u in range(self.U):
                m[u] = torch.fft.irfft2(self.A[u] * s[u] + self.B[u] * nl[u], s=(self.Ny, self.Nx))

    def local(self):
        p, m = self.p, self.m
        f = torch.zeros_like(m[0])
        for u in range(self.U):
            x = m[u]
            f += p.lambda_[u] * x + 0.5 * p.alpha[u][u] * x ** 2 + p.gamma[u][u] / 3.0 * x ** 3 + 0.25 * p.delta[u] * x ** 4
            for v in range(u + 1, self.U):
                f += p.alpha[u][v] * x * m[v] + 0.5 * p.gamma[u][v] * (x * x * m[v] + x * m[v] ** 2)
        return f

    def density(self):
        """f(r) of the current box."""
        p, m, shape = self.p, self.m, (self.Ny, self.Nx)
        k2 = self.k2(self.dx, self.dy)
        s = [torch.fft.rfft2(m[u]) for u in range(self.U)]
        eta = [torch.fft.irfft2(torch.exp(-0.5 * k2 / p.sigma ** 2) * s[u], s=shape) for u in range(self.U)]
        f = self.local()
        for u in range(self.U):
            f += 0.5 * p.beta[u][u] * m[u] * torch.fft.irfft2(self.operator(u, k2) * s[u], s=shape)
            for v in range(u + 1, self.U):
                f += p.beta[u][v] * m[u] * torch.fft.irfft2((p.mu2[u][v] - k2) ** 2 * s[v], s=shape)
                f += p.epsilon[u][v] * eta[u] * eta[v]
        return f

    def energy(self, boxes):
        """<f> of the current fields for each of the boxes."""
        p, n = self.p, self.Nx * self.Ny
        s = [torch.fft.rfft2(self.m[u]) / n for u in range(self.U)]
        w = torch.full((self.Nx // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
        w[0] = w[-1] = 1.0
        local, out = float(self.local().mean()), []
        for dx, dy in boxes:
            k2 = self.k2(dx, dy)
            e = torch.zeros_like(k2)
            for u in range(self.U):
                e += 0.5 * p.beta[u][u] * self.operator(u, k2) * (s[u].real ** 2 + s[u].imag ** 2)
                for v in range(u + 1, self.U):
                    e += self.coupling(u, v, k2) * (s[u].real * s[v].real + s[u].imag * s[v].imag)
            out.append(local + float((e * w).sum()))
        return out

    def optimise(self, d):
        x, y = self.dx, self.dy
        f = self.energy([(x, y), (x - d, y), (x + d, y), (x, y - d), (x, y + d)])
        nx = (d * (f[1] - f[2]) + 2 * x * (-2 * f[0] + f[1] + f[2])) / (2 * (f[1] - 2 * f[0] + f[2]))
        ny = (d * (f[3] - f[4]) + 2 * y * (-2 * f[0] + f[3] + f[4])) / (2 * (f[3] - 2 * f[0] + f[4]))
        dr, most = math.hypot(self.Nx * (nx - x), self.Ny * (ny - y)), math.pi / math.sqrt(3.0)
        if dr > most:
            q = most / dr
            nx, ny = q * nx + (1 - q) * x, q * ny + (1 - q) * y
        self.set_box(nx, ny)


def exact_network(flat, x):
    """The network on [B, 2, T, T] doubles with the given (BF16-valued) weights, as the header defines it."""
    w = {k: flat[o:o + int(np.prod(s))].reshape(s) for k, (o, s) in fno.layout().items()}
    T, MX, MY = x.shape[-1], fno.MODES_X, fno.MODES_Y
    rows = list(range(MY // 2)) + list(range(T - MY // 2, T))
    v = torch.einsum("ci,bixy->bcxy", w["P"], x) + w["p"][None, :, None, None]
    for l in range(fno.LAYERS):
        V = torch.fft.rfft2(v)[:, :, rows, :MX]
        R = torch.complex(w["Rr%d" % l], w["Ri%d" % l])
        full = torch.zeros(v.shape[0], v.shape[1], T, T // 2 + 1, device=v.device, dtype=V.dtype)
        full[:, :, rows, :MX] = torch.einsum("bikm,iokm->bokm", V, R)
        z = torch.einsum("oi,bixy->boxy", w["W%d" % l], v) + w["b%d" % l][None, :, None, None] \
            + torch.fft.irfft2(full, s=(T, T))
        v = torch.nn.functional.gelu(z) if l < fno.LAYERS - 1 else z
    return x + torch.einsum("jc,bcxy->bjxy", w["Q"], v) + w["q"][None, :, None, None]


def exact(case, seed):
    kind = case["kind"]
    if kind == "relax":
        p, dx, f0 = relax_problem(case, seed)
        e = Exact(p, case["Nx"], case["Ny"], dx, dx, f0, case["scheme"])
        e.step(case["steps"])
        if case["optimise"]:
            e.optimise(1e-4)
        f = e.energy([(e.dx, e.dy)])[0]
        return {"fields": e.m, "f": f, "nave": e.m.mean(dim=(1, 2)), "box": np.array([e.dx, e.dy])}
    if kind == "batch":
        fields, f = [], []
        for p, N, dx, f0 in batch_problems(case, seed):
            e = Exact(p, N, N, dx, dx, f0)
            e.step(case["steps"])
            f.append(e.energy([(dx, dx)])[0])
            fields.append(e.m.reshape(-1))
        return {"fields": torch.cat(fields), "f": np.array(f)}
    if kind == "snapshot":
        p, dx, f0 = relax_problem(case, seed)
        e = Exact(p, case["Nx"], case["Ny"], dx, dx, f0)
        return {"f": e.energy([(dx, dx)])[0], "nave": f0.mean(dim=(1, 2)), "fr": e.density(), "fields": f0}
    w = torch.tensor(fno.bf16_round(network_weights(case, seed)), device="cuda", dtype=torch.float64)
    if kind == "train":
        w.requires_grad_(True)
        x, y = (t.double() for t in network_tiles(case, seed))
        total = 0.0
        for i in range(case["batch"]):  # one tile at a time: the gradient adds up
            part = ((exact_network(w, x[i:i + 1]) - y[i:i + 1]) ** 2).sum() / x.numel()
            part.backward()
            total += float(part.detach())
        return {"loss": total, "grad": w.grad}
    _, _, dx, mean, amp, lat = model(2)
    Nx, Ny, T = case["Nx"], case["Ny"], case["tile"]
    f0 = states(Nx, Ny, dx, mean, amp, lat, seed)
    out, halo, core = torch.empty_like(f0), T // 4, T // 2
    with torch.no_grad():
        for by in range(-(-Ny // core)):
            ys = (torch.arange(T, device="cuda") + by * core - halo) % Ny
            ye = min(core, Ny - by * core)
            for bx in range(-(-Nx // core)):
                xs = (torch.arange(T, device="cuda") + bx * core - halo) % Nx
                xe = min(core, Nx - bx * core)
                v = exact_network(w, f0[:, ys][:, :, xs].float().double()[None])[0]
                out[:, by * core:by * core + ye, bx * core:bx * core + xe] = v[:, halo:halo + ye, halo:halo + xe]
    return {"fields": out - (out - f0).mean(dim=(1, 2), keepdim=True)}
