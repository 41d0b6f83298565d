"""Workloads of the lattice library and its emulator, for timing and comparison.

Each case is one piece of work that a program built on this package asks for
through its public entry points:

  lattice   one output interval of a run (`gabe_b200.Lattice`): the steps
            between two outputs -- queued at once, or one by one with the
            energies read after each, as the drop-in driver does -- then the
            scalars, the |k|-binned spectra and the state
  output    what an output slice of a run reads: spectra, means and
            variances, a plane of field values (no steps)
  ensemble  an output interval of a batched parameter sweep: steps of many
            lattices of uneven size, then every lattice's log spectra
  forward   emulator queries (`gabe_b200.emulator.MLP.forward`)
  train     one pass over a training set in shuffled batches

`listed` gives fixed ones, `draw` others of the same ranges, `prepare` what a
program holds before the call, `run` one pass, `work` what a pass cannot do
without, and `exact` the same outputs from plain FP64 tensor arithmetic.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gabe_b200 as gb
from gabe_b200 import emulator, ensemble

L_BOX, PHI0, G2_OVER_LAMBDA = 20.0, 0.342, 100.0
LAM, GSQ = 1.0 / PHI0 ** 2, G2_OVER_LAMBDA / PHI0 ** 2  # program units
AMPLITUDE = math.sqrt(9e-14) * PHI0
MLP_SHAPE = (4, 256, 4, 192)  # inputs, width, hidden layers, outputs


def listed():
    return [
        # the drop-in driver on the 64^3 FP64 run: every step's energies are read, spectra every 100 steps
        {"name": "driver_64_fp64", "kind": "lattice", "N": 64, "precision": "fp64", "gws": False, "steps": 100,
         "dt": 0.01, "each_step": True},
        # the lattice re-run of one parameter point that the emulator flagged
        {"name": "rerun_64_fp32_gw", "kind": "lattice", "N": 64, "precision": "fp32", "gws": True, "steps": 50,
         "dt": 0.01, "each_step": False},
        # a size that is no power of two
        {"name": "run_96_fp32_gw", "kind": "lattice", "N": 96, "precision": "fp32", "gws": True, "steps": 250,
         "dt": 0.01, "each_step": False},
        # an ordinary single run with gravitational waves
        {"name": "run_128_fp32_gw", "kind": "lattice", "N": 128, "precision": "fp32", "gws": True, "steps": 250,
         "dt": 0.01, "each_step": False},
        # preheating without gravitational waves: the field sweeps alone
        {"name": "fields_256_fp32", "kind": "lattice", "N": 256, "precision": "fp32", "gws": False, "steps": 250,
         "dt": 0.01, "each_step": False},
        # the reference's own precision with gravitational waves
        {"name": "run_256_fp64_gw", "kind": "lattice", "N": 256, "precision": "fp64", "gws": True, "steps": 50,
         "dt": 0.01, "each_step": False},
        # the headline lattice, at a time step inside the stability region
        {"name": "run_512_fp32_gw", "kind": "lattice", "N": 512, "precision": "fp32", "gws": True, "steps": 100,
         "dt": L_BOX / 512 / 40, "each_step": False},
        # an output slice of the headline lattice
        {"name": "output_512_fp32_gw", "kind": "output", "N": 512, "precision": "fp32", "gws": True, "steps": 2,
         "dt": L_BOX / 512 / 40},
        # the parameter sweep: 256 lattices of 32^3 .. 128^3, log spectra every 50 steps
        {"name": "ensemble_256", "kind": "ensemble", "lattices": 256, "steps": 50, "gws": True, "nlog": 64},
        # one parameter point's history (41 output times) from the emulator: the smallest call
        {"name": "query_41", "kind": "forward", "rows": 41, "fp32_act": False},
        # screening a large parameter grid
        {"name": "forward_1m", "kind": "forward", "rows": 1 << 20, "fp32_act": False},
        # one epoch over ~20k (parameter, time) samples
        {"name": "train_epoch", "kind": "train", "samples": 20000, "batch": 512, "fp32_act": False},
    ]


def draw(rng):
    def log_uniform(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choices(("lattice", "output", "ensemble", "forward", "train"), (9, 3, 2, 4, 2))[0]
    if kind in ("lattice", "output"):
        # FP32 storage takes multiples of 16, FP64 multiples of 4
        fp32 = rng.random() < 0.6
        q = 16 if fp32 else 4
        N = max(q, int(round(log_uniform(32, 400 if fp32 else 256) / q)) * q)
        case = {"kind": kind, "N": N, "precision": "fp32" if fp32 else "fp64", "gws": rng.random() < 0.7}
        dt = round(min(0.01, L_BOX / N / 8) * rng.uniform(0.5, 1.0), 5)
        if kind == "output":
            return dict(case, steps=rng.randint(1, 4), dt=dt)
        each = rng.random() < 0.3
        steps = int(min(250, max(10, 4e8 / N ** 3)) * rng.uniform(0.7, 1.0))
        return dict(case, steps=steps, dt=dt, each_step=each)
    if kind == "ensemble":
        return {"kind": kind, "lattices": int(log_uniform(4, 200)), "steps": rng.randint(10, 50),
                "gws": rng.random() < 0.85, "nlog": rng.choice((32, 64))}
    if kind == "forward":
        fp32_act = rng.random() < 0.2
        return {"kind": kind, "rows": int(log_uniform(1, 1 << (17 if fp32_act else 20))), "fp32_act": fp32_act}
    return {"kind": kind, "samples": int(log_uniform(2000, 30000)), "batch": int(log_uniform(64, 1500)),
            "fp32_act": rng.random() < 0.2}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _initial_state(N, seed):
    """Vacuum fluctuations about the homogeneous inflaton: FP64 fields and
    momenta [2][N][N][N], and the adot of the homogeneous energy."""
    dev = _device()
    g = _generator(seed, dev)
    f = torch.empty((2, N, N, N), dtype=torch.float64, device=dev)
    d = torch.empty_like(f)
    hubble = math.sqrt(8 * math.pi / 3 * 0.25 * LAM * PHI0 ** 4)
    n2 = _n2(N, dev)
    for q, m2 in enumerate((3 * LAM * PHI0 ** 2, GSQ * PHI0 ** 2)):
        omega = torch.sqrt(n2 * (2 * math.pi / L_BOX) ** 2 + m2)
        amp = AMPLITUDE * N ** 1.5 / torch.sqrt(2 * omega * L_BOX ** 3)
        amp[0, 0, 0] = 0
        w = torch.fft.rfftn(torch.randn((N, N, N), generator=g, device=dev, dtype=torch.float64))
        f[q] = torch.fft.irfftn(w.mul_(amp), s=(N, N, N))
        w = torch.fft.rfftn(torch.randn((N, N, N), generator=g, device=dev, dtype=torch.float64))
        d[q] = torch.fft.irfftn(w.mul_(amp.mul_(omega)), s=(N, N, N)).sub_(f[q], alpha=hubble)
        del w, amp, omega
    f[0] += PHI0
    return f, d, hubble


def _mlp_data(seed, rows, targets):
    """Standardised inputs and targets, and the network's parameters (flat)."""
    dev = _device()
    g = _generator(seed, dev)
    n_in, width, depth, n_out = MLP_SHAPE
    sizes = [n_in] + [width] * depth + [n_out]
    flat = []
    for k, n in zip(sizes[:-1], sizes[1:]):
        flat.append((2 * torch.rand((k, n), generator=g, device=dev) - 1).mul_(math.sqrt(6 / (k + n))).reshape(-1))
        flat.append(0.02 * torch.randn(n, generator=g, device=dev))
    x = torch.randn((rows, n_in), generator=g, device=dev)
    t = None
    if targets:
        mix = torch.randn((n_in, n_out), generator=g, device=dev)
        t = torch.tanh(x @ mix) + 0.1 * torch.randn((rows, n_out), generator=g, device=dev)
        # log bins without native bins hold NaN
        t[:, torch.rand(n_out, generator=g, device=dev) < 0.1] = float("nan")
    return torch.cat(flat), x, t, g


def _permutation(case, g):
    n, batch = case["samples"], min(case["batch"], case["samples"])
    nb = n // batch
    return torch.randperm(n, generator=g, device=_device())[: nb * batch].to(torch.int32).contiguous(), batch, nb


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("lattice", "output"):
        N = case["N"]
        f, d, adot = _initial_state(N, seed)
        lat = gb.Lattice(N, L=L_BOX, dt=case["dt"], gws=case["gws"], tile_shape="auto",
                         precision=gb.FP32 if case["precision"] == "fp32" else gb.FP64)
        shape = (2, N, N, N)
        host = [torch.empty(shape, dtype=torch.float64, pin_memory=True) for _ in range(2)]
        # h and l come back whole up to 96^3; above, a program reads them as spectra
        if case["gws"] and kind == "lattice" and N <= 96:
            host += [torch.empty((12, N, N, N // 2 + 1), dtype=torch.float64, pin_memory=True) for _ in range(2)]
        host[0].copy_(f)
        host[1].copy_(d)
        del f, d
        torch.cuda.empty_cache()
        lat.upload_ptrs(host[0].data_ptr(), host[1].data_ptr(), None, None, 1.0, adot)
        if kind == "output":
            lat.step(case["steps"])
            lat.sync()
        return {"case": case, "lat": lat, "host": host}
    if kind == "ensemble":
        N, g, amp, seeds = ensemble.sample_parameters(case["lattices"], int(seed))
        ens = gb.Ensemble(N, g, amp, seeds, L=L_BOX, gws=case["gws"], nlog=case["nlog"], tiles="auto",
                          log_top_bin=gb.numbins(max(ensemble.SIZES)))
        ens.init()
        return {"case": case, "ens": ens}
    rows = case["rows"] if kind == "forward" else case["samples"]
    flat, x, t, g = _mlp_data(seed, rows, kind == "train")
    n_in, width, depth, n_out = MLP_SHAPE
    net = emulator.MLP(n_in=n_in, width=width, depth=depth, n_out=n_out, fp32_act=case["fp32_act"],
                       max_rows=max(1024, min(rows, 1 << 20) if kind == "forward" else case["batch"]))
    net.set_params(flat.cpu().numpy())
    state = {"case": case, "net": net, "x": x, "t": t}
    if kind == "train":
        state["perm"], state["batch"], state["nb"] = _permutation(case, g)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _stored(case, v):
    """Quantities whose digits are those of the storage precision."""
    v = torch.as_tensor(v)
    return v.to(torch.float32) if case["precision"] == "fp32" else v


def _spectra(case, table):
    """The spectra table by column, the zero-mode bin apart (it holds the mean)."""
    table = torch.as_tensor(table)
    out = {"k": table[:, 0].contiguous(), "zero_mode": _stored(case, table[0])}
    names = ("P_phi", "D2_phi", "P_chi", "D2_chi", "P_gw", "Omega_gw")
    for c, name in enumerate(names[: table.shape[1] - 1], 1):
        out[name] = _stored(case, table[1:, c].contiguous())
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "lattice":
        lat, host = state["lat"], state["host"]
        out = {}
        if case["each_step"]:
            energies = []
            for _ in range(case["steps"]):
                lat.step(1)
                energies.append(list(lat.calc_energy().values()))
            out["energies"] = np.array(energies)
        else:
            lat.step(case["steps"])
        out["scalars"] = np.array(list(lat.scalars().values()))
        out["spectra"] = _spectra(case, lat.spec_out())
        lat.download_ptrs(*[h.data_ptr() for h in host])
        # FP32 storage keeps phi about its homogeneous value in FP64; chi's is zero
        out["state"] = {"phi": host[0][0], "dphi": host[1][0], "chi": _stored(case, host[0][1]),
                        "dchi": _stored(case, host[1][1])}
        if len(host) > 2:
            out["state"].update(h=_stored(case, host[2]), l=_stored(case, host[3]))
        return out
    if kind == "output":
        lat = state["lat"]
        mv = lat.meansvars()
        rows = lat.field_slice(2, 2)
        return {"spectra": _spectra(case, lat.spec_out()), "means": mv[:, 0].copy(),
                "variances": _stored(case, mv[:, 1].copy()), "phi": rows[:, 0].copy(),
                "chi": _stored(case, rows[:, 1].copy()), "rho": rows[:, 2].copy()}
    if kind == "ensemble":
        ens = state["ens"]
        ens.step(case["steps"])
        logs, counts, native = ens.log_spectra()
        # FP32 storage: the spectra carry its digits
        return {"log_spectra": logs.astype(np.float32), "counts": counts, "native": native[:, :3].astype(np.float32),
                "native_counts": native[:, 3].copy(), "scalars": ens.scalars()}
    net = state["net"]
    if kind == "forward":
        return net.forward(state["x"])
    net.reset_batches()
    net.train_batches(state["x"], state["t"], state["perm"], state["batch"], state["nb"])
    loss, steps = net.train_loss()
    return {"params": net.get_params(), "loss": np.float32(loss), "steps": steps}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _mlp_macs():
    n_in, width, depth, n_out = MLP_SHAPE
    return n_in * width + (depth - 1) * width * width + width * n_out


def _step_work(N, w, gws):
    """Bytes and operations of one step: the state read once and written once
    (fields, momenta and, with gravitational waves, four complex amplitudes
    per k-point); about 100 operations per site and stage for the fields,
    and ten real 3-D transforms plus the projection and update of h, l."""
    sites, modes = N ** 3, N * N * (N // 2 + 1)
    bytes_, flops = 2 * 4 * sites * w, 200 * sites
    if gws:
        bytes_ += 2 * 8 * modes * w
        flops += 10 * 2.5 * sites * 3 * math.log2(N) + 200 * modes
    return bytes_, flops


def work(case):
    kind = case["kind"]
    if kind in ("lattice", "output"):
        N, w = case["N"], 4 if case["precision"] == "fp32" else 8
        sites, modes = N ** 3, N * N * (N // 2 + 1)
        # spectra: two fields read, transformed and binned, with the momenta of h
        out_b = 2 * sites * w + (4 * modes * w if case["gws"] else 0)
        out_f = 2 * 2.5 * sites * 3 * math.log2(N) + 40 * modes
        if kind == "output":
            rows = (N // 2) ** 2
            return {"bytes": out_b + 24 * rows, "flops": out_f + 8 * sites}
        b, f = _step_work(N, w, case["gws"])
        down = 4 * sites * (w + 8)
        if case["gws"] and N <= 96:
            down += 8 * modes * w + 24 * modes * 8
        return {"bytes": case["steps"] * b + out_b + down, "flops": case["steps"] * f + out_f}
    if kind == "ensemble":
        # the expected sum over sizes drawn uniformly
        b = f = 0.0
        for N in ensemble.SIZES:
            sb, sf = _step_work(N, 4, case["gws"])
            b += case["steps"] * sb + 8 * N ** 3
            f += case["steps"] * sf + 15 * N ** 3 * math.log2(N)
        share = case["lattices"] / len(ensemble.SIZES)
        return {"bytes": share * b, "flops": share * f}
    n_in, width, depth, n_out = MLP_SHAPE
    params = _mlp_macs() + depth * width + n_out
    if kind == "forward":
        return {"bytes": 4 * case["rows"] * (n_in + n_out) + 4 * params, "flops": 2.0 * case["rows"] * _mlp_macs()}
    batch = min(case["batch"], case["samples"])
    nb = case["samples"] // batch
    # per batch: its rows, and parameters and moments read and written
    return {"bytes": nb * (4 * batch * (n_in + n_out) + 6 * 4 * params), "flops": nb * 6.0 * batch * _mlp_macs()}


# ---------------------------------------------------------------------------
# the same outputs in plain FP64
# ---------------------------------------------------------------------------
def _n2(N, dev):
    i = torch.arange(N, device=dev, dtype=torch.float64)
    i = torch.where(i <= N // 2, i, i - N)
    k = torch.arange(N // 2 + 1, device=dev, dtype=torch.float64)
    return i[:, None, None] ** 2 + i[None, :, None] ** 2 + k[None, None, :] ** 2


def _roll(x, shift, axis):
    return torch.roll(x, shift, axis)


class _Exact:
    """The step and the outputs of one lattice in FP64 tensors."""

    def __init__(self, case, seed):
        self.N, self.dt, self.gws = case["N"], case["dt"], case["gws"]
        self.dx = L_BOX / self.N
        self.f, self.d, self.adot = _initial_state(self.N, seed)
        self.a = 1.0
        self.stage1 = None
        self.e = self.energies(self.f, self.d, self.a)
        self.h = self.l = None
        if self.gws:
            dev, N = self.f.device, self.N
            self.h = torch.zeros((6, N, N, N // 2 + 1), dtype=torch.complex128, device=dev)
            self.l = torch.zeros_like(self.h)
            self.n2 = _n2(N, dev)
            i = torch.arange(N, device=dev, dtype=torch.float64)
            i = torch.where(i <= N // 2, i, i - N)
            k = torch.arange(N // 2 + 1, device=dev, dtype=torch.float64)
            inv = torch.where(self.n2 > 0, self.n2, torch.ones_like(self.n2)).rsqrt()
            u = (i[:, None, None] * inv, i[None, :, None] * inv, k[None, None, :] * inv)
            self.P = {(a, b): (1.0 if a == b else 0.0) - u[a] * u[b] for a in range(3) for b in range(a, 3)}

    @staticmethod
    def potential(f):
        return 0.25 * LAM * f[0] ** 4 + 0.5 * GSQ * f[0] ** 2 * f[1] ** 2

    @staticmethod
    def force(f, q):
        return LAM * f[0] ** 3 + GSQ * f[1] ** 2 * f[0] if q == 0 else GSQ * f[0] ** 2 * f[1]

    def laplacian(self, x):
        y = -6.0 * x
        for ax in range(3):
            y += _roll(x, -1, ax)
            y += _roll(x, 1, ax)
        return y.div_(self.dx * self.dx)

    def energies(self, f, d, a):
        kin = 0.5 * float((d[0] ** 2 + d[1] ** 2).mean())
        pot = float(self.potential(f).mean())
        grad = 0.0
        for q in range(2):
            for ax in range(3):
                grad += float((_roll(f[q], -1, ax) - f[q]).square_().mean())
        grad *= 0.5 / (self.dx * self.dx) / a ** 2
        return kin, pot, grad, kin + pot + grad

    def source(self, f, dxx):
        """dx^3 times the transverse-traceless part of the transformed source."""
        S = [None] * 6
        pairs = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))
        for q in range(2):
            g = [(_roll(f[q], -1, ax) - _roll(f[q], 1, ax)).mul_(0.5 / self.dx) for ax in range(3)]
            for c, (a, b) in enumerate(pairs):
                p = g[a] * g[b]
                S[c] = p if S[c] is None else S[c].add_(p)
        tr = (S[0] + S[3] + S[5]) / 3
        for c in (0, 3, 5):
            S[c] -= tr
        S = [torch.fft.rfftn(s).mul_(dxx) for s in S]
        at = {p: c for c, p in enumerate(pairs)}
        full = lambda M, a, b: M[(a, b)] if a <= b else M[(b, a)]  # noqa: E731
        Sm = {p: S[c] for p, c in at.items()}
        PS = {(a, b): sum(full(self.P, a, m) * full(Sm, m, b) for m in range(3)) for a in range(3) for b in range(3)}
        trace = PS[(0, 0)] + PS[(1, 1)] + PS[(2, 2)]
        T = []
        for a, b in pairs:
            t = sum(PS[(a, m)] * full(self.P, m, b) for m in range(3)) - 0.5 * self.P[(a, b)] * trace
            t[0, 0, 0] = 0
            T.append(t)
        return T

    def gw_rate(self, h, l, T, a, adot, c):
        kk = self.n2 * ((2 * math.pi / L_BOX) ** 2 / a ** 2)
        return -kk * h - (3 * adot / a) * l + (16 * math.pi / a ** 2) * T[c]

    def step(self):
        dt, hdt, a0, ad0 = self.dt, 0.5 * self.dt, self.a, self.adot
        f1 = self.f + hdt * self.d
        d1 = torch.empty_like(self.d)
        for q in range(2):
            rate = self.laplacian(self.f[q]) / a0 ** 2 - self.force(self.f, q) - 3 * ad0 / a0 * self.d[q]
            d1[q] = self.d[q] + hdt * rate
        a1 = a0 + hdt * ad0
        e1 = self.energies(f1, d1, a1)
        ad1 = math.sqrt(8 * math.pi / 3 * e1[3]) * a1
        if self.gws:
            T0, T1 = self.source(self.f, self.dx ** 3), self.source(f1, self.dx ** 3)
            for c in range(6):
                h0, l0 = self.h[c], self.l[c]
                l1 = l0 + hdt * self.gw_rate(h0, l0, T0, a0, ad0, c)
                h1 = h0 + hdt * l0
                self.l[c] = l0 + dt * self.gw_rate(h1, l1, T1, a1, ad1, c)
                self.h[c] = h0 + dt * l1
        self.f = self.f + dt * d1
        d0 = self.d
        self.d = torch.empty_like(d0)
        for q in range(2):
            rate = self.laplacian(f1[q]) / a1 ** 2 - self.force(f1, q) - 3 * ad1 / a1 * d1[q]
            self.d[q] = d0[q] + dt * rate
        self.a = a0 + dt * ad1
        self.e = self.energies(self.f, self.d, self.a)
        self.adot = math.sqrt(8 * math.pi / 3 * self.e[3]) * self.a
        self.stage1 = (a1, ad1, e1)

    def scalars(self):
        a1, ad1, e1 = self.stage1
        rows = [(self.a, a1), (self.adot, ad1)] + [(self.e[c], e1[c]) for c in range(4)]
        return np.array(rows)

    def spectra(self):
        N, dev = self.N, self.f.device
        n2 = _n2(N, dev)
        nb = int(math.sqrt(3.0) * N / 2 + 1)
        b = torch.sqrt(n2).to(torch.int64).reshape(-1)
        w = torch.full((N // 2 + 1,), 2.0, dtype=torch.float64, device=dev)
        w[0] = w[-1] = 1.0

        def binned(p):
            return torch.bincount(b, (p * w).reshape(-1), minlength=nb)[:nb].cpu()

        cnt = binned(torch.ones_like(n2)).clamp_(min=1)
        q = torch.arange(nb, dtype=torch.float64)
        kb = 2 * math.pi * q / L_BOX
        norm = (L_BOX / N) ** 6 * (2 * math.pi / L_BOX) ** 3
        cols = [kb]
        for x in range(2):
            F = torch.fft.rfftn(self.f[x])
            p = binned(F.real ** 2 + F.imag ** 2) * norm / cnt
            cols += [p, kb ** 3 * p / (2 * math.pi ** 2)]
        if self.gws:
            # the kz = 0 plane is read at kz = N/2, as the reference's loop does
            p = sum(m * (self.l[c].real ** 2 + self.l[c].imag ** 2) for c, m in enumerate((1, 2, 2, 1, 2, 1)))
            p[..., 0] = p[..., -1]
            p = binned(p) / cnt
            hub2 = 8 * math.pi / 3 * self.e[3]
            cols += [p * norm, 4e-5 / 100 ** 0.333 / 24 / math.pi ** 2 / L_BOX ** 3 / hub2 * kb ** 3 * p, kb]
        return torch.stack(cols, 1)

    def density_rows(self):
        """phi, chi and the energy density on every second point of the i = 0 plane."""
        def grad(x, ax):
            return (_roll(x, 2, ax) / 12 - 2 / 3 * _roll(x, 1, ax) + 2 / 3 * _roll(x, -1, ax)
                    - _roll(x, -2, ax) / 12) / self.dx

        rho = self.potential(self.f)
        for q in range(2):
            g2 = sum(grad(self.f[q], ax) ** 2 for ax in range(3))
            rho = rho + 0.5 * self.d[q] ** 2 + 0.5 * g2 / self.a ** 2
        pick = lambda x: x[0, ::2, ::2].reshape(-1).cpu()  # noqa: E731
        return pick(self.f[0]), pick(self.f[1]), pick(rho)


def _components(x):
    """Six complex components as (re, im) of each."""
    return torch.stack([p for c in range(6) for p in (x[c].real, x[c].imag)]).cpu()


def _exact_lattice(case, seed):
    if case["N"] ** 3 * case["steps"] > 6e9:
        return None
    e = _Exact(case, seed)
    wide = dict(case, precision="fp64")
    if case["kind"] == "output":
        for _ in range(case["steps"]):
            e.step()
        phi, chi, rho = e.density_rows()
        mean = [float(e.f[q].mean()) for q in range(2)]
        return {"spectra": _spectra(wide, e.spectra()), "means": np.array(mean),
                "variances": np.array([float((e.f[q] - mean[q]).square().mean()) for q in range(2)]),
                "phi": phi, "chi": chi, "rho": rho}
    out, energies = {}, []
    for _ in range(case["steps"]):
        e.step()
        energies.append([*e.e, e.a, e.adot])
    if case["each_step"]:
        out["energies"] = np.array(energies)
    out["scalars"] = e.scalars()
    out["spectra"] = _spectra(wide, e.spectra())
    f, d = e.f.cpu(), e.d.cpu()
    out["state"] = {"phi": f[0], "dphi": d[0], "chi": f[1], "dchi": d[1]}
    if case["gws"] and case["N"] <= 96:
        out["state"].update(h=_components(e.h), l=_components(e.l))
    return out


def _layers(flat):
    n_in, width, depth, n_out = MLP_SHAPE
    sizes = [n_in] + [width] * depth + [n_out]
    out, o = [], 0
    for k, n in zip(sizes[:-1], sizes[1:]):
        out.append((flat[o:o + k * n].view(k, n), flat[o + k * n:o + k * n + n]))
        o += k * n + n
    return out


def _network(flat, x):
    layers = _layers(flat)
    for W, b in layers[:-1]:
        x = torch.nn.functional.silu(x @ W + b)
    W, b = layers[-1]
    return x @ W + b


def exact(case, seed):
    kind = case["kind"]
    if kind in ("lattice", "output"):
        return _exact_lattice(case, seed)
    if kind == "ensemble":
        return None  # the library draws the initial states
    flat, x, t, g = _mlp_data(seed, case["rows"] if kind == "forward" else case["samples"], kind == "train")
    flat, x = flat.double(), x.double()
    if kind == "forward":
        return torch.cat([_network(flat, part) for part in x.split(1 << 17)])
    perm, batch, nb = _permutation(case, g)
    lr, b1, b2, eps = 1e-3, 0.9, 0.999, 1e-8
    m, v, losses = torch.zeros_like(flat), torch.zeros_like(flat), []
    t = t.double()
    for s in range(nb):
        idx = perm[s * batch:(s + 1) * batch].long()
        flat.requires_grad_(True)
        y, tb = _network(flat, x[idx]), t[idx]
        ok = torch.isfinite(tb)
        loss = ((y - torch.where(ok, tb, torch.zeros_like(tb))) * ok).square().sum() / ok.sum()
        grad, = torch.autograd.grad(loss, flat)
        flat = flat.detach()
        losses.append(float(loss.detach()))
        m.mul_(b1).add_(grad, alpha=1 - b1)
        v.mul_(b2).addcmul_(grad, grad, value=1 - b2)
        flat = flat - lr * (m / (1 - b1 ** (s + 1))) / (torch.sqrt(v / (1 - b2 ** (s + 1))) + eps)
    return {"params": flat, "loss": sum(losses) / len(losses), "steps": None}
