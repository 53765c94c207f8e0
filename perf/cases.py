"""The calls whose time matters to a user of the propagator, one case each.

A case is a dict of plain numbers, texts and truth values.  `listed()` gives
the fixed ones, `draw()` more of the same ranges, `prepare()` what a program
holds before the call, `run()` one pass through the public entry points,
`work()` the bytes and operations a pass cannot do without, and `exact()`
what the same inputs give in float64 in plain torch.

Kinds:
  forward       plain modelling of one model (acoustic_forward_kernel, or
                AcousticPropagator with api='propagator')
  gradient      modelling, misfit and backward of one model
  batch         acoustic_gradient_batched over a list of models
  volume        3-D modelling; volume_gradient: 3-D modelling + backward
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from geobrain_b200 import wave

DEVICE = "cuda:0" if torch.cuda.is_available() else "cpu"
TAPS = {4: (9 / 8, -1 / 24), 8: (1225 / 1024, -245 / 3072, 49 / 5120, -5 / 7168)}


def _case(name, kind, **kw):
    base = dict(kind=kind, api="kernel", nz=100, nx=200, ny=0, nabc=20, dx=10.0, dt=1e-3, nt=100, order=8, shots=1,
                receivers=100, free_surface=False, misfit="l2", imaging="fp32", cache="auto", snapshots="fp32",
                rho=False, wavelet=False, absorbing="damping", models=1, uneven=False)
    base.update(kw)
    return dict(name=name, **base) if name else base


def listed():
    return [
        # One shot on a small model through the propagator object, as an
        # interactive forward-modelling script runs it: all latency.
        _case("forward_small", "forward", api="propagator", nz=100, nx=200, nt=1000, order=4, receivers=200),
        # One shot of a survey-sized model: fills the GPU once, no more.
        _case("forward_one_shot", "forward", nz=400, nx=1200, nabc=30, dt=8e-4, nt=500, receivers=1200),
        # A whole survey modelled at once, 4th order and energy maps (defaults).
        _case("forward_survey", "forward", nz=400, nx=1200, nabc=30, dt=8e-4, nt=150, order=4, shots=32,
              receivers=1200),
        # One FWI iteration of a small section with a free surface and the
        # trace-normalised misfit, through the propagator, everything default.
        _case("gradient_section", "gradient", api="propagator", nz=88, nx=200, nt=600, order=4, shots=40,
              receivers=200, free_surface=True, misfit="normalized"),
        # The gradient of one shot on a small model: one particle of a
        # sampler, or a stochastic (single-shot) update.
        _case("gradient_one_shot", "gradient", nz=100, nx=200, nt=600, order=4, receivers=200),
        # The FWI gradient of a survey with compact imaging fields.
        _case("gradient_survey", "gradient", nz=400, nx=1200, nabc=30, dt=8e-4, nt=160, shots=32, receivers=1200,
              imaging="fp24"),
        # Multi-parameter inversion with source estimation on a ragged grid:
        # gradients of vp, rho and the wavelets under a free surface.
        _case("gradient_multi", "gradient", nz=301, nx=597, nabc=25, nt=240, shots=5, receivers=149,
              free_surface=True, rho=True, wavelet=True),
        # A model whose history does not fit: 16-bit checkpoints, recompute.
        _case("gradient_recompute", "gradient", nz=1000, nx=3000, nabc=40, dx=5.0, dt=4e-4, nt=64, shots=16,
              receivers=3000, imaging="fp24", cache="none", snapshots="fp16"),
        # The gradient under the convolutional absorbing layers.
        _case("gradient_cpml", "gradient", nz=400, nx=1200, nabc=30, dt=8e-4, nt=150, shots=8, receivers=1200,
              imaging="fp24", absorbing="cpml"),
        # An ensemble of unlike models (particles, targets), gradients at once.
        _case("batch_uneven", "batch", nz=256, nx=512, nt=150, shots=8, receivers=512, imaging="fp24", models=12,
              uneven=True),
        # 3-D modelling of a few shots, and its gradient on a ragged volume.
        _case("volume", "volume", nz=200, ny=200, nx=200, nt=30, order=4, shots=4, receivers=2500),
        _case("volume_gradient", "volume_gradient", nz=130, ny=149, nx=171, nabc=18, nt=40, order=4, shots=4,
              receivers=800, free_surface=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "gradient", "gradient", "gradient", "batch", "volume", "volume_gradient"])
    budget = 1.2e9                     # shot x cell x step of a pass; the largest listed case does 3e9
    if kind.startswith("volume"):
        nz, ny, nx = (rng.randint(60, 200) for _ in range(3))
        c = _case(None, kind, nz=nz, ny=ny, nx=nx, nabc=rng.randint(10, 20), order=4, shots=rng.randint(1, 5),
                  receivers=rng.randint(50, 2500), free_surface=rng.random() < 0.5,
                  rho=kind == "volume_gradient" and rng.random() < 0.3)
        cells = c["shots"] * (nz + 2 * c["nabc"]) * (ny + 2 * c["nabc"]) * (nx + 2 * c["nabc"])
        c["nt"] = int(max(8, min(rng.randint(20, 80), budget / 2 / cells)))
        return c
    nz, nx = _log_int(rng, 60, 500), _log_int(rng, 100, 1300)
    order = rng.choice([4, 8])
    shots = _log_int(rng, 1, 40)
    c = _case(None, kind, nz=nz, nx=nx, nabc=rng.randint(12, 40), order=order, shots=shots,
              receivers=rng.randint(10, nx), free_surface=rng.random() < 0.4)
    if kind == "forward":
        c["api"] = rng.choice(["kernel", "propagator"])
    elif kind == "gradient":
        c["misfit"] = rng.choice(["l2", "l2", "normalized"])
        c["imaging"] = rng.choice(["fp32", "fp24", "fp24", "bf16"])
        c["absorbing"] = "cpml" if rng.random() < 0.2 else "damping"
        c["rho"] = rng.random() < 0.25
        c["wavelet"] = rng.random() < 0.2
        if c["absorbing"] == "damping" and rng.random() < 0.25:
            c["cache"], c["snapshots"] = "none", rng.choice(["fp32", "fp24", "fp16"])
    else:
        c["models"] = rng.randint(3, 16)
        c["uneven"] = rng.random() < 0.6
        c["shots"] = rng.randint(1, 12)
        c["imaging"] = rng.choice(["fp32", "fp24"])
        c["nz"], c["nx"] = rng.randint(80, 260), rng.randint(120, 520)
        c["receivers"] = rng.randint(10, c["nx"])
    cells = c["shots"] * c["models"] * (c["nz"] + 2 * c["nabc"]) * (c["nx"] + 2 * c["nabc"])
    c["nt"] = int(max(16, min(_log_int(rng, 60, 1000), budget / cells)))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _ricker(nt, dt, f0):
    n = min(nt, 2 * int(2.2 / f0 / dt / 2) + 1)
    t = (np.arange(nt) - (2 * int(2.2 / f0 / dt / 2) + 1) // 2) * dt
    a = (math.pi * f0 * t) ** 2
    w = (1 - 2 * a) * np.exp(-a)
    w[n:] = 0
    return w.astype(np.float32)


def _smooth(shape, gen, cells):
    """Unit-scale smooth random field: coarse noise, interpolated."""
    coarse = [max(3, s // cells + 2) for s in shape]
    x = torch.randn(1, 1, *coarse, generator=gen)
    mode = "bilinear" if len(shape) == 2 else "trilinear"
    return F.interpolate(x.to(DEVICE), size=tuple(shape), mode=mode, align_corners=True)[0, 0]


def _sub_cases(case):
    """The models of a batch, each as a case of its own."""
    subs = []
    for i in range(case["models"]):
        c = dict(case)
        if case["uneven"]:
            f = (0.5, 1.0, 1.5, 0.75)[i % 4]
            c["nz"], c["nx"] = int(case["nz"] * f) + i % 3, int(case["nx"] * f) + i % 5
            c["shots"] = max(1, (case["shots"], case["shots"] // 2, case["shots"] + 3)[i % 3])
            c["nt"] = max(8, int(case["nt"] * (1.0, 0.7, 1.3)[(i // 2) % 3]))
            c["receivers"] = min(case["receivers"], c["nx"])
        subs.append(c)
    return subs


def _inputs(case, seed):
    """Model, survey, wavelets and observed traces of one model (float32)."""
    gen = torch.Generator().manual_seed(int(seed) & 0x7fffffff)
    three = case["ny"] > 0
    nz, nx, ny, dx, dt, nt, S, NR = (case[k] for k in ("nz", "nx", "ny", "dx", "dt", "nt", "shots", "receivers"))
    shape = (nz, ny, nx) if three else (nz, nx)
    depth = torch.linspace(0, 1, nz, device=DEVICE).reshape(-1, *([1] * (len(shape) - 1)))
    vp = 1700 + 1700 * depth + 200 * _smooth(shape, gen, 9)
    top = torch.randint(1, nz, (4,), generator=gen).tolist()
    for t in top:
        vp[t:t + max(2, nz // 10)] += float(torch.rand(1, generator=gen)) * 500 - 250
    vp = vp.clamp(1500, 4400).to(torch.float32).contiguous()
    rho = (310.0 * vp.double() ** 0.25).float() if case["api"] == "propagator" else \
        (2200 + 100 * _smooth(shape, gen, 12)).to(torch.float32).contiguous()
    spread = np.round(np.linspace(0, nx - 1, S + 2)[1:-1]).astype(np.int64)
    f0 = 10.0 if dx < 10 or nx > 600 else 15.0
    src_v = np.stack([_ricker(nt, dt, f0) * np.float32(1 + 0.05 * (s % 3)) for s in range(S)])
    pos = dict(src_x=spread, src_z=np.full(S, 3 if case["free_surface"] else 1, np.int64))
    if three:
        side = max(1, int(math.sqrt(NR)))
        gx = np.round(np.linspace(0, nx - 1, side)).astype(np.int64)
        gy = np.round(np.linspace(0, ny - 1, -(-NR // side))).astype(np.int64)
        yy, xx = np.meshgrid(gy, gx, indexing="ij")
        pos.update(src_y=np.round(np.linspace(0, ny - 1, S + 2)[1:-1]).astype(np.int64),
                   rcv_x=xx.reshape(-1)[:NR].copy(), rcv_y=yy.reshape(-1)[:NR].copy(),
                   rcv_z=np.full(NR, 2, np.int64))
    else:
        pos.update(rcv_x=np.round(np.linspace(0, nx - 1, NR)).astype(np.int64), rcv_z=np.full(NR, 2, np.int64))
    vmax = float(vp.max())
    if three:
        damp = wave.bc_pml_3d(nx, ny, nz, dx, dx, dx, case["nabc"], vmax, free_surface=False)
    else:
        damp = wave.bc_pml(nx, nz, dx, dx, case["nabc"], vmax, free_surface=False)
    inp = dict(vp=vp, rho=rho, damp=torch.tensor(damp, dtype=torch.float32, device=DEVICE),
               src_v=torch.tensor(src_v, device=DEVICE), pos=pos, vmax=vmax, f0=f0)
    if "gradient" in case["kind"] or case["kind"] == "batch":
        # observed traces: a direct wave of each source at its own speed, with noise
        n = len(pos["rcv_x"])
        off = np.abs(pos["rcv_x"][None, :] - pos["src_x"][:, None]) * dx
        tt = torch.tensor(off / (1600.0 + 300.0 * float(torch.rand(1, generator=gen))), device=DEVICE)[:, None, :]
        t = (torch.arange(nt, device=DEVICE, dtype=torch.float64) * dt)[None, :, None] - tt - 1.1 / f0
        a = (math.pi * f0 * t) ** 2
        obs = 1e-3 * (1 - 2 * a) * torch.exp(-a) / (1 + torch.tensor(off, device=DEVICE)[:, None, :] / 200).sqrt()
        obs = obs + 2e-6 * torch.randn(1, nt, n, generator=gen).to(DEVICE)
        inp["obs"] = obs.float().contiguous()
    return inp


def _kwargs(case, inp):
    kw = dict(nx=case["nx"], nz=case["nz"], dx=case["dx"], dz=case["dx"], nt=case["nt"], dt=case["dt"],
              nabc=case["nabc"], free_surface=case["free_surface"], src_n=case["shots"], src_v=inp["src_v"],
              rcv_n=len(inp["pos"]["rcv_x"]), damp=inp["damp"], vp=inp["vp"], rho=inp["rho"],
              device=torch.device(DEVICE), **inp["pos"])
    if case["ny"]:
        kw.update(ny=case["ny"], dy=case["dx"])
    return kw


def _propagator(case, inp, grad):
    grid = wave.GridConfig(nx=case["nx"], nz=case["nz"], dx=case["dx"], dz=case["dx"])
    bound = wave.BoundaryConfig(type="pml", n_layers=case["nabc"], free_surface=case["free_surface"])
    model = wave.AcousticModel(grid=grid, boundary=bound, vp=inp["vp"].cpu().numpy(), rho=inp["rho"].cpu().numpy(),
                               vp_grad=grad, device=DEVICE)
    src = wave.Source(nt=case["nt"], dt=case["dt"], f0=inp["f0"])
    w = inp["src_v"].cpu().numpy()
    for s, (x, z) in enumerate(zip(inp["pos"]["src_x"], inp["pos"]["src_z"])):
        src.add_source(x=int(x), z=int(z), wavelet=w[s])
    rcv = wave.Receiver(nt=case["nt"], dt=case["dt"])
    rcv.add_receivers(x=inp["pos"]["rcv_x"], z=inp["pos"]["rcv_z"], rcv_type="pr")
    return model, wave.AcousticPropagator(model, wave.Survey(src, rcv), device=DEVICE, fd_order=case["order"])


def prepare(case, seed):
    if case["kind"] == "batch":
        subs = _sub_cases(case)
        ins = [_inputs(c, seed * 1000 + i) for i, c in enumerate(subs)]
        return dict(case=case, obs=[i["obs"] for i in ins], models=[_kwargs(c, i) for c, i in zip(subs, ins)])
    inp = _inputs(case, seed)
    st = dict(case=case, obs=inp.get("obs"), vmax=inp["vmax"])
    if case["api"] == "propagator":
        st["model"], st["prop"] = _propagator(case, inp, case["kind"] == "gradient")
    else:
        st["kw"] = _kwargs(case, inp)
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
KEYS = ("p", "vx", "vz", "forward_wavefield_p", "forward_wavefield_vx", "forward_wavefield_vz")
KEYS3 = ("p", "vx", "vy", "vz", "forward_wavefield_p", "forward_wavefield_vx", "forward_wavefield_vy",
         "forward_wavefield_vz")


def _l2(p, obs):
    return 0.5 * (p - obs).square().sum()


def _options(case):
    o = dict(imaging_dtype=case["imaging"], snapshot_dtype=case["snapshots"], absorbing=case["absorbing"])
    if case["cache"] == "none":
        o["imaging_cache"] = 0
    return o


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forward":
        with torch.no_grad():
            if case["api"] == "propagator":
                res = state["prop"].forward()
                return {k: getattr(res, k) for k in KEYS}
            return wave.acoustic_forward_kernel(fd_order=case["order"], **state["kw"])
    if kind == "volume":
        with torch.no_grad():
            return wave.acoustic_forward_kernel_3d(**state["kw"])
    if kind == "batch":
        obs = state["obs"]

        def residual(i, p):
            r = p - obs[i]
            return 0.5 * r.square().sum(), r
        losses, grads = wave.acoustic_gradient_batched(state["models"], residual, fd_order=case["order"],
                                                       imaging_dtype=case["imaging"])
        return {"loss": losses, "vp": grads}
    misfit = wave.misfit.normalized_trace_l2 if case["misfit"] == "normalized" else _l2
    if case["api"] == "propagator":
        model = state["model"]
        model.vp.grad = None
        res = state["prop"].forward(**_options(case))
        loss = misfit(res.p, state["obs"])
        loss.backward()
        return {"loss": loss.detach(), "p": res.p.detach(), "vp": model.vp.grad}
    kw = dict(state["kw"])
    leaves = {"vp": kw["vp"].detach().requires_grad_(True)}
    if case["rho"]:
        leaves["rho"] = kw["rho"].detach().requires_grad_(True)
    if case["wavelet"]:
        leaves["src_v"] = kw["src_v"].detach().requires_grad_(True)
    kw.update(leaves)
    if kind == "volume_gradient":
        out = wave.acoustic_forward_kernel_3d(**kw)
    else:
        out = wave.acoustic_forward_kernel(fd_order=case["order"], **_options(case), **kw)
    loss = misfit(out["p"], state["obs"])
    loss.backward()
    return {"loss": loss.detach(), "p": out["p"].detach(), **{k: v.grad for k, v in leaves.items()}}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
ON_CHIP = 100e6                        # bytes of wavefield that can stay on the chip between steps


def _dims(case):
    n = case["nabc"]
    return [case["nz"] + 2 * n, case["nx"] + 2 * n] + ([case["ny"] + 2 * n] if case["ny"] else [])


def _state_bytes(case):
    return 4.0 * (len(_dims(case)) + 1) * math.prod(_dims(case)) * case["shots"]


def _work_one(case, streams):
    dims = _dims(case)
    cells = math.prod(dims)
    model = case["nz"] * case["nx"] * max(1, case["ny"])
    fields, half = len(dims) + 1, case["order"] // 2
    S, nt = case["shots"], case["nt"]
    units = S * cells * nt
    grad = "gradient" in case["kind"] or case["kind"] == "batch"
    passes = 2 if grad else 1
    bytes_ = 4.0 * (2 * model + cells + S * nt) + 4.0 * S * nt * case["receivers"] * fields
    if streams:                                            # the wavefield is read and written once a step
        bytes_ += passes * units * (8.0 * fields + 8.0 / S)
    if grad:                                               # imaging fields written and read
        e = {"fp32": 4, "fp24": 3, "bf16": 2}[case["imaging"]]
        bytes_ += 2.0 * e * units * ((1 + len(dims)) if case["rho"] else 1)
        bytes_ += 4.0 * (2 * S * nt * case["receivers"] + model * (2 if case["rho"] else 1))
    else:
        bytes_ += 4.0 * fields * model
    flops = units * (2.0 * len(dims) * (3 * half) + 3.0 * fields) * passes
    return bytes_, flops


def work(case):
    subs = _sub_cases(case) if case["kind"] == "batch" else [case]
    streams = sum(_state_bytes(c) for c in subs) > ON_CHIP
    got = [_work_one(c, streams) for c in subs]
    return {"bytes": sum(b for b, _ in got), "flops": sum(f for _, f in got)}


# ---------------------------------------------------------------------------
# the same in float64, in plain torch
# ---------------------------------------------------------------------------
def _cut(f, box, axis, by):
    """The part of f in `box` ((lo, hi) per axis, ends included), moved by `by` along `axis`."""
    sl = [slice(None)]
    for a, (lo, hi) in enumerate(box):
        d = by if a == axis else 0
        sl.append(slice(lo + d, hi + 1 + d))
    return f[tuple(sl)]


def _lay(g, box, shape):
    pads = []
    for (lo, hi), n in reversed(list(zip(box, shape))):
        pads += [lo, n - 1 - hi]
    return F.pad(g, pads)


class _Scheme:
    """Staggered velocity-pressure leapfrog, axes (z, x) or (z, y, x)."""

    def __init__(self, case, inp, vp, rho, vmax):
        n, dt, dz = case["nabc"], case["dt"], case["dx"]
        self.case, self.dt = case, dt
        R = self.R = case["order"] // 2
        self.taps = TAPS[case["order"]]
        three = case["ny"] > 0
        pad = lambda t: F.pad(t[None, None], (n,) * (6 if three else 4), mode="replicate")[0, 0]  # noqa: E731
        c, den = pad(vp), pad(rho)
        self.a1, self.a2 = den * c * c * dt / dz, dt / (den * dz)
        self.shape = sh = tuple(c.shape)
        D = len(sh)
        fs = self.fs = n if case["free_surface"] else 1
        if three:
            Nz, Ny, Nx = sh
            self.pbox = [(fs + 1, Nz - 3), (2, Ny - 3), (2, Nx - 3)]
            self.vbox = {2: [(fs, Nz - 2), (1, Ny - 2), (1, Nx - 3)], 1: [(fs, Nz - 2), (1, Ny - 3), (1, Nx - 2)],
                         0: [(fs, Nz - 3), (1, Ny - 2), (1, Nx - 2)]}
        else:
            Nz, Nx = sh
            self.pbox = [(max(fs + 1, R), Nz - 1 - R), (R, Nx - 1 - R)]
            self.vbox = {1: [(fs, Nz - 2), (R - 1, Nx - 1 - R)], 0: [(max(fs, R - 1), Nz - 1 - R), (1, Nx - 2)]}
        self.cpml = case["absorbing"] == "cpml"
        damp = inp["damp"].double()
        self.k1 = damp * dt
        self.kv = {}
        for a in range(D):
            k = torch.zeros_like(damp)
            lo, hi = (fs, sh[0] - 3) if a == 0 else (1, sh[a] - 3)
            m = hi - lo + 1
            k.narrow(a, lo, m).copy_(0.5 * (damp.narrow(a, lo, m) + damp.narrow(a, lo + 1, m)) * dt)
            self.kv[a] = k
        if self.cpml:
            self.prof = [self._profile(sh[a], n, dz, dt, vmax, not (a == 0 and case["free_surface"]), a) for a in range(D)]
        self.nabc, self.D = n, D
        p = inp["pos"]
        names = ("z", "y", "x") if three else ("z", "x")
        self.src = [torch.as_tensor(p["src_" + k] + n, device=DEVICE) for k in names]
        self.rcv = [torch.as_tensor(p["rcv_" + k] + n, device=DEVICE) for k in names]

    def _profile(self, N, n, dx, dt, vmax, low, axis):
        d0 = -3.0 * vmax * math.log(1e-6) / (2.0 * n * dx)

        def one(c):
            r = (n - c) / n if low and c < n else (c - (N - 1 - n)) / n if c > N - 1 - n else 0.0
            return math.exp(-d0 * min(r, 1.0) ** 2 * dt)
        view = [1] * 2
        view[axis] = -1
        return [torch.tensor([one(i + h) for i in range(N)], dtype=torch.float64, device=DEVICE).reshape(view)
                for h in (0.0, 0.5)]

    def start(self, S):
        z = torch.zeros((S,) + self.shape, dtype=torch.float64, device=DEVICE)
        return tuple(z for _ in range(1 + self.D + (2 * self.D if self.cpml else 0)))

    def step(self, st, w):
        """(p, v of each axis, and the memory variables) one step on; w: (S,) source samples."""
        D, sh = self.D, self.shape
        p, v, psi = st[0], list(st[1:1 + D]), list(st[1 + D:])
        b = self.pbox
        cutb = tuple(slice(lo, hi + 1) for lo, hi in b)
        parts = [sum(c * (_cut(v[a], b, a, k) - _cut(v[a], b, a, -1 - k)) for k, c in enumerate(self.taps))
                 for a in range(D)]
        if self.cpml:
            for a in range(D):
                at = tuple(cutb[a] if i == a else slice(None) for i in range(D))
                bb = self.prof[a][0][at]
                old = _cut(psi[a], b, 0, 0)
                new = bb * old + (bb - 1) * parts[a]
                psi[a] = psi[a] + _lay(new - old, b, sh)
                parts[a] = parts[a] + new
            p = p - _lay(self.a1[cutb] * sum(parts), b, sh)
        else:
            p = p - _lay(self.a1[cutb] * sum(parts) + self.k1[cutb] * _cut(p, b, 0, 0), b, sh)
        S = p.shape[0]
        at = (torch.arange(S, device=DEVICE), *self.src)
        p = p.index_put(at, self.dt * w, accumulate=True)
        fs = self.fs
        if self.case["free_surface"]:
            p = torch.cat([p[:, :fs - 1], -p[:, fs + 1:fs + 2], p[:, fs:]], 1)
        for a in range(D):
            b = self.vbox[a]
            cutb = tuple(slice(lo, hi + 1) for lo, hi in b)
            g = sum(c * (_cut(p, b, a, 1 + k) - _cut(p, b, a, -k)) for k, c in enumerate(self.taps))
            if self.cpml:
                sl = tuple(cutb[a] if i == a else slice(None) for i in range(D))
                bb = self.prof[a][1][sl]
                old = _cut(psi[D + a], b, 0, 0)
                new = bb * old + (bb - 1) * g
                psi[D + a] = psi[D + a] + _lay(new - old, b, sh)
                v[a] = v[a] - _lay(self.a2[cutb] * (g + new), b, sh)
            else:
                v[a] = v[a] - _lay(self.a2[cutb] * g + self.kv[a][cutb] * _cut(v[a], b, 0, 0), b, sh)
        if self.case["free_surface"]:
            v[0] = torch.cat([v[0][:, :fs - 1], v[0][:, fs:fs + 1], v[0][:, fs:]], 1)
        return (p, *v, *psi)

    def record(self, f):
        return f[(slice(None), *self.rcv)]


def _names(D):
    return ("p", "vx", "vz") if D == 2 else ("p", "vx", "vy", "vz")


def _fields(st, D):
    """p and the velocities in the order of _names."""
    return (st[0],) + tuple(st[1 + a] for a in range(D - 1, -1, -1))


def _exact_forward(case, inp):
    sc = _Scheme(case, inp, inp["vp"].double(), inp["rho"].double(), inp["vmax"])
    D, n = sc.D, case["nabc"]
    inner = (slice(None),) + tuple(slice(n, s - n) for s in sc.shape)
    w = inp["src_v"].double()
    st = sc.start(case["shots"])
    tr = [[] for _ in range(D + 1)]
    en = [0.0] * (D + 1)
    for it in range(case["nt"]):
        st = sc.step(st, w[:, it])
        for i, f in enumerate(_fields(st, D)):
            tr[i].append(sc.record(f))
            en[i] = en[i] + f[inner].square().sum(0)
    out = {k: torch.stack(t, 1) for k, t in zip(_names(D), tr)}
    out.update({"forward_wavefield_" + k: e for k, e in zip(_names(D), en)})
    return out


def _normalized(p, obs):
    m = lambda t: t / t.abs().amax(1, keepdim=True).clamp_min(1e-30)  # noqa: E731
    live = (obs.abs().sum(1) + p.abs().sum(1)) > 0
    sq = (m(obs) - m(p)).square().sum(1)
    return torch.where(sq > 0, torch.where(sq > 0, sq, 1.0).sqrt(), 0.0)[live].sum()


def _exact_gradient(case, inp, shots):
    """Loss, pressure traces and gradients of some of the shots."""
    vp = inp["vp"].double().requires_grad_(True)
    rho = inp["rho"].double().requires_grad_(case["rho"])
    w = inp["src_v"][shots].double().requires_grad_(case["wavelet"])
    pos = {k: (v[shots] if k.startswith("src") else v) for k, v in inp["pos"].items()}
    sc = _Scheme(case, dict(inp, pos=pos), vp, rho, inp["vmax"])
    nt = case["nt"]
    seg = max(1, int(math.sqrt(nt)) // (2 if sc.D == 3 else 1))

    def piece(a1, a2, ww, t0, t1, *st):
        sc.a1, sc.a2 = a1, a2
        got = []
        for it in range(t0, t1):
            st = sc.step(st, ww[:, it])
            got.append(sc.record(st[0]))
        return (torch.stack(got, 1), *st)

    a1, a2 = sc.a1, sc.a2
    st, tr = sc.start(w.shape[0]), []
    for t0 in range(0, nt, seg):
        got, *st = checkpoint(piece, a1, a2, w, t0, min(nt, t0 + seg), *st, use_reentrant=False)
        tr.append(got)
    p = torch.cat(tr, 1)
    obs = inp["obs"][shots].double()
    loss = (_normalized if case["misfit"] == "normalized" else _l2)(p, obs)
    loss.backward()
    return loss.detach(), p.detach(), vp.grad, rho.grad, w.grad


def _exact_one(case, inp):
    S = case["shots"]
    cells = (case["nz"] + 2 * case["nabc"]) * (case["nx"] + 2 * case["nabc"]) * (case["ny"] + 2 * case["nabc"] if case["ny"] else 1)
    at_once = max(1, int(6e6 // cells))
    parts = [_exact_gradient(case, inp, list(range(s, min(S, s + at_once)))) for s in range(0, S, at_once)]
    out = {"loss": sum(p[0] for p in parts), "p": torch.cat([p[1] for p in parts]), "vp": sum(p[2] for p in parts)}
    if case["rho"]:
        out["rho"] = sum(p[3] for p in parts)
    if case["wavelet"]:
        out["src_v"] = torch.cat([p[4] for p in parts])
    return out


def exact(case, seed):
    if case["kind"] == "batch":
        got = [_exact_one(c, _inputs(c, seed * 1000 + i)) for i, c in enumerate(_sub_cases(case))]
        return {"loss": torch.stack([g["loss"] for g in got]), "vp": [g["vp"] for g in got]}
    inp = _inputs(case, seed)
    if case["api"] == "propagator":      # the model's own density, from vp
        inp["rho"] = 310.0 * inp["vp"].double() ** 0.25
    if "gradient" in case["kind"]:
        return _exact_one(case, inp)
    with torch.no_grad():
        return _exact_forward(case, inp)
