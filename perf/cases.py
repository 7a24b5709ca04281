"""The work that is timed: what a user of this framework has it do, through `usx` and `usx.capi`.

A case is a dict of plain values; its `kind` names the path:

  das       one frame (or one Doppler sequence) of a beamforming plan: delay-and-sum, coherence factor, DMAS
  mv        one minimum-variance frame (the FP32 solver, the host API's default)
  learned   one learned-minimum-variance frame with the shipped network and its gates
  simulate  the point-scatterer simulator: scatterers to RF
  demod     RF to IQ
  flow      colour flow of one ensemble, or of several of uneven length in one call
  strain    axial displacement between two frames, then strain
  display   envelope, time-gain compensation, log compression, scan conversion
  pipeline  usx.ImagingPipeline.process_frame on a host acquisition (RF in host memory, frame back)
  train     one training step of the learned-MV network (forward, backward, Adam)

Sizes are those of the configurations in tests/configs.py, of bench.py and of the test fixtures;
`draw` spreads over the same ranges.

Acquisitions are made from a seeded speckle phantom: every scatterer leaves an impulse of its own
delay, phase and spreading loss in each trace (summed as 64-bit integers, so that the order does not
matter), the traces are convolved with the probe's pulse, and receive noise is added.
"""

from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "ultrasound-engine_gb300" / "python"))

import usx  # noqa: E402
from usx import capi  # noqa: E402
from usx import learned as usx_learned  # noqa: E402

C0 = 1540.0
PLANE, DIVERGING, FOCUSED = 1, 2, 0
DAS, DMAS, MV, LEARNED = 0, 1, 2, 3
RECT, HANN, TUKEY = 0, 1, 3

# The probes of tests/configs.py and of the golden fixtures (elements, pitch, element width, f0).
PROBES = {"linear128": (128, 300e-6, 270e-6, 5e6),
          "phased64": (64, 200e-6, 180e-6, 2.5e6),
          "linear32": (32, 300e-6, 270e-6, 5e6)}
BANDWIDTH = 0.6


def listed():
    return [
        # A look at a small region with a short aperture: launch and call latency.
        dict(name="das_small", kind="das", probe="linear32", tx="plane", n_tx=3, span=9.0, z0=6.0, z1=22.0,
             n0=16, n1=40, f_number=1.5, window=HANN, combiner=DAS, cf=False, frames=1, tuned=False),
        # Phased-array cardiac view: 31 diverging waves, DMAS.
        dict(name="das_sector", kind="das", probe="phased64", tx="diverging", n_tx=31, span=45.0, z0=5.0, z1=80.0,
             n0=256, n1=1024, f_number=1.75, window=HANN, combiner=DMAS, cf=False, frames=1, tuned=False),
        # The headline frame: 75 plane waves onto 512 x 1024, the plan autotuned as a scanner's would be.
        dict(name="das_frame", kind="das", probe="linear128", tx="plane", n_tx=75, span=16.0, z0=5.0, z1=60.0,
             n0=512, n1=1024, f_number=1.5, window=HANN, combiner=DAS, cf=False, frames=1, tuned=True),
        # The same frame by minimum variance, subarrays up to 64.
        dict(name="mv_frame", kind="mv", probe="linear128", tx="plane", n_tx=75, span=16.0, z0=5.0, z1=60.0,
             n0=512, n1=1024, f_number=1.5, subarray=64, range_avg=2, tuned=True),
        # And by the learned minimum variance (the benchmark's default workload).
        dict(name="learned_frame", kind="learned", probe="linear128", tx="plane", n_tx=75, span=16.0, z0=5.0, z1=60.0,
             n0=512, n1=1024, f_number=1.5, tuned=True),
        # One simulated acquisition of the 100,000-scatterer phantom.
        dict(name="simulate_phantom", kind="simulate", probe="linear128", tx="plane", n_tx=75, span=16.0, z1=60.0,
             scatterers=100_000, noise=True),
        # Demodulation of the headline acquisition.
        dict(name="demod_acquisition", kind="demod", probe="linear128", n_tx=75, z1=60.0, taps=33, decimation=1),
        # A Doppler cine loop: eight ensembles of 8 to 32 pulses, quadratic wall filter, Loupas.
        dict(name="flow_batch", kind="flow", n_ens=8, pulses=32, n0=256, n1=512, order=2, loupas=True, ka=4, kl=1),
        # Elastography: tracking with lags of +/- 8 samples, 2 mm strain fit.
        dict(name="strain_map", kind="strain", n0=256, n1=1024, ka=8, kl=2, max_lag=8, fit=57),
        # The display chain of one B-mode frame.
        dict(name="display_bmode", kind="display", n0=512, n1=1024, width=512, height=800, sector=False),
        # What a caller of the host API does per frame: 11 plane waves, RF in host memory.
        dict(name="pipeline_11pw", kind="pipeline", probe="linear128", n_tx=11, span=9.0, z0=5.0, z1=50.0,
             n0=256, n1=640, f_number=1.75, cf=False),
        # One minibatch of the network's training.
        dict(name="train_step", kind="train", rows=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["das", "das", "das", "mv", "learned", "simulate", "demod", "flow", "strain", "display",
                       "pipeline", "train"])
    if kind == "das":
        probe = rng.choice(["linear128", "linear128", "phased64", "linear32"])
        tx = "diverging" if probe == "phased64" else rng.choice(["plane", "plane", "focused"])
        frames = rng.choice([1, 1, 1, _log_int(rng, 2, 16)])
        n_tx = _log_int(rng, 1, 75) if frames == 1 else rng.choice([1, 3])
        n0, n1 = _log_int(rng, 16, 512), _log_int(rng, 32, 1024)
        work = n0 * n1 * n_tx * frames * PROBES[probe][0]
        comb, cf = rng.choice([(DAS, False), (DAS, False), (DAS, True), (DMAS, False)])
        return dict(kind="das", probe=probe, tx=tx, n_tx=n_tx, span=rng.choice([5.0, 9.0, 16.0]) if tx != "diverging"
                    else 45.0, z0=rng.choice([5.0, 6.0, 10.0]), z1=rng.choice([22.0, 35.0, 50.0, 60.0]), n0=n0, n1=n1,
                    f_number=rng.choice([1.0, 1.5, 1.75]), window=rng.choice([RECT, HANN, TUKEY]), combiner=comb,
                    cf=cf, frames=frames, tuned=work >= 1e9 and frames == 1)
    if kind in ("mv", "learned"):
        probe = "linear128" if kind == "learned" else rng.choice(["linear128", "phased64"])
        c = dict(kind=kind, probe=probe, tx="plane", n_tx=_log_int(rng, 1, 16), span=9.0, z0=5.0,
                 z1=rng.choice([35.0, 50.0, 60.0]), n0=_log_int(rng, 16, 256), n1=_log_int(rng, 100, 1024),
                 f_number=rng.choice([1.5, 1.75]), tuned=False)
        if kind == "mv":
            c.update(subarray=rng.choice([16, 24, 32, 48, 64]), range_avg=rng.choice([1, 2, 2]))
        return c
    if kind == "simulate":
        probe = rng.choice(["linear128", "phased64"])
        return dict(kind="simulate", probe=probe, tx="plane" if probe == "linear128" else "diverging",
                    n_tx=_log_int(rng, 1, 12), span=9.0 if probe == "linear128" else 45.0,
                    z1=rng.choice([40.0, 50.0, 60.0]), scatterers=_log_int(rng, 500, 20_000),
                    noise=rng.random() < 0.5)
    if kind == "demod":
        taps, dec = rng.choice([(33, 1), (33, 1), (21, 1), (21, 2), (33, 4), (47, 1)])
        return dict(kind="demod", probe=rng.choice(["linear128", "phased64", "linear32"]), n_tx=_log_int(rng, 1, 75),
                    z1=rng.choice([20.0, 40.0, 60.0]), taps=taps, decimation=dec)
    if kind == "flow":
        n_ens = rng.choice([1, 1, 2, 5])
        return dict(kind="flow", n_ens=n_ens, pulses=_log_int(rng, 6, 32), n0=_log_int(rng, 12, 256),
                    n1=_log_int(rng, 30, 512), order=rng.choice([0, 1, 2]), loupas=rng.random() < 0.8,
                    ka=rng.choice([2, 4, 6]), kl=rng.choice([0, 1, 2]))
    if kind == "strain":
        return dict(kind="strain", n0=_log_int(rng, 12, 256), n1=_log_int(rng, 64, 1024), ka=rng.choice([4, 8, 12]),
                    kl=rng.choice([0, 1, 2]), max_lag=rng.choice([4, 8, 12]), fit=rng.choice([9, 31, 57]))
    if kind == "display":
        return dict(kind="display", n0=_log_int(rng, 16, 512), n1=_log_int(rng, 64, 1024),
                    width=_log_int(rng, 50, 800), height=_log_int(rng, 50, 800), sector=rng.random() < 0.5)
    if kind == "pipeline":
        return dict(kind="pipeline", probe=rng.choice(["linear128", "linear32"]), n_tx=_log_int(rng, 1, 11), span=9.0,
                    z0=5.0, z1=rng.choice([35.0, 50.0]), n0=_log_int(rng, 32, 256), n1=_log_int(rng, 64, 640),
                    f_number=1.75, cf=rng.random() < 0.3)
    return dict(kind="train", rows=128 * _log_int(rng, 4, 64))


# ------------------------------------------------------------------ geometry, in plain numpy

def _f32(v):
    """A number as the float32 that the descriptors carry, in 64 bits."""
    return float(np.float32(v))


class Setup:
    """Probe, transmits, grid and acquisition of a case, with the float32 values the calls receive."""

    def __init__(self, case):
        self.n_el, pitch, width, f0 = PROBES[case["probe"]]
        self.pitch, self.width, self.f0, self.c = _f32(pitch), _f32(width), _f32(f0), _f32(C0)
        self.fs = _f32(4.0 * f0)
        depth = case["z1"] * 1e-3
        aperture = (self.n_el - 1) * pitch + width
        self.n_smp = int(math.ceil((2.0 * depth / C0 + aperture / C0 + 4.0 / f0) * self.fs))
        self.prf = _f32(0.95 * C0 / (2.0 * depth))
        self.half_aperture = 0.5 * aperture
        ex = (np.arange(self.n_el, dtype=np.float32) - np.float32(0.5 * (self.n_el - 1))) * np.float32(pitch)
        self.ex = ex.astype(np.float32)
        self.frames = case.get("frames", 1)
        self.tx = [t for _ in range(self.frames) for t in self._transmits(case)]

    def _transmits(self, case):
        kind, n, span = case.get("tx", "plane"), case["n_tx"], math.radians(case.get("span", 0.0))
        out = []
        for k in range(n):
            s = 0.0 if n == 1 else -1.0 + 2.0 * k / (n - 1)
            x = self.ex.astype(np.float64)
            half, origin, focus, angle = self.half_aperture, 0.0, (0.0, 0.0, 0.03), 0.0
            if kind == "plane":
                angle = _f32(s * span)
                delay = x * math.sin(angle) / self.c
            elif kind == "diverging":  # virtual source 10 mm behind the array
                angle = _f32(s * span)
                focus = (_f32(-0.01 * math.sin(angle)), 0.0, _f32(-0.01 * math.cos(angle)))
                delay = (np.hypot(x - focus[0], focus[2]) - math.hypot(focus[0], focus[2])) / self.c
            else:  # beams across the aperture, focused at 20 mm, F/2
                origin = _f32(0.6 * s * self.half_aperture)
                focus = (origin, 0.0, _f32(0.02))
                half = min(half, 0.5 * 0.02 / 2.0)
                delay = (0.02 - np.hypot(x - origin, 0.02)) / self.c
            u = (x - origin) / half
            apod = np.where(np.abs(u) < 1, 0.5 * (1 + np.cos(np.pi * u)), 0.0)
            out.append(dict(type={"plane": PLANE, "diverging": DIVERGING, "focused": FOCUSED}[kind], angle=angle,
                            focus=focus, origin=(origin, 0.0, 0.0),
                            delays=np.where(apod > 0, delay, 0).astype(np.float32), apodization=apod.astype(np.float32)))
        return out

    def channel(self, is_iq):
        return capi.Channel(capi.Probe(self.n_el, self.pitch, self.width, 5e-3, self.f0, BANDWIDTH),
                            capi.Medium(self.c, 0.5, 1000.0), capi.Acquisition(self.fs, self.n_smp, 0.0, self.prf),
                            self.tx, is_iq, self.f0 if is_iq else 0.0)


def _grid(case):
    """(axis0, axis1, points): a Cartesian grid over the aperture, a sector for the phased array."""
    n0, n1 = case["n0"], case["n1"]
    z = np.linspace(case["z0"] * 1e-3, case["z1"] * 1e-3, n1).astype(np.float32)
    if case["probe"] == "phased64" and case.get("tx") == "diverging":
        th = np.linspace(-math.pi / 4, math.pi / 4, n0).astype(np.float32)
        x = z[None, :] * np.sin(th)[:, None]
        zz = z[None, :] * np.cos(th)[:, None]
        a0, gtype = th, 1
    else:
        n_el, pitch, width, _ = PROBES[case["probe"]]
        half = 0.5 * ((n_el - 1) * pitch + width)
        a0, gtype = np.linspace(-half, half, n0).astype(np.float32), 0
        x, zz = np.repeat(a0[:, None], n1, 1), np.repeat(z[None, :], n0, 0)
    pts = np.stack([x, np.zeros_like(x), zz], -1).astype(np.float32).reshape(-1, 3)
    return gtype, a0, z, pts


def _arrival(t, px, pz, c):
    """Ideal transmit arrival time at points."""
    if t["type"] == PLANE:
        return ((px - t["origin"][0]) * math.sin(t["angle"]) + pz * math.cos(t["angle"])) / c
    fx, fz, ox = t["focus"][0], t["focus"][2], t["origin"][0]
    if t["type"] == DIVERGING:
        return (torch.hypot(px - fx, pz - fz) - math.hypot(ox - fx, fz)) / c
    length = math.hypot(fx - ox, fz)
    proj = ((px - fx) * (fx - ox) + (pz - fz) * fz) / length
    return (length + torch.where(proj >= 0, 1.0, -1.0) * torch.hypot(px - fx, pz - fz)) / c


# ------------------------------------------------------------------ inputs

def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + salt)


def _phantom(s, case, seed, n):
    """Seeded speckle over the field of view, with an anechoic disc and bright points: x, z, amplitude."""
    g = _gen(seed, 1)
    u = torch.rand((2, n), device="cuda", generator=g)
    amp = torch.randn(n, device="cuda", generator=g)
    z0, z1 = 4e-3, case["z1"] * 1e-3 * 1.03
    half = s.half_aperture * 1.1 if case["probe"] != "phased64" else 0.7 * z1
    x, z = (2 * u[0] - 1) * half, z0 + u[1] * (z1 - z0)
    amp[(x.square() + (z - 0.5 * z1).square()) < 0.003 ** 2] = 0
    bright = torch.arange(min(8, n), device="cuda")
    amp[bright] = 20.0
    return x, z, amp


def _echoes(case, s, seed, rf):
    """[event][channel][sample] IQ of the phantom (complex64), or the RF that carries it (float32)."""
    x, z, amp = _phantom(s, case, seed, 20_000 if case["n_tx"] * s.frames > 1 else 8_000)
    ex = torch.from_numpy(s.ex).cuda()
    r = torch.hypot(x[:, None] - ex[None], z[:, None])
    rx, gain = r / s.c, (amp / (200.0 * z.clamp_min(4e-3)))[:, None] * (0.01 / r) * 2.0 ** 24
    n_ev, n = len(s.tx), s.n_smp
    acc = torch.zeros((n_ev, 2, s.n_el * n), dtype=torch.int64, device="cuda")
    col = torch.arange(s.n_el, device="cuda")[None] * n
    for e, t in enumerate(s.tx):
        tau = _arrival(t, x, z, s.c)[:, None] + rx
        if s.frames > 1:  # a slow drift between the frames of a sequence
            tau = tau + 1.5e-9 * (e // (n_ev // s.frames))
        k = torch.round(tau * s.fs).long()
        ok = (k >= 0) & (k < n)
        idx = (col + k.clamp(0, n - 1))[ok]
        ph = (-2 * math.pi * s.f0) * tau
        for part, f in enumerate((torch.cos, torch.sin)):
            acc[e, part].index_add_(0, idx, (gain * f(ph)).round().long()[ok])
    sig = math.sqrt(2 * math.log(2)) / (math.pi * BANDWIDTH * s.f0) * s.fs
    taps = [math.exp(-0.5 * (j / sig) ** 2) for j in range(-8, 9)]
    g = _gen(seed, 2)
    out = torch.empty((n_ev, s.n_el, n), dtype=torch.float32 if rf else torch.complex64, device="cuda")
    for e in range(n_ev):
        v = acc[e].view(2, s.n_el, n).float() * 2.0 ** -24
        p = torch.nn.functional.pad(v, (8, 8))
        y = sum(h * p[..., j:j + n] for j, h in enumerate(taps))
        y = y + 1e-3 * torch.randn(y.shape, device="cuda", generator=g)
        if rf:
            w = 2 * math.pi * s.f0 / s.fs * torch.arange(n, device="cuda", dtype=torch.float64)
            out[e] = (y[0] * torch.cos(w).float() - y[1] * torch.sin(w).float())
        else:
            out[e] = torch.complex(y[0], y[1])
    return out


def _speckle(n0, n1, g, axial=4.0):
    """Complex speckle envelope [n0][n1], correlated over a few samples."""
    v = torch.randn((2, n0 + 2, n1 + 16), device="cuda", generator=g)
    taps = [math.exp(-0.5 * ((j - 8) / axial) ** 2) for j in range(17)]
    v = sum(h * v[..., j:j + n1] for j, h in enumerate(taps))
    v = 0.5 * v[:, :-2] + v[:, 1:-1] + 0.5 * v[:, 2:]
    return torch.complex(v[0], v[1])


def _flow_lengths(case):
    full = case["pulses"]
    return [full] if case["n_ens"] == 1 else [max(4, full * q // 32) for k in range(case["n_ens"])
                                              for q in ((8, 12, 16, 32)[k % 4],)]


def _flow_axis(case):
    return np.linspace(0.010, 0.010 + 49e-6 * (case["n1"] - 1), case["n1"]).astype(np.float32)


def _flow_input(case, seed):
    """Ensembles [frame][n0][n1]: drifting tissue, a vessel with a parabolic profile, noise."""
    g = _gen(seed, 3)
    n0, n1 = case["n0"], case["n1"]
    k = 4 * math.pi * 5e6 / C0 * 49e-6 * torch.arange(n1, device="cuda")
    carrier = torch.polar(torch.ones_like(k), k)
    d = (torch.arange(n1, device="cuda")[None] - (0.3 * n1 + 0.4 * n1 * torch.arange(n0, device="cuda")[:, None] / n0))
    prof = (1 - (d / (0.12 * n1)).square()).clamp_min(0)
    frames = []
    for n in _flow_lengths(case):
        tissue, blood = 10 * _speckle(n0, n1, g) * carrier, _speckle(n0, n1, g) * carrier * (prof > 0)
        for e in range(n):
            one = torch.ones_like(prof)
            f = tissue * torch.polar(one, 0.02 * e * one) + blood * torch.polar(one, 1.4 * e * prof)
            noise = torch.randn((2, n0, n1), device="cuda", generator=g)
            frames.append(f + 0.1 * torch.complex(noise[0], noise[1]))
    return torch.stack(frames).to(torch.complex64).contiguous()


def _strain_axis(case):
    return np.linspace(0.012, 0.012 + 35.2e-6 * (case["n1"] - 1), case["n1"]).astype(np.float32)


def _strain_input(case, seed):
    """A frame before and after a compression of about 0.5%, stiffer at the centre."""
    g = _gen(seed, 4)
    n0, n1 = case["n0"], case["n1"]
    env = _speckle(n0, n1 + 32, g, 6.0)
    j = torch.arange(n1, device="cuda", dtype=torch.float32)
    soft = torch.full((n0, n1), 0.005, device="cuda")
    lat = torch.arange(n0, device="cuda")[:, None] / n0 - 0.5
    soft[(lat.square() + ((j[None] / n1) - 0.5).square()) < 0.02] = 0.00125
    u = torch.cumsum(soft, 1)
    u = u / u.max().clamp_min(1.0) * min(5.0, float(u.max()))
    k = 4 * math.pi * 5e6 / C0 * 35.2e-6
    pos = (j[None] - u).clamp_min(0) + 8
    i = pos.floor().long()
    f = pos - i
    after = env.gather(1, i) * (1 - f) + env.gather(1, i + 1) * f
    before = env[:, 8:8 + n1] * torch.polar(torch.ones_like(j), k * j)
    after = after * torch.polar(torch.ones_like(pos), k * (j[None] - u))
    n = torch.randn((4, n0, n1), device="cuda", generator=g) * 0.05
    return (before + torch.complex(n[0], n[1])).contiguous(), (after + torch.complex(n[2], n[3])).contiguous()


def _display_grid(case):
    n0, n1 = case["n0"], case["n1"]
    if case["sector"]:
        return _grid(dict(probe="phased64", tx="diverging", n0=n0, n1=n1, z0=5.0, z1=80.0))
    return _grid(dict(probe="linear128", n0=n0, n1=n1, z0=5.0, z1=45.0))


def _display_input(case, seed):
    g = _gen(seed, 5)
    n1 = case["n1"]
    return (_speckle(case["n0"], n1, g) * torch.exp(-torch.linspace(0, 4, n1, device="cuda"))).contiguous()


TRAIN_DIMS = (256, 256, 256, 256, 128)


def _train_input(case, seed):
    """(parameters, x, target): He-uniform weights, features in the network's range, unit targets."""
    g = _gen(seed, 6)
    rng = np.random.default_rng(int(seed) + 17)
    p = [q for a, b in zip(TRAIN_DIMS[:-1], TRAIN_DIMS[1:])
         for q in (rng.uniform(-1, 1, a * b) * math.sqrt(6.0 / a), rng.normal(0, 0.01, b))]
    x = torch.randn((case["rows"], TRAIN_DIMS[0]), device="cuda", generator=g) * 0.7
    t = torch.randn((case["rows"], TRAIN_DIMS[-1]), device="cuda", generator=g)
    return np.concatenate(p).astype(np.float32), x, t


# ------------------------------------------------------------------ what the program has in hand

@functools.lru_cache(maxsize=None)
def _context():
    """One context per device, on torch's stream."""
    return capi.Context(0, stream=torch.cuda.current_stream().cuda_stream)


@functools.lru_cache(maxsize=None)
def _network():
    return usx_learned.load_mlp(_context())


def _bf_config(case):
    kw = dict(f_number=case["f_number"], rx_window=case.get("window", HANN))
    if case["kind"] == "das":
        kw.update(combiner=case["combiner"], coherence_factor=int(case["cf"]))
    elif case["kind"] == "mv":
        kw.update(combiner=MV, mv_subarray=case["subarray"], mv_diagonal_loading=0.01,
                  mv_range_average=case["range_avg"])
    else:
        kw.update(combiner=LEARNED, mv_subarray=64, mv_diagonal_loading=0.01, mv_range_average=2)
    return capi.bf_config(**kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pipeline":
        return _prepare_pipeline(case, seed)
    ctx = _context()
    st = dict(case=case, ctx=ctx)
    if kind in ("das", "mv", "learned"):
        s = Setup(case)
        gtype, a0, a1, pts = _grid(case)
        st["iq"] = _echoes(case, s, seed, rf=False)
        plan = ctx.plan(s.channel(True), capi.Grid(gtype, a0, a1, pts), _bf_config(case))
        if kind == "mv":
            plan.set_mv_mode(3)
        if kind == "learned":
            w = usx_learned.DEFAULT_WEIGHTS
            plan.set_learned(_network(), usx_learned.trained_gate(w))
            plan.set_learned_refine(usx_learned.trained_refine(w))
            plan.set_learned_subspace(True, usx_learned.trained_share_gate(w))
            plan.set_learned_level_gate(usx_learned.trained_level_gate(w))
            plan.set_learned_level_window(*usx_learned.trained_level_window(w))
            plan.set_mv_mode(3)
        st["plan"] = plan
        st["out"] = torch.empty((s.frames, len(a0), len(a1)), dtype=torch.complex64, device="cuda")
        if case["tuned"]:
            plan.autotune(st["iq"].data_ptr(), st["out"].data_ptr(), repeats=1)
    elif kind == "simulate":
        s = Setup(case)
        st["channel"] = s.channel(False)
        x, z, amp = _phantom(s, case, seed, case["scatterers"])
        st["scat"] = torch.zeros((len(x), 8), device="cuda")
        st["scat"][:, 0], st["scat"][:, 2], st["scat"][:, 3] = x, z, amp
        st["out"] = torch.empty((len(s.tx), s.n_el, s.n_smp), device="cuda")
        st["noise"] = torch.randn(st["out"].shape, device="cuda", generator=_gen(seed, 7)) if case["noise"] else None
        st["cfg"] = capi.sim_config(noise_db=-60.0 if case["noise"] else -200.0)
    elif kind == "demod":
        s = Setup(case)
        st["channel"], st["rf"] = s.channel(False), _echoes(case, s, seed, rf=True)
        st["cfg"] = capi.demod_config(filter_taps=case["taps"], decimation=case["decimation"])
        n_out = -(-s.n_smp // case["decimation"])
        st["out"] = torch.empty((len(s.tx), s.n_el, n_out), dtype=torch.complex64, device="cuda")
    elif kind == "flow":
        st["ens"], st["axis"] = _flow_input(case, seed), _flow_axis(case)
        st["lengths"] = np.array(_flow_lengths(case), np.int32)
        st["offsets"] = np.concatenate([[0], np.cumsum(st["lengths"])[:-1]]).astype(np.int64)
        shape = (case["n_ens"], case["n0"], case["n1"])
        st["cfg"] = capi.doppler_config(polynomial_order=case["order"], loupas=int(case["loupas"]),
                                        kernel_axial=case["ka"], kernel_lateral=case["kl"])
        for k in ("velocity", "power", "variance"):
            st[k] = torch.empty(shape, device="cuda")
        st["valid"] = torch.empty(shape, dtype=torch.uint8, device="cuda")
    elif kind == "strain":
        st["before"], st["after"] = _strain_input(case, seed)
        st["axis"] = _strain_axis(case)
        for k in ("axial", "correlation", "strain"):
            st[k] = torch.empty((case["n0"], case["n1"]), device="cuda")
    elif kind == "display":
        gtype, a0, a1, pts = _display_grid(case)
        st["frame"], st["grid"] = _display_input(case, seed), capi.Grid(gtype, a0, a1, pts)
        st["points"] = torch.from_numpy(pts).cuda()
        for k in ("env", "tgc", "log"):
            st[k] = torch.empty((case["n0"], case["n1"]), device="cuda")
        st["out"] = torch.empty((case["height"], case["width"]), device="cuda")
    else:
        p, st["x"], st["target"] = _train_input(case, seed)
        st["net"] = capi.Mlp(ctx, TRAIN_DIMS)
        st["net"].set_params(p)
    return st


def _prepare_pipeline(case, seed):
    """Host RF as a data-acquisition card leaves it, and the pipeline of its geometry."""
    s = Setup(case)
    rf = _echoes(case, s, seed, rf=True).cpu().numpy()
    probe = usx.Probe()
    probe.n_elements, probe.pitch, probe.element_width = s.n_el, s.pitch, s.width
    probe.center_frequency, probe.bandwidth = s.f0, BANDWIDTH
    acq = usx.Acquisition()
    acq.sampling_frequency, acq.n_samples, acq.prf, acq.t0 = s.fs, s.n_smp, s.prf, 0.0
    txs = []
    for t in s.tx:
        x = usx.Transmit()
        x.type, x.angle = usx.TransmitType.PLANE_WAVE, t["angle"]
        x.delays, x.apodization = t["delays"], t["apodization"]
        txs.append(x)
    half = 0.5 * probe.aperture_width()
    grid = usx.ScanGrid.cartesian(-half, half, case["n0"], case["z0"] * 1e-3, case["z1"] * 1e-3, case["n1"])
    cfg = usx.PipelineConfig()
    b = usx.BeamformerConfig()
    b.f_number, b.coherence_factor = case["f_number"], case["cf"]
    cfg.beamformer = b
    raw = usx.ChannelData.from_rf(rf, probe, usx.Medium(), acq, txs)
    return dict(case=case, pipeline=usx.ImagingPipeline(grid, cfg), raw=raw)


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "pipeline":
        return np.asarray(st["pipeline"].process_frame(st["raw"]).data)
    ctx = st["ctx"]
    if kind in ("das", "mv", "learned"):
        iq, out = st["iq"], st["out"]
        if out.shape[0] > 1:
            st["plan"].execute_sequence(case["n_tx"], out.shape[0], iq.data_ptr(), out.data_ptr(), out[0].numel())
        else:
            st["plan"].execute(iq.data_ptr(), out.data_ptr())
        return out
    if kind == "simulate":
        noise = st["noise"]
        ctx.simulate(st["channel"], st["cfg"], st["scat"].data_ptr(), st["scat"].shape[0],
                     None if noise is None else noise.data_ptr(), st["out"].data_ptr())
        return st["out"]
    if kind == "demod":
        ctx.demodulate(st["channel"], st["cfg"], st["rf"].data_ptr(), st["out"].data_ptr())
        return st["out"]
    if kind == "flow":
        maps = [st[k] for k in ("velocity", "power", "variance", "valid")]
        ptrs = [m.data_ptr() for m in maps]
        if case["n_ens"] == 1:
            ctx.color_flow(st["ens"].data_ptr(), int(st["lengths"][0]), case["n0"], case["n1"], st["axis"], 5e6, 5e3,
                           C0, st["cfg"], *ptrs)
        else:
            ctx.color_flow_batch(st["ens"].data_ptr(), st["lengths"], st["offsets"], case["n0"], case["n1"],
                                 st["axis"], 5e6, 5e3, C0, st["cfg"], *ptrs)
        return maps
    if kind == "strain":
        n0, n1 = case["n0"], case["n1"]
        ctx.axial_displacement(st["before"].data_ptr(), st["after"].data_ptr(), n0, n1, st["axis"], 5e6, C0,
                               case["ka"], case["kl"], case["max_lag"], st["axial"].data_ptr(),
                               st["correlation"].data_ptr())
        ctx.axial_strain(st["axial"].data_ptr(), n0, n1, st["axis"], case["fit"], st["strain"].data_ptr())
        return [st["axial"], st["correlation"], st["strain"]]
    if kind == "display":
        n0, n1 = case["n0"], case["n1"]
        ctx.envelope(st["frame"].data_ptr(), n0, n1, 5e6, st["env"].data_ptr())
        ctx.apply_tgc(st["env"].data_ptr(), n0, n1, st["points"].data_ptr(), 0.5, 5e6, st["tgc"].data_ptr())
        ctx.log_compress(st["tgc"].data_ptr(), n0 * n1, 60.0, 0.0, 0.0, st["log"].data_ptr())
        ctx.scan_convert(st["log"].data_ptr(), st["grid"], case["width"], case["height"], 0.0, st["out"].data_ptr())
        return [st["env"], st["tgc"], st["log"], st["out"]]
    loss, grad = st["net"].train_step(st["x"].data_ptr(), st["target"].data_ptr(), None, case["rows"], 1e-3,
                                      want_loss=True, want_grad=True)
    return [loss, grad]


# ------------------------------------------------------------------ the work that cannot be avoided

def _active(case):
    """Active channels per pixel (the receive aperture |x_e - x| <= z / (2 F#))."""
    n_el, pitch, _, _ = PROBES[case["probe"]]
    pts = _grid(case)[3].astype(np.float64)
    half = 0.5 * pts[:, 2] / case["f_number"]
    mid = 0.5 * (n_el - 1)
    lo = np.maximum(0, np.ceil(mid + (pts[:, 0] - half) / pitch))
    hi = np.minimum(n_el - 1, np.floor(mid + (pts[:, 0] + half) / pitch))
    return np.maximum(0, hi - lo + 1)


def work(case):
    kind = case["kind"]
    if kind in ("das", "mv", "learned", "pipeline"):
        s = Setup(case)
        act, n_pix, n_ev = _active(case), case["n0"] * case["n1"], len(s.tx)
        data = n_ev * s.n_el * s.n_smp * (4 if kind == "pipeline" else 8)
        byt = data + 20.0 * n_pix * s.frames
        flops = 20.0 * float(act.sum()) * n_ev  # a complex interpolation, rotation and sum
        if kind == "pipeline":
            flops += 4.0 * 33 * n_ev * s.n_el * s.n_smp
        if kind == "mv":
            L = np.clip(np.minimum(case["subarray"], act // 2), 2, None)
            K = (2 * case["range_avg"] + 1) * (act - L + 1)
            flops += float((4 * L ** 2 * K + 4 / 3 * L ** 3 + 16 * L ** 2)[act >= 4].sum())
        if kind == "learned":
            L = np.clip(np.minimum(64, act // 2), 2, None)
            flops += float((8 * 5 * (act - L + 1) * (L + 36) + 8 * 5 * act * 7)[act >= 4].sum())
            flops += 2.0 * n_pix * sum(a * b for a, b in zip(TRAIN_DIMS[:-1], TRAIN_DIMS[1:]))
        return dict(bytes=byt, flops=flops)
    if kind == "simulate":
        s = Setup(case)
        rf = len(s.tx) * s.n_el * s.n_smp
        pairs = float(case["scatterers"]) * len(s.tx) * s.n_el
        # Per (scatterer, event, element): the incident pulse's taps and about 60 echo samples.
        return dict(bytes=32.0 * case["scatterers"] + 4.0 * rf * (2 if case["noise"] else 1), flops=pairs * (4 * 61 + 4 * 60))
    if kind == "demod":
        s = Setup(case)
        n, m = len(s.tx) * s.n_el * s.n_smp, len(s.tx) * s.n_el * (-(-s.n_smp // case["decimation"]))
        return dict(bytes=4.0 * n + 8.0 * m, flops=2.0 * n + 4.0 * case["taps"] * m)
    n_pix = case.get("n0", 0) * case.get("n1", 0)
    if kind == "flow":
        lens = _flow_lengths(case)
        return dict(bytes=n_pix * (8.0 * sum(lens) + 13.0 * len(lens)),
                    flops=float(n_pix) * sum(4.0 * n * n + 30.0 * n for n in lens))
    if kind == "strain":
        return dict(bytes=n_pix * 28.0, flops=float(n_pix) * (2 * case["max_lag"] + 1) * 24.0)
    if kind == "display":
        return dict(bytes=n_pix * (8.0 + 12.0 + 12.0) + 4.0 * case["width"] * case["height"], flops=60.0 * n_pix)
    n_par = sum(a * b + b for a, b in zip(TRAIN_DIMS[:-1], TRAIN_DIMS[1:]))
    return dict(bytes=4.0 * case["rows"] * (256 + 128) + 24.0 * n_par, flops=6.0 * case["rows"] * n_par)


# ------------------------------------------------------------------ the same in 64 bits

def exact(case, seed):
    kind = case["kind"]
    if kind in ("das", "pipeline"):
        s = Setup(case)
        if kind == "das":
            data, pts, cfg = _echoes(case, s, seed, rf=False), _grid(case)[3], case
        else:
            rf = _echoes(case, s, seed, rf=True)
            data, pts = _exact_demod(rf, s, 33, 1), _grid(dict(case, tx="plane"))[3]
            cfg = dict(case, window=HANN, combiner=DAS)
        return _exact_das(cfg, s, data, pts)
    if kind in ("mv", "learned"):
        return _exact_capon(case, seed)
    if kind == "simulate":
        # 10^11 echo samples in 64 bits take minutes; the smaller acquisitions a few seconds.
        if case["scatterers"] * case["n_tx"] > 300_000:
            return None
        return _exact_simulate(case, seed)
    if kind == "demod":
        s = Setup(case)
        return _exact_demod(_echoes(case, s, seed, rf=True), s, case["taps"], case["decimation"])
    return {"flow": _exact_flow, "strain": _exact_strain, "display": _exact_display, "train": _exact_train}[kind](case, seed)


def _window(w, u):
    t = 0.5 * (u + 1)
    if w == HANN:
        v = 0.5 * (1 - torch.cos(2 * math.pi * t))
    elif w == TUKEY:  # alpha 0.5
        a = 0.5
        v = torch.ones_like(u)
        v = torch.where(t < a / 2, 0.5 * (1 + torch.cos(2 * math.pi / a * (t - a / 2))), v)
        v = torch.where(t > 1 - a / 2, 0.5 * (1 + torch.cos(2 * math.pi / a * (t - 1 + a / 2))), v)
    else:
        v = torch.ones_like(u)
    return torch.where((u < -1) | (u > 1), torch.zeros_like(v), v)


def _aperture(s, pts, f_number, window, dtype):
    """Receive weights [pixel][channel]; in float32 they say which channels count as active."""
    ex = torch.from_numpy(s.ex).cuda().to(dtype)
    half = 0.5 * pts[:, 2:3].to(dtype) / f_number
    return _window(window, (ex[None] - pts[:, 0:1].to(dtype)) / half.clamp_min(1e-9))


def _sensitivity(s, t, px, pz):
    """Transmit illumination weight: the firing aperture's band, widened by diffraction, Tukey 0.4."""
    on = s.ex[t["apodization"] != 0].astype(np.float64)
    lo, hi = float(on[0]), float(on[-1])
    if t["type"] == PLANE:
        shift = pz * math.tan(t["angle"])
        a, b = lo + shift, hi + shift
    else:
        fx, zf = t["focus"][0], t["focus"][2]
        a, b = lo + (fx - lo) * pz / zf, hi + (fx - hi) * pz / zf
        a, b = torch.minimum(a, b), torch.maximum(a, b)
    wide = (pz / max(hi - lo, s.pitch)).clamp(0.5, 20.0) * (s.c / s.f0)
    a, b = a - wide, b + wide
    u = (px - 0.5 * (a + b)) / (0.5 * (b - a))
    tt, al = 0.5 * (u + 1), 0.4
    v = torch.ones_like(u)
    v = torch.where(tt < al / 2, 0.5 * (1 + torch.cos(2 * math.pi / al * (tt - al / 2))), v)
    v = torch.where(tt > 1 - al / 2, 0.5 * (1 + torch.cos(2 * math.pi / al * (tt - 1 + al / 2))), v)
    return torch.where((u < -1) | (u > 1), torch.zeros_like(v), v)


def _compound(s, iq, pts, events):
    """Compounded, focused channel samples [pixel][channel] (complex128), without receive weights."""
    px, pz = pts[:, 0].double(), pts[:, 2].double()
    ex = torch.from_numpy(s.ex).cuda().double()
    rt = torch.hypot(px[:, None] - ex[None], pz[:, None]) / s.c
    y = torch.zeros(rt.shape, dtype=torch.complex128, device="cuda")
    for e in events:
        t = s.tx[e]
        tau, tw = _arrival(t, px, pz, s.c), _sensitivity(s, t, px, pz)
        idx = (tau[:, None] + rt) * s.fs
        k = idx.floor()
        f = idx - k
        k = k.long()
        ok = (k >= 0) & (k + 1 < s.n_smp)
        k = k.clamp(0, s.n_smp - 2).t()
        tr = iq[e].to(torch.complex128)
        a, b = tr.gather(1, k).t(), tr.gather(1, k + 1).t()
        w = torch.polar(tw, 2 * math.pi * s.f0 * tau)
        y += w[:, None] * torch.where(ok, a + (b - a) * f, torch.zeros_like(a))
    return y * torch.polar(torch.ones_like(rt), 2 * math.pi * s.f0 * rt)


def _exact_das(case, s, iq, pts):
    pts = torch.from_numpy(pts).cuda()
    n_ev = len(s.tx) // s.frames
    out = torch.empty((s.frames, pts.shape[0]), dtype=torch.complex128, device="cuda")
    for fr in range(s.frames):
        for p0 in range(0, pts.shape[0], 65536):
            p = pts[p0:p0 + 65536]
            act = _aperture(s, p, case["f_number"], case["window"], torch.float32) > 0
            ap = _aperture(s, p, case["f_number"], case["window"], torch.float64) * act
            y = _compound(s, iq, p, range(fr * n_ev, (fr + 1) * n_ev)) * ap
            n_act = act.sum(1)
            if case["combiner"] == DMAS:
                v = y / y.abs().sqrt().clamp_min(1e-300)
                z = 0.5 * (v.sum(1).square() - v.square().sum(1)) / (0.5 * (n_act - 1).clamp_min(1))
            else:
                z = y.sum(1)
            if case["cf"]:
                inc = y.abs().square().sum(1)
                z = z * torch.where(inc > 0, y.sum(1).abs().square() / (n_act * inc), torch.zeros_like(inc))
            out[fr, p0:p0 + 65536] = torch.where(n_act > 0, z, torch.zeros_like(z))
    if case["kind"] == "pipeline":
        return out.reshape(case["n0"], case["n1"]).cpu().numpy()
    return out.reshape(s.frames, case["n0"], case["n1"])


def _exact_demod(rf, s, taps, dec):
    n = np.arange(taps) - taps // 2
    fc = min(max(0.5 * s.f0 / s.fs, 1e-4), 0.499)
    h = 2 * fc * np.sinc(2 * fc * n) * (0.54 - 0.46 * np.cos(2 * np.pi * np.arange(taps) / (taps - 1)))
    h = h / h.sum()
    t = torch.arange(s.n_smp, device="cuda", dtype=torch.float64) / s.fs
    rot = torch.polar(torch.ones_like(t), -2 * math.pi * s.f0 * t)
    out = []
    for e in range(rf.shape[0]):
        m = torch.nn.functional.pad(rf[e].double() * rot, (taps // 2, taps // 2))
        out.append(2 * sum(float(h[j]) * m[:, taps - 1 - j:taps - 1 - j + s.n_smp] for j in range(taps))[:, ::dec])
    return torch.stack(out)


def _exact_capon(case, seed):
    """Minimum variance: per pixel the spatially smoothed, range-averaged covariance, loaded and solved.
    For the learned method the network's weights, the subspace solve and the level gate around it."""
    learned = case["kind"] == "learned"
    s = Setup(case)
    iq, pts = _echoes(case, s, seed, rf=False), torch.from_numpy(_grid(case)[3]).cuda()
    n0, n1 = case["n0"], case["n1"]
    sub, ra, loading = (64, 2, _f32(0.01)) if learned else (case["subarray"], case["range_avg"], _f32(0.01))
    n_pix = n0 * n1
    y = torch.zeros((n0, n1 + 2 * ra, s.n_el), dtype=torch.complex128, device="cuda")
    act = torch.empty((n_pix, s.n_el), dtype=torch.bool, device="cuda")
    step = max(1, 65536 // n1)
    for i in range(0, n0, step):
        p = pts[i * n1:(i + step) * n1]
        on = _aperture(s, p, case["f_number"], HANN, torch.float32) > 0
        act[i * n1:(i + step) * n1] = on
        y[i:i + step, ra:ra + n1] = (_compound(s, iq, p, range(len(s.tx))) * on).view(-1, n1, s.n_el)
    n_act, first = act.sum(1), act.to(torch.uint8).argmax(1)
    j = torch.arange(n_pix, device="cuda") % n1
    n_d = (torch.minimum(j + ra, torch.full_like(j, n1 - 1)) - (j - ra).clamp_min(0) + 1).double()
    out = torch.zeros(n_pix, dtype=torch.complex128, device="cuda")
    trace = torch.zeros(n_pix, dtype=torch.float64, device="cuda")
    sub_out = torch.zeros_like(out)
    yf = y.view(-1, s.n_el)
    net = _exact_network() if learned else None
    for n in n_act.unique().tolist():
        all_pix = (n_act == n).nonzero()[:, 0]
        L = min(max(sub, 2), max(2, n // 2))
        n_sub = n - L + 1
        for pix in all_pix.split(max(64, int(2e9 / (16 * max(1, L * n_sub * (2 * ra + 1)))))):
            row = (pix // n1) * (n1 + 2 * ra) + pix % n1 + ra
            ch = first[pix, None] + torch.arange(n, device="cuda")
            centre = yf[row[:, None], ch] if n else None
            if n < 4:
                out[pix] = centre.sum(1) if n else 0
                continue
            rows = torch.stack([yf[(row + d)[:, None], ch] for d in range(-ra, ra + 1)], 1)
            x = rows.unfold(2, n_sub, 1).permute(0, 2, 1, 3).reshape(len(pix), L, -1)
            R = torch.bmm(x, x.mH) / (n_d[pix] * n_sub)[:, None, None]
            tr = R.diagonal(dim1=1, dim2=2).real.sum(1)
            eps = (loading * tr / L).clamp_min(1e-20)
            avg = centre.unfold(1, n_sub, 1).mean(2)
            A = R + eps[:, None, None] * torch.eye(L, device="cuda")
            w = _ones_solve(A)
            out[pix] = n * (w.conj() * avg).sum(1) / w.sum(1)
            if learned:
                trace[pix] = tr
                sub_out[pix] = n * _exact_subspace(net, R, A, avg, n, L)
    if learned:
        t = trace.view(n0, n1)
        live = t > 0
        level = torch.where(live, t.clamp_min(1e-300).log(), 0.0).sum(0) / live.sum(0).clamp_min(1)
        gate = math.log(usx_learned.trained_level_gate(usx_learned.DEFAULT_WEIGHTS))
        hot = (t.clamp_min(1e-300).log() - level[None] > gate).view(-1)
        out = torch.where((n_act >= 4) & ~hot, sub_out, out)
    return out.view(1, n0, n1)


def _ones_solve(A):
    """A^-1 1 of positive definite matrices by an explicit Cholesky factor (column by column, batched)."""
    A = A.clone()
    L = A.shape[1]
    b = torch.ones(A.shape[:2], dtype=A.dtype, device="cuda")
    for c in range(L):  # left half: factor and forward substitution
        A[:, c:, c] /= A[:, c, c].real.sqrt()[:, None]
        b[:, c] /= A[:, c, c]
        if c + 1 < L:
            col = A[:, c + 1:, c]
            A[:, c + 1:, c + 1:] -= col[:, :, None] * col[:, None, :].conj()
            b[:, c + 1:] -= col * b[:, c:c + 1]
    for c in range(L - 1, -1, -1):
        b[:, c] = (b[:, c] - (A[:, c + 1:, c].conj() * b[:, c + 1:]).sum(1)) / A[:, c, c]
    return b


def _exact_network():
    raw = (ROOT / "ultrasound-engine_gb300" / "weights" / "learned_mv_128ch_l64.bin").read_bytes()
    n = int(np.frombuffer(raw, "<i4", 1, 8)[0])
    dims = np.frombuffer(raw, "<i4", n + 1, 12)
    p, o, layers = torch.from_numpy(np.frombuffer(raw, "<f4", offset=12 + 4 * (n + 1)).copy()).cuda(), 0, []
    for a, b in zip(dims[:-1].tolist(), dims[1:].tolist()):
        layers.append((p[o:o + a * b].view(a, b).bfloat16().double(), p[o + a * b:o + a * b + b].double()))
        o += a * b + b
    return layers


def _exact_subspace(net, R, A, avg, n, L):
    """Output of the Capon problem within span{DFT beams 0, +-1, +-2, +-3, the network's direction}."""
    P = R.shape[0]
    f = torch.zeros((P, 256), dtype=torch.float64, device="cuda")
    r0 = R.diagonal(dim1=1, dim2=2).real.mean(1)
    for m in range(1, L):
        r = R.diagonal(offset=-m, dim1=1, dim2=2).mean(1) / r0
        f[:, 2 * m], f[:, 2 * m + 1] = r.real, r.imag
    f[:, 0], f[:, 1] = L / 64.0, n / 128.0
    u = avg.sum(1)
    u = u / u.abs().clamp_min(1e-300)
    a = avg * u.conj()[:, None] / avg.abs().square().mean(1).sqrt()[:, None]
    f[:, 128:128 + 2 * L] = torch.view_as_real(a).reshape(P, -1)
    h = f.float().bfloat16().double()  # the network's inputs and activations are BF16
    for k, (W, b) in enumerate(net):
        h = h @ W + b
        if k + 1 < len(net):
            h = h.clamp_min(0).float().bfloat16().double()
    w = torch.view_as_complex(h.view(P, 64, 2).contiguous())[:, :L] / L
    i = torch.arange(L, device="cuda", dtype=torch.float64)
    beams = [0, 1, -1, 2, -2, 3, -3][:L]
    Q = torch.stack([torch.polar(torch.full_like(i, L ** -0.5), 2 * math.pi * b * i / L) for b in beams], 1)
    q = w - (w @ Q.conj()) @ Q.t()
    keep = (q.abs().square().sum(1) > 1e-4 * w.abs().square().sum(1))[:, None]
    q = torch.where(keep, q / q.abs().square().sum(1).sqrt().clamp_min(1e-300)[:, None], torch.zeros_like(q))
    B = torch.cat([Q[None].expand(P, -1, -1), q[:, :, None]], 2)
    G = B.mH @ A @ B
    G[:, -1, -1] = torch.where(keep[:, 0], G[:, -1, -1], torch.ones_like(G[:, -1, -1]))
    rhs = B.mH.sum(2)
    c = torch.linalg.solve(G, rhs[:, :, None])[:, :, 0]
    wc = (B @ c[:, :, None])[:, :, 0]
    return (wc.conj() * avg).sum(1) / wc.conj().sum(1)


def _exact_simulate(case, seed):
    s = Setup(case)
    x, z, amp = (v.double() for v in _phantom(s, case, seed, case["scatterers"]))
    x, z, amp = x[amp != 0], z[amp != 0], amp[amp != 0]
    ex = torch.from_numpy(s.ex).cuda().double()
    r = torch.hypot(x[:, None] - ex[None], z[:, None])
    sin = (x[:, None] - ex[None]) / r
    arg = math.pi * s.width * sin * s.f0 / s.c
    resp = (1 - sin.square()).clamp_min(0).sqrt() * torch.special.sinc(arg / math.pi) / r
    resp = resp * torch.pow(10.0, -(0.5 * s.f0 * 1e-6 * 100.0) * r / 20.0)
    sigma = math.sqrt(2 * math.log(2)) / (math.pi * BANDWIDTH * s.f0)
    fo = 4 * s.fs
    nh = int(math.ceil(3 * sigma * fo))
    half, P = nh / fo, 2 * nh + 1
    tp = torch.arange(-nh, nh + 1, device="cuda", dtype=torch.float64) / fo
    pulse = torch.exp(-0.5 * (tp / sigma).square()) * torch.cos(2 * math.pi * s.f0 * tp)
    out = torch.zeros((len(s.tx), s.n_el, s.n_smp), dtype=torch.float64, device="cuda")
    taps = torch.arange(P + 1, device="cuda")
    lead = torch.cat([pulse, pulse.new_zeros(1)])   # this slot's tap
    lag = torch.cat([pulse.new_zeros(1), pulse])    # the tap before it
    for e, t in enumerate(s.tx):
        on = np.nonzero(t["apodization"])[0].tolist()
        dly = torch.from_numpy(t["delays"]).cuda().double()
        arr = r / s.c + dly[None]
        t_lo, t_hi = arr[:, on].amin(1), arr[:, on].amax(1)
        span = torch.minimum(t_hi - t_lo + 2 * half, torch.full_like(t_lo, 30e-6 + 2 * half))
        begin = t_lo - half
        n_inc = (span * fo).ceil().long() + 2
        W = int(n_inc.max())
        inc = torch.zeros((len(x), W + 1), dtype=torch.float64, device="cuda")
        for q in on:
            a = float(t["apodization"][q]) * resp[:, q]
            ctr = (arr[:, q] - begin) * fo
            fr = (ctr - ctr.floor())[:, None]
            slot = (ctr.floor().long() - P // 2)[:, None] + taps[None]
            nx = (slot >= 1) & (slot < n_inc[:, None])
            th = (slot >= 0) & (slot + 1 < n_inc[:, None])
            v = a[:, None] * (lag[None] * fr * nx + lead[None] * (1 - fr) * th)
            inc.scatter_add_(1, torch.where(nx | th, slot, W), v)
        inc = inc[:, :W]
        keep = inc.abs() >= inc.abs().amax(1, keepdim=True) * 10 ** (-40.0 / 20.0)
        lo = keep.to(torch.uint8).argmax(1)
        hi = W - 1 - keep.flip(1).to(torch.uint8).argmax(1)
        t0 = begin + lo.double() / fo
        m = hi - lo + 1
        for q in range(s.n_el):
            d = r[:, q] / s.c
            start = t0 + d
            n_lo = (start * s.fs).ceil().long().clamp_min(0)
            n_hi = ((start + (m - 1).double() / fo) * s.fs).floor().long().clamp_max(s.n_smp - 1)
            wide = int((n_hi - n_lo).max()) + 1
            if wide <= 0:
                continue
            smp = n_lo[:, None] + torch.arange(wide, device="cuda")[None]
            u = (smp.double() / s.fs - start[:, None]) * fo
            k = u.floor().long()
            ok = (smp <= n_hi[:, None]) & (k >= 0) & (k + 1 < m[:, None])
            kk = (lo[:, None] + k).clamp(0, W - 2)
            a, b = inc.gather(1, kk), inc.gather(1, kk + 1)
            v = (amp * resp[:, q])[:, None] * (a + (b - a) * (u - k))
            out[e, q].index_add_(0, smp[ok], v[ok])
    if case["noise"]:
        g = torch.randn(out.shape, device="cuda", generator=_gen(seed, 7))
        out = out + g.double() * out.abs().amax((1, 2), keepdim=True) * 10 ** (-60.0 / 20.0)
    return out


def _exact_flow(case, seed):
    ens = _flow_input(case, seed).to(torch.complex128)
    axis = _flow_axis(case).astype(np.float64)
    dz, maps, o = float(np.float32(axis[1] - axis[0])), [], 0
    ka, kl = case["ka"], case["kl"]

    def box(v):
        p = torch.nn.functional.pad(v, (ka, ka, kl, kl))
        return sum(p[i:i + v.shape[0], k:k + v.shape[1]] for i in range(2 * kl + 1) for k in range(2 * ka + 1))

    for n in _flow_lengths(case):
        z = ens[o:o + n]
        o += n
        x = np.linspace(-1, 1, n)
        basis, _ = np.linalg.qr(np.stack([x ** d for d in range(min(case["order"], n - 1) + 1)], 1))
        M = torch.from_numpy(np.eye(n) - basis @ basis.T).cuda().to(torch.complex128)
        z = torch.einsum("ij,jkl->ikl", M, z)
        r00 = box(z.abs().square().sum(0))
        r01 = box((z[:-1].conj() * z[1:]).sum(0))
        r10 = torch.nn.functional.pad((z[:, :, :-1].conj() * z[:, :, 1:]).sum(0), (0, 1))
        r10 = box(r10)
        coh = r01.abs() / r00
        var = (2 * (1 - coh)).clamp(0, 1)
        f = torch.full_like(r00, 5e6)
        if case["loupas"]:
            est = r10.angle() * C0 / (4 * math.pi * dz)
            f = torch.where((est > 0.25 * 5e6) & (est < 2 * 5e6), est, f)
        vel = torch.where(coh < _f32(0.35), torch.zeros_like(f), -r01.angle() * C0 * 5e3 / (4 * math.pi * f))
        maps.append((vel, r00, var))
    vel, power, var = (torch.stack(v) for v in zip(*maps))
    return [vel, power, var, None]


def _exact_strain(case, seed):
    a, b = (v.to(torch.complex128) for v in _strain_input(case, seed))
    axis = _strain_axis(case).astype(np.float64)
    dz, n0, n1 = float(np.float32(axis[1] - axis[0])), case["n0"], case["n1"]
    ka, kl, ml = case["ka"], case["kl"], case["max_lag"]

    def box(v):
        p = torch.nn.functional.pad(v, (ka, ka, kl, kl))
        p = sum(p[i:i + n0] for i in range(2 * kl + 1))
        return sum(p[:, k:k + n1] for k in range(2 * ka + 1))

    r10 = box(torch.nn.functional.pad(a[:, :-1].conj() * a[:, 1:], (0, 1)))
    est = r10.angle() * C0 / (4 * math.pi * dz)
    f = torch.where((est > 0.25 * 5e6) & (est < 2 * 5e6), est, torch.full_like(est, 5e6))
    best = torch.full((n0, n1), -1.0, dtype=torch.float64, device="cuda")
    arg, lagmap = torch.zeros_like(best), torch.zeros_like(best)
    j = torch.arange(n1, device="cuda")
    for lag in range(-ml, ml + 1):
        ok = ((j + lag >= 0) & (j + lag < n1)).double()[None]
        bl = b[:, (j + lag).clamp(0, n1 - 1)]
        R = box(a.conj() * bl * ok)
        ea, eb = box(a.abs().square() * ok), box(bl.abs().square() * ok)
        cr = torch.where((ea > 0) & (eb > 0), R.abs() / (ea * eb).sqrt().clamp_min(1e-300), best)
        up = cr > best
        best, arg, lagmap = torch.where(up, cr, best), torch.where(up, R.angle(), arg), torch.where(up, float(lag), lagmap)
    axial = lagmap * dz - arg * C0 / (4 * math.pi * f)
    half = max(1, case["fit"] // 2)
    pad = torch.nn.functional.pad(torch.stack([axial, torch.ones_like(axial)]), (half, half))
    sx = sy = sxx = sxy = cnt = 0
    for d in range(-half, half + 1):
        v, one = pad[0][:, half + d:half + d + n1], pad[1][:, half + d:half + d + n1]
        cnt, sx, sy, sxx, sxy = cnt + one, sx + d * dz * one, sy + v, sxx + (d * dz) ** 2 * one, sxy + d * dz * v
    return [axial, best.clamp(0, 1), (cnt * sxy - sx * sy) / (cnt * sxx - sx * sx)]


def _exact_display(case, seed):
    gtype, a0, a1, pts = _display_grid(case)
    n0, n1, W, H = case["n0"], case["n1"], case["width"], case["height"]
    env = _display_input(case, seed).to(torch.complex128).abs()
    p = torch.from_numpy(pts).cuda().double().view(n0, n1, 3)
    tgc = env * torch.pow(10.0, 2 * 0.5 * 5.0 * (p[..., 2] * 100).clamp_min(0) / 20.0)
    log = ((20 * torch.log10(tgc / tgc.max()) + 60.0) / 60.0).clamp(0, 1)

    def place(dtype):
        """Grid coordinates of the raster and what lies inside the sector."""
        def lin(lo, hi, n):
            return lo + (hi - lo) * (torch.arange(n, device="cuda", dtype=dtype) / (n - 1))
        q = torch.from_numpy(pts).cuda().to(dtype)
        b0, b1 = torch.from_numpy(a0).cuda().to(dtype), torch.from_numpy(a1).cuda().to(dtype)
        zz = lin(q[:, 2].min(), q[:, 2].max(), H)[:, None].expand(H, W)
        xx = lin(q[:, 0].min(), q[:, 0].max(), W)[None].expand(H, W)
        inside = torch.ones((H, W), dtype=torch.bool, device="cuda")
        if gtype == 1:
            rr, th = torch.sqrt(xx * xx + zz * zz), torch.atan2(xx, zz)
            inside = (rr >= b1[0]) & (rr <= b1[-1]) & (th >= b0[0]) & (th <= b0[-1])
            xx, zz = th, rr
        return (xx - b0[0]) / (b0[-1] - b0[0]) * (n0 - 1), (zz - b1[0]) / (b1[-1] - b1[0]) * (n1 - 1), inside

    u32, v32, inside = place(torch.float32)  # the cell of a pixel is chosen in float32
    u, v, _ = place(torch.float64)
    i, j = u32.floor().long(), v32.floor().long()
    inside = inside & (i >= 0) & (j >= 0) & (i + 1 < n0) & (j + 1 < n1)
    i, j = i.clamp(0, max(0, n0 - 2)), j.clamp(0, max(0, n1 - 2))
    fu, fv = u - i, v - j
    px = ((log[i, j] * (1 - fu) + log[i + 1, j] * fu) * (1 - fv) + (log[i, j + 1] * (1 - fu) + log[i + 1, j + 1] * fu) * fv)
    return [env, tgc, log, torch.where(inside, px, torch.zeros_like(px))]


def _exact_train(case, seed):
    p, x, target = _train_input(case, seed)
    q, o, leaves, layers = torch.from_numpy(p).cuda(), 0, [], []
    for a, b in zip(TRAIN_DIMS[:-1], TRAIN_DIMS[1:]):
        W = q[o:o + a * b].view(a, b).bfloat16().double().requires_grad_()
        c = q[o + a * b:o + a * b + b].double().requires_grad_()
        o += a * b + b
        layers.append((W, c))
        leaves += [W, c]
    h = x.bfloat16().double()
    for k, (W, c) in enumerate(layers):
        h = h @ W + c
        if k + 1 < len(layers):
            h = h.clamp_min(0)
    loss = (h - target.double()).square().mean()
    grads = torch.autograd.grad(loss, leaves)
    return [loss.item(), torch.cat([g.reshape(-1) for g in grads]).cpu().numpy()]
