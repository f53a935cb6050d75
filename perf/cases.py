"""The work a user of this package has it do, as cases that can be timed.

Each case is one call (or one differentiated call) of the public interface at
a size from this repository's benchmark, tests or documented workloads:

* ``signal`` / ``jacobian``: a compiled MRF train over tissue maps, the
  signal alone or with fused Jacobian columns (dictionary building, model
  evaluation over a slice);
* ``gradient`` / ``precision``: one step of sequence design, the signal's
  (or the Jacobian's) cotangent pulled back to flips, TRs and tissue;
* ``offaxis``: the same gradient with RF phases, B0 and B1phase maps;
* ``train``: a default-phase CPMG echo train through ``fse_sim``;
* ``batch``: many uneven CPMG protocols in one captured launch;
* ``match``: dictionary matching of noisy signals;
* ``map``: Levenberg-Marquardt mapping of noisy signals.

The reference values (``exact``) and the synthetic measurements come from the
plain float64 recursion in this file, not from the package.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from torchsim_gb300 import DictionaryMatcher, GaussNewton, MRFSimulator, TrustRegion, engine, fse_sim
from torchsim_gb300.batching import BatchEntry, SequenceBatch
from torchsim_gb300.sequence import fse_events, mrf_events, program_for

BOUNDS = {"T1": (50.0, 5000.0), "T2": (2.0, 1000.0), "M0": (0.0, 5.0)}
START = (550.0, 55.0, 1.0)  # medians of the tissue ranges


def listed():
    return [
        # One 32 x 32 slice through a known sequence: latency decides.
        dict(name="signal_slice", kind="signal", voxels=1024, pulses=880, states=10),
        # The published dictionary benchmark: 500 repetitions, 32 orders.
        dict(name="signal_dictionary", kind="signal", voxels=100_000, pulses=500, states=32),
        # The slice again with the two columns a T1/T2 fit linearises with.
        dict(name="jacobian_slice", kind="jacobian", voxels=1024, pulses=880, states=10,
             diff="T1,T2"),
        # The published Jacobian benchmark.
        dict(name="jacobian_published", kind="jacobian", voxels=100_000, pulses=500, states=32,
             diff="T1,T2"),
        # The benchmark's dictionary: 128 x 64 x 32 atoms, three columns.
        dict(name="jacobian_dictionary", kind="jacobian", voxels=262_144, pulses=880, states=20,
             diff="T1,T2,B1"),
        # Sequence design against a target signal: 600 flips and TRs.
        dict(name="gradient_design", kind="gradient", voxels=16_384, pulses=600, states=20),
        # Sequence design against a Cramer-Rao bound of four parameters.
        dict(name="precision_design", kind="precision", voxels=16_384, pulses=600, states=20,
             diff="T1,T2,B1,M0"),
        # A phase-cycled, off-resonant train and its gradients.
        dict(name="offaxis_gradient", kind="offaxis", voxels=16_384, pulses=600, states=20),
        # Default-phase fast spin echo over a multi-slice volume, with T1, T2 columns.
        dict(name="echo_train", kind="train", voxels=65_536, pulses=48, states=32, diff="T1,T2"),
        # A protocol sweep: uneven CPMG trains in one launch.
        dict(name="cpmg_batch", kind="batch", sequences=96, longest=64),
        # Matching a slice stack against a mid-sized dictionary.
        dict(name="match_dictionary", kind="match", voxels=16_384, atoms=65_536, pulses=500, top_k=1),
        # Mapping one 128 x 128 slice with ten steps.
        dict(name="map_slice", kind="map", voxels=16_384, pulses=880, states=10, steps=10),
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["signal", "signal", "jacobian", "jacobian", "jacobian", "gradient",
                       "gradient", "precision", "offaxis", "train", "batch", "match", "map"])
    if kind == "batch":
        return dict(kind=kind, sequences=_spread(rng, 4, 96), longest=rng.randint(12, 64))
    if kind == "match":
        return dict(kind=kind, voxels=_spread(rng, 256, 16_384), atoms=_spread(rng, 2048, 65_536),
                    pulses=_spread(rng, 64, 880), top_k=rng.choice([1, 1, 2, 5]))
    if kind == "map":
        return dict(kind=kind, voxels=_spread(rng, 512, 32_768), pulses=_spread(rng, 200, 880),
                    states=rng.choice([8, 10, 10, 15]), steps=rng.choice([5, 10]))
    if kind == "train":
        return dict(kind=kind, voxels=_spread(rng, 512, 131_072), pulses=rng.randint(8, 64),
                    states=rng.choice([8, 10, 16, 25, 32]), diff=rng.choice(["", "T1,T2", "T2,B1"]))
    case = dict(kind=kind, voxels=0, pulses=_spread(rng, 100, 1000),
                states=rng.choice([6, 8, 10, 10, 13, 16, 20, 20, 27, 32, 40]))
    case["voxels"] = _spread(rng, 256, 131_072 if kind in ("signal", "jacobian") else 32_768)
    if kind == "jacobian":
        case["diff"] = rng.choice(["T1", "T1,T2", "T1,T2", "T1,T2,M0", "T1,T2,B1", "T1,T2,B1,M0"])
    if kind == "precision":
        case["diff"] = rng.choice(["T1,T2", "T1,T2,M0", "T1,T2,B1,M0"])
    # Every order, pulse and voxel counts alike: large sizes are not drawn together.
    most = {"signal": 4e9, "jacobian": 3e9}.get(kind, 2.5e8)
    work = case["voxels"] * case["pulses"] * case["states"]
    if work > most:
        case["voxels"] = max(257, int(case["voxels"] * most / work))
    return case


# ---- inputs --------------------------------------------------------------------

DEVICE = "cuda"


class _Draws:
    """Seeded draws on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def uniform(self, low, high, *shape):
        return low + (high - low) * torch.rand(shape, device=DEVICE, generator=self.gen)

    def log_uniform(self, low, high, *shape):
        return torch.exp(self.uniform(math.log(low), math.log(high), *shape))

    def cotangent(self, *shape):
        return torch.randn(shape, dtype=torch.complex64, device=DEVICE, generator=self.gen)

    def tissue(self, voxels):
        """T1 (ms), T2 (ms) and B1 as the benchmark's workloads draw them."""
        t1 = self.log_uniform(100, 3000, voxels)
        t2 = torch.minimum(self.log_uniform(10, 300, voxels), 0.999 * t1)
        return t1, t2, self.uniform(0.7, 1.3, voxels)


def _schedule(pulses):
    """The benchmark's flip train (5 to 60 to 2 degrees, then held), any length."""
    up = (pulses * 300 + 439) // 880
    hold = pulses - 2 * up
    return np.concatenate([np.linspace(5, 60, up), np.linspace(60, 2, up),
                           np.full(hold, 2.0)]).astype(np.float32)


def _batch_entries(case, seed):
    """The benchmark's uneven protocols: the case alone decides their lengths
    and voxel counts, the seed their flips, spacings and tissue."""
    sizes = np.random.default_rng(1000 * case["sequences"] + case["longest"])
    rng = np.random.default_rng(seed)
    entries = []
    for _ in range(case["sequences"]):
        echoes = int(sizes.integers(min(8, case["longest"]), case["longest"] + 1))
        voxels = int(round(np.exp(sizes.uniform(np.log(1e3), np.log(6.4e4)))))
        entries.append(dict(flip=rng.uniform(100, 180, echoes).astype(np.float32),
                            esp=float(rng.uniform(5, 15)),
                            t1=rng.uniform(300, 3000, voxels).astype(np.float32),
                            t2=rng.uniform(10, 300, voxels).astype(np.float32),
                            b1=rng.uniform(0.7, 1.3, voxels).astype(np.float32)))
    return entries


def _inputs(case, seed):
    """What the case is computed from: tensors on the GPU and plain values."""
    kind, rand = case["kind"], _Draws(seed)
    if kind == "batch":
        return dict(entries=_batch_entries(case, seed))
    V, P = case["voxels"], case["pulses"]
    s = {}
    if kind == "match":
        t1, t2, b1 = rand.tissue(case["atoms"])
        atoms = _samples(_schedule(P), 10.0, t1, t2, b1, 16)
        truth = torch.randint(0, case["atoms"], (V,), device=DEVICE, generator=rand.gen)
        turn = torch.polar(rand.uniform(0.5, 1.5, V), rand.uniform(-math.pi, math.pi, V))
        signal = atoms[truth] * turn[:, None]
        noise = rand.cotangent(V, P) * (signal.abs().mean() / 50)
        return dict(atoms=atoms, grid=torch.stack((t1, t2, b1), 1), signal=signal + noise)
    s["t1"], s["t2"], s["b1"] = rand.tissue(V)
    if kind == "map":
        m0 = rand.uniform(0.5, 1.5, V)
        signal = _samples(_schedule(P), 10.0, s["t1"], s["t2"], s["b1"], case["states"]) * m0[:, None]
        s["signal"] = signal + rand.cotangent(V, P) * (signal.abs().mean() / 50)
        return s
    if kind == "train":
        s["flip"] = rand.uniform(100, 180, P).cpu()
        return s
    if kind in ("signal", "jacobian"):
        s["flip"], s["tr"] = torch.from_numpy(_schedule(P)), 10.0
        return s
    s["flip"], s["tr"] = rand.uniform(5, 70, P), rand.uniform(8, 15, P)
    s["seed"] = rand.cotangent(V, P)
    if kind == "precision":
        s["m0"] = rand.uniform(0.5, 1.5, V)
        s["seed_jac"] = rand.cotangent(V, len(case["diff"].split(",")), P) * 100.0
    if kind == "offaxis":
        s["phases"] = rand.uniform(-40, 40, P).cpu()
        s["b0"], s["b1_phase"] = rand.uniform(-40, 40, V), rand.uniform(-0.5, 0.5, V)
        s["flip"], s["tr"] = s["flip"].cpu(), s["tr"].cpu()
    return s


def _names(case):
    return tuple(n for n in case.get("diff", "").split(",") if n)


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        batch = SequenceBatch([BatchEntry(fse_events(e["flip"], e["esp"], phases_deg=90.0),
                                          2 * len(e["flip"]), e["t1"], e["t2"], e["b1"])
                               for e in s["entries"]], torch.device(DEVICE, 0))
        batch.tune(use_cache=False)
        batch.capture()
        return dict(kind=kind, batch=batch)
    if kind == "match":
        matcher = DictionaryMatcher(dictionary=s["atoms"], parameters=s["grid"], top_k=case["top_k"])
        return dict(kind=kind, matcher=matcher, signal=s["signal"])
    s.update(kind=kind, states=case.get("states"), names=_names(case))
    if kind in ("signal", "jacobian", "map"):
        flip, tr = (s["flip"], s["tr"]) if kind != "map" else (_schedule(case["pulses"]), 10.0)
        s["program"] = program_for(mrf_events(flip, tr))
    if kind in ("signal", "jacobian"):
        s["maps"] = engine.tissue_maps(torch.device(DEVICE, 0), case["voxels"], s["t1"], s["t2"],
                                       None, s["b1"], None)
    if kind == "map":
        s["loop"] = GaussNewton(TrustRegion(), max_iterations=case["steps"])
    if kind in ("gradient", "precision", "offaxis"):
        for name in ("t1", "t2", "flip", "tr", "b0"):
            if name in s:
                s[name].requires_grad_(True)
    return s


def run(s):
    kind = s["kind"]
    if kind == "signal":
        return engine.forward(s["program"], s["maps"], s["states"])
    if kind == "jacobian":
        return engine.forward_tangents(s["program"], s["maps"], s["states"], s["names"])
    if kind == "gradient":
        signal = MRFSimulator(flip=s["flip"], TR=s["tr"], states=s["states"]).simulate(
            T1=s["t1"], T2=s["t2"], B1=s["b1"])
        leaves = [s[k] for k in ("flip", "tr", "t1", "t2")]
        return signal.detach(), *torch.autograd.grad(signal, leaves, s["seed"])
    if kind == "precision":
        signal, jac = MRFSimulator(flip=s["flip"], TR=s["tr"], states=s["states"]).jacobian(
            s["names"], T1=s["t1"], T2=s["t2"], B1=s["b1"], M0=s["m0"])
        leaves = [s[k] for k in ("flip", "tr", "t1", "t2")]
        return signal.detach(), jac.detach(), *torch.autograd.grad((signal, jac), leaves,
                                                                   (s["seed"], s["seed_jac"]))
    if kind == "offaxis":
        signal = MRFSimulator(flip=s["flip"], TR=s["tr"], phases=s["phases"],
                              states=s["states"]).simulate(
            T1=s["t1"], T2=s["t2"], B1=s["b1"], B0=s["b0"], B1phase=s["b1_phase"])
        leaves = [s[k] for k in ("flip", "tr", "t1", "t2", "b0")]
        return signal.detach(), *torch.autograd.grad(signal, leaves, s["seed"])
    if kind == "train":
        return fse_sim(s["flip"], 8.0, s["t1"], s["t2"], B1=s["b1"], TR=3000.0,
                       states=s["states"], diff=s["names"] or None)
    if kind == "batch":
        s["batch"].run()
        return s["batch"].out
    if kind == "match":
        found = s["matcher"].match(s["signal"])
        return dict(parameters=found.parameters, indices=found.indices, scores=found.scores,
                    scales=found.scales, densities=found.densities)
    found = s["loop"].minimize_program(s["program"], s["signal"], torch.tensor(START), BOUNDS,
                                       s["states"], b1=s["b1"])
    return dict(maps=found.x)


def work(case):
    """Each input read and each output written once; per order of one voxel
    through one pulse 18 FP32 operations for the signal and 42 per tangent
    (relaxation and rotation), twice as many again to pull a cotangent back,
    and 70 instead of 18 where the planes are complex."""
    kind = case["kind"]
    k = len(_names(case))
    if kind == "batch":
        # The mean protocol: half way between the shortest and the longest,
        # and the mean of the log-uniform voxel count.
        echoes = (min(8, case["longest"]) + case["longest"]) / 2
        voxels = case["sequences"] * (6.4e4 - 1e3) / math.log(64)
        return {"bytes": voxels * (12 + 8 * echoes), "flops": 18.0 * voxels * 2 * echoes * echoes}
    V, P = case["voxels"], case["pulses"]
    if kind == "match":
        A = case["atoms"]
        return {"bytes": 8.0 * P * (V + A) + 40.0 * V * case["top_k"], "flops": 4.0 * V * A * P}
    updates = float(V) * P * case["states"]
    if kind == "map":
        return {"bytes": 8.0 * V * P + 40 * V, "flops": updates * 102 * (case["steps"] + 1)}
    out = 8.0 * V * P * (1 + k)
    stateful = sum(n != "M0" for n in _names(case))
    if kind in ("signal", "jacobian"):
        return {"bytes": out + 12 * V, "flops": updates * (18 + 42 * stateful)}
    if kind == "train":
        return {"bytes": out + 12 * V, "flops": updates * (70 + 160 * stateful)}
    if kind == "offaxis":
        return {"bytes": 2 * out + 40 * V, "flops": updates * 70 * 3}
    return {"bytes": 2 * out + 24 * V, "flops": updates * (18 + 42 * stateful) * 3}


# ---- the recursion in plain float64 ----------------------------------------------


def _played(flip):
    """The angle (rad, float32) a hard pulse of ``flip`` degrees plays; the
    area is the hard pulse envelope's integral on its raster."""
    return 2.0 * torch.pi * torch.abs(torch.deg2rad(flip.to(torch.float32)) * 0.15915493667125702)


def _intervals(tr, pulses):
    """The waits (s) before each pulse of an MRF train: differences of a
    float32 clock in microseconds that advances by each TR (ms)."""
    tr = torch.as_tensor(tr, dtype=torch.float32).detach().cpu().reshape(-1).expand(pulses)
    walk = np.cumsum(np.concatenate([np.float32([0.0]), (tr * 1e-3).numpy()]), dtype=np.float32)
    clock = torch.from_numpy(np.float32(1e6) * walk[:pulses])
    return (torch.diff(clock, prepend=clock.new_zeros(1)) * 1e-6).to(torch.float32)


def _mrf_values(flip, tr):
    """Played flips (rad) and waits (s) as float64 on the GPU, through which
    gradients reach ``flip`` (deg) and ``tr`` (ms) in float64."""
    flip = torch.as_tensor(flip)
    with torch.no_grad():
        angle = _played(flip).to(DEVICE, torch.float64)
        wait = _intervals(tr, flip.numel()).to(DEVICE, torch.float64)
    if flip.requires_grad:
        f = flip.to(DEVICE, torch.float64)
        angle = angle + (f - f.detach()) * (math.pi / 180)
        r = torch.as_tensor(tr).to(DEVICE, torch.float64)
        wait = wait + torch.cat([r.new_zeros(1), (r - r.detach())[:-1] * 1e-3])
    return angle, wait


def _mrf(angle, wait, t1, t2, b1, states, names=()):
    """The inversion-prepared real-subspace train: recorded F+[0] of the
    signal and of its derivatives along ``names``, (1 + k, V, P) float64. The
    systems are stacked in front; T1, T2, B1 couple to the signal."""
    V = t1.shape[0]
    C = 1 + len(names)
    col = {n: 1 + i for i, n in enumerate(names)}
    zero = torch.zeros((V, states), dtype=torch.float64, device=t1.device)
    p = torch.zeros((C, V, states), dtype=torch.float64, device=t1.device)
    m = p.clone()
    z = p.clone()
    z[0, :, 0] = -1.0  # the ideal inversion
    first = torch.zeros(states, dtype=torch.float64, device=t1.device)
    first[0] = 1.0
    t1, t2, b1 = t1[:, None], t2[:, None], b1[:, None]
    out = []

    def stacked(terms):
        return torch.stack([terms.get(c, zero) for c in range(C)])

    for k in range(angle.shape[0]):
        e1, e2 = torch.exp(-1e3 * wait[k] / t1), torch.exp(-1e3 * wait[k] / t2)
        k1, k2 = e1 * 1e3 * wait[k] / t1**2, e2 * 1e3 * wait[k] / t2**2
        add_p, add_m, add_z = {}, {}, {0: (1 - e1) * first}
        if "T1" in col:
            add_z[col["T1"]] = k1 * (z[0] - first)
        if "T2" in col:
            add_p[col["T2"]], add_m[col["T2"]] = k2 * p[0], k2 * m[0]
        p, m, z = e2 * p, e2 * m, e1 * z + stacked(add_z)
        if add_p:
            p, m = p + stacked(add_p), m + stacked(add_m)
        a = angle[k] * b1
        si, co = torch.sin(a), torch.cos(a)
        s, d = p + m, p - m
        turn = 0.5 * co * d - si * z
        zn = 0.5 * si * d + co * z
        pn, mn = 0.5 * s + turn, 0.5 * s - turn
        if "B1" in col:
            g = angle[k]
            pn = pn + stacked({col["B1"]: -g * zn[0]})
            mn = mn + stacked({col["B1"]: g * zn[0]})
            zn = zn + stacked({col["B1"]: g * turn[0]})
        p, m, z = pn, mn, zn
        out.append(p[:, :, 0])
        m = torch.cat([m[..., 1:], torch.zeros_like(m[..., :1])], -1)
        p = torch.cat([-m[..., :1], p[..., :-1]], -1)
    return torch.stack(out, -1)


def _samples(flip, tr, t1, t2, b1, states):
    """An MRF signal as a program would have it stored: complex64 on the
    imaginary-free axis the simulators return it on."""
    angle, wait = _mrf_values(flip, tr)
    with torch.no_grad():
        v = _mrf(angle, wait, t1.double(), t2.double(), b1.double(), states)[0]
    return torch.complex(-v, torch.zeros_like(v)).to(torch.complex64)


def _complex_step(p, m, z, angle, phase):
    """One pulse at ``phase`` on the complex planes (V, states)."""
    si, co = torch.sin(angle)[:, None], torch.cos(angle)[:, None]
    u = torch.polar(torch.ones_like(phase), phase)[:, None]
    a, b = 0.5 * (1 + co), 0.5 * (1 - co)
    pn = a * p + u * u * b * m - 1j * u * si * z
    mn = (u * u).conj() * b * p + a * m + 1j * u.conj() * si * z
    zn = -0.5j * u.conj() * si * p + 0.5j * u * si * m + co * z
    return pn, mn, zn


def _complex_shift(p, m):
    m = torch.cat([m[:, 1:], torch.zeros_like(m[:, :1])], -1)
    return torch.cat([m[:, :1].conj(), p[:, :-1]], -1), m


def _complex_start(V, states):
    p = torch.zeros((V, states), dtype=torch.complex128, device=DEVICE)
    z = p.clone()
    z[:, 0] = 1.0
    return p, p.clone(), z


def _first_order(states):
    first = torch.zeros((1, states), dtype=torch.complex128, device=DEVICE)
    first[0, 0] = 1.0
    return first


def _offaxis(angle, wait, phase, t1, t2, b1, b0, b1_phase, states):
    """The MRF train with RF phases, off-resonance and transmit phase:
    1j F+[0] in the receiver's frame, (V, P) complex128."""
    p, m, z = _complex_start(t1.shape[0], states)
    z = -z
    first = _first_order(states)
    out = []
    for k in range(angle.shape[0]):
        e1 = torch.exp(-1e3 * wait[k] / t1)[:, None]
        turn = torch.polar(torch.exp(-1e3 * wait[k] / t2), -2 * math.pi * b0 * wait[k])[:, None]
        p, m, z = turn * p, turn.conj() * m, e1 * z + (1 - e1) * first
        p, m, z = _complex_step(p, m, z, angle[k] * b1, phase[k] + b1_phase)
        out.append(1j * p[:, 0] * torch.polar(torch.ones_like(phase[k]), -phase[k]))
        p, m = _complex_shift(p, m)
    return torch.stack(out, -1)


def _echoes(flip, esp, exc_phase, phase, t1, t2, b1, states):
    """F+[0] at each echo of a CPMG train in the receiver's frame, (V, P)."""
    V, dev = t1.shape[0], DEVICE
    angle = _played(flip).to(dev, torch.float64)
    excite = _played(torch.tensor([90.0])).to(dev, torch.float64)
    count = angle.shape[0]
    clock = [0.0]
    for j in range(count):
        echo = (j + 1) * (esp * 1e-3)
        clock += [1e6 * (echo - 0.5 * (esp * 1e-3)), 1e6 * echo]
    wait = (np.diff(np.array(clock)) * 1e-6).astype(np.float32).astype(np.float64)
    p, m, z = _complex_start(V, states)
    first = _first_order(states)
    exc = torch.full((V,), exc_phase, dtype=torch.float64, device=dev)
    ref = torch.full((V,), phase, dtype=torch.float64, device=dev)
    p, m, z = _complex_step(p, m, z, excite * b1, exc)

    def relax(p, m, z, dt):
        e1, e2 = torch.exp(-1e3 * dt / t1)[:, None], torch.exp(-1e3 * dt / t2)[:, None]
        return e2 * p, e2 * m, e1 * z + (1 - e1) * first

    out = []
    for j in range(count):
        p, m, z = relax(p, m, z, wait[2 * j])
        p, m = _complex_shift(p, m)
        p, m, z = _complex_step(p, m, z, angle[j] * b1, ref)
        p, m = _complex_shift(p, m)
        p, m, z = relax(p, m, z, wait[2 * j + 1])
        out.append(p[:, 0] * torch.polar(torch.ones_like(ref), -ref))
    return torch.stack(out, -1)


def _fse(flip, t1, t2, b1, states, esp=8.0, tr=3000.0):
    """``fse_sim`` of the ``train`` cases: the echoes with their recovery."""
    s = _echoes(flip, esp, float(np.float32(math.pi / 2)), 0.0, t1, t2, b1, states)
    rec = torch.exp(-(tr - esp * flip.numel()) / t1)[:, None]
    return s * (1 - rec) / (1 - rec * s)


def _pieces(voxels, per_voxel, most=1.6e10):
    """Voxel ranges whose working set stays below ``most`` bytes."""
    step = max(1, int(most / per_voxel))
    return [slice(a, min(a + step, voxels)) for a in range(0, voxels, step)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "map":
        return None  # where ten steps end is not a closed value
    s = _inputs(case, seed)
    if kind == "batch":
        parts = []
        for e in s["entries"]:
            t1, t2, b1 = (torch.from_numpy(e[k]).to(DEVICE, torch.float64) for k in ("t1", "t2", "b1"))
            turn = float(np.float32(math.pi / 2))
            parts.append(_echoes(torch.from_numpy(e["flip"]), e["esp"], turn, turn, t1, t2, b1,
                                 2 * len(e["flip"])).reshape(-1))
        return torch.cat(parts)
    if kind == "match":
        atoms = torch.nn.functional.normalize(s["atoms"].real.double(), dim=1)
        power = torch.linalg.vector_norm(s["atoms"].real.double(), dim=1)
        scores, densities = [], []
        for v in s["signal"].split(2048):
            norm = torch.linalg.vector_norm(v.to(torch.complex128), dim=1)[:, None]
            both = torch.hypot(v.real.double() @ atoms.mT, v.imag.double() @ atoms.mT)
            best, where = both.topk(case["top_k"], dim=1)
            scores.append(best / norm)
            densities.append(best / power[where])
        return dict(parameters=None, indices=None, scores=torch.cat(scores), scales=None,
                    densities=torch.cat(densities))
    t1, t2, b1 = (s[k].double() for k in ("t1", "t2", "b1"))
    V, P, S, names = case["voxels"], case["pulses"], case["states"], _names(case)
    if kind == "train":
        base = (t1, t2, b1)
        signal = _fse(s["flip"], *base, S)
        if not names:
            return signal
        cols = []
        for name in names:
            i = ("T1", "T2", "B1").index(name)
            cols.append(torch.func.jvp(
                lambda x, i=i: _fse(s["flip"], *base[:i], x, *base[i + 1:], S),
                (base[i],), (torch.ones_like(t1),))[1])
        return signal, torch.stack(cols, 1)
    stateful = [n for n in names if n != "M0"]
    if kind in ("signal", "jacobian"):
        angle, wait = _mrf_values(s["flip"], s["tr"])
        signal, jac = [], []
        for part in _pieces(V, (1 + len(stateful)) * (240.0 * S + 40.0 * P), 4e10):
            v = -_mrf(angle, wait, t1[part], t2[part], b1[part], S, stateful)
            signal.append(v[0])
            jac.append(torch.stack([v[0] if n == "M0" else v[1 + stateful.index(n)]
                                    for n in names], 1) if names else None)
        signal = torch.cat(signal)
        signal = torch.complex(signal, torch.zeros_like(signal))
        if not names:
            return signal
        jac = torch.cat(jac)
        return signal, torch.complex(jac, torch.zeros_like(jac))
    leaves = [s["flip"], s["tr"]]
    for x in leaves:
        x.requires_grad_(True)
    signals, jacs, voxel, shared = [], [], [], [0.0, 0.0]
    systems = 1 + len(stateful) if kind != "offaxis" else 4
    for part in _pieces(V, systems * 8.0 * S * P * 30, 4e10):
        local = [x[part].clone().requires_grad_(True) for x in (t1, t2)]
        angle, wait = _mrf_values(*leaves)
        seed = s["seed"][part].to(torch.complex128)
        if kind == "offaxis":
            b0 = s["b0"][part].double().requires_grad_(True)
            local.append(b0)
            phase = torch.deg2rad(s["phases"]).to(DEVICE, torch.float64)
            signal = _offaxis(angle, wait, phase, *local[:2], b1[part], b0,
                              s["b1_phase"][part].double(), S)
            loss = (seed.conj() * signal).real.sum()
        else:
            v = -_mrf(angle, wait, *local, b1[part], S, stateful)
            m0 = s["m0"][part].double()[:, None] if kind == "precision" else 1.0
            signal = m0 * v[0]
            loss = (seed.real * signal).sum()
        if kind == "precision":
            jac = torch.stack([v[0] if n == "M0" else m0 * v[1 + stateful.index(n)]
                               for n in names], 1)
            loss = loss + (s["seed_jac"][part].real.double() * jac).sum()
            jacs.append(torch.complex(jac.detach(), torch.zeros_like(jac)))
        grads = torch.autograd.grad(loss, [*leaves, *local])
        shared = [a + g.double() for a, g in zip(shared, grads[:2])]
        voxel.append(grads[2:])
        signal = signal.detach()
        signals.append(signal if signal.is_complex() else torch.complex(signal, torch.zeros_like(signal)))
        del loss, grads, signal
    out = [torch.cat(signals)]
    if kind == "precision":
        out.append(torch.cat(jacs))
    return (*out, *shared, *(torch.cat(x) for x in zip(*voxel)))
