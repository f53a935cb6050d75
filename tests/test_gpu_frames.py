"""The complex gradient sweeps (csrc/epg_complex_adjoint.cu), whose states are
held in the frame of the last pulse, on streams where a frame can be lost:
samples before the first pulse, several to a pulse and none, pulses back to back
without an interval between them, inversions, spoiling and shifts anywhere, runs
without a pulse longer than a warp, more ops than one staging chunk, several
trains; at state counts on the shapes where the reverse holds twice the
forward's orders per lane and on those where it does not. Against the FP64
oracle, at the tolerances of the complex gradient tests."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.helpers import draw_tissue, max_rel

pytestmark = pytest.mark.gpu
SIGNAL_TOL, GRAD_TOL = 1e-5, 1e-4


def _stream(events, trains, seed):
    from torchsim_gb300 import sequence as S

    rng = np.random.default_rng(seed)
    kind = rng.choice([S.RF, S.ADC, 0], events, p=[0.45, 0.45, 0.1]).astype(np.int32)
    kind[:3] = S.ADC
    if events > 500:
        kind[200:280] = S.ADC  # a long readout
    action = np.zeros(events, np.uint8)
    adc = kind == S.ADC
    action[adc] = S.RECORD
    action[rng.random(events) < 0.5] |= S.SHIFT_AFTER
    action[rng.random(events) < 0.02] |= S.SPOIL_AFTER
    inversion = (kind == S.RF) & (rng.random(events) < 0.05)
    action[inversion] |= S.INVERSION
    output = np.full(events, -1, np.int32)
    output[adc] = np.arange(adc.sum())
    shape = (trains, events)
    duration = rng.uniform(1e-3, 8e-3, shape) * (rng.random(events) < 0.7)
    return S.PackedEvents(
        duration=duration.astype(np.float32), kind=kind,
        flip=(rng.uniform(0.1, 1.5, shape) * (kind == S.RF)).astype(np.float32),
        phase=rng.uniform(-7, 7, shape).astype(np.float32), action=action, output_index=output,
        time_us=np.zeros(int(adc.sum()), np.float32), echo=np.zeros(int(adc.sum()), bool))


@pytest.mark.parametrize("events,states,trains,voxels", [
    (12, 4, 1, 33), (60, 10, 2, 7), (90, 20, 1, 41), (90, 16, 3, 5), (70, 33, 1, 9), (40, 64, 1, 3),
    (33, 8, 1, 129), (2400, 20, 1, 6)])
def test_frames(cuda, events, states, trains, voxels):
    from torchsim_gb300 import engine
    from torchsim_gb300.sequence import Program

    ev = _stream(events, trains, events + states)
    rng = np.random.default_rng(states)
    t1, t2, b1 = draw_tissue(18, voxels)
    m0 = rng.uniform(0.5, 1.5, voxels).astype(np.float32)
    b0 = rng.uniform(-40, 40, voxels).astype(np.float32)
    b1p = rng.uniform(-0.5, 0.5, voxels).astype(np.float32)
    inv = rng.uniform(0.8, 1.0, voxels).astype(np.float32)
    prog = Program(ev, phased=True)
    tissue = engine.tissue_maps(cuda, voxels, t1, t2, m0, b1, inv)
    off, keep = engine.offaxis_maps(cuda, voxels, b1p, b0)
    sig, traj = engine.forward_complex_trajectory(prog, tissue, states, off)
    p = O.Packed(t1, t2, ev.duration, ev.kind, ev.flip, ev.action, ev.output_index, states, m0=m0,
                 b1=b1, inversion=inv)
    p.phase_rad, p.b1_phase_rad, p.b0_hz = ev.phase, b1p, b0
    ref = O.forward_complex(p, "f64")
    assert max_rel(sig.cpu().numpy().reshape(ref.shape), 1j * ref) <= SIGNAL_TOL
    seed = (rng.standard_normal(sig.shape) + 1j * rng.standard_normal(sig.shape)).astype(np.complex64)
    grads = {n: torch.zeros(voxels, device=cuda) for n in engine.COMPLEX_GRAD_NAMES[:7]}
    for n in engine.COMPLEX_GRAD_NAMES[7:]:
        grads[n] = torch.zeros((trains, ev.events), device=cuda)
    engine.adjoint_complex(prog, tissue, states, torch.from_numpy(seed).to(cuda), traj, grads, off)
    want = O.adjoint_complex(p, seed.reshape(ref.shape), "f64")
    for name in engine.COMPLEX_GRAD_NAMES:
        got = grads[name].cpu().numpy().reshape(want[name].shape)
        ref_g = want[name]
        if name == "duration_s":
            # Zero durations are folded away on the merged program.
            formed = np.broadcast_to(ev.duration != 0, ev.duration.shape).reshape(want[name].shape)
            got, ref_g = got[formed], ref_g[formed]
        assert max_rel(got, ref_g) <= GRAD_TOL, name
