"""The recorded-train sweep (csrc/epg_train.cuh) where it can go wrong: state
counts on and off its launch shapes' sizes, ragged voxel counts, trains around
its staging chunk and record runs, several trains, every column and output
layout. The general sweep of the same events (compiled unmerged, which gives
it an op per event) is the comparison; each is within the stated tolerance of
the oracle, so they are within twice that of each other."""

from __future__ import annotations

import ctypes
from dataclasses import replace

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.helpers import draw_tissue, max_rel, packed_from_events

pytestmark = pytest.mark.gpu
SIGNAL_TOL, JACOBIAN_TOL = 1e-5, 1e-4


def _events(pulses, TI=0.0, trains=1, inversion=True):
    from torchsim_gb300.sequence import mrf_events

    rng = np.random.default_rng(pulses)
    ev = mrf_events(rng.uniform(3, 60, pulses).astype(np.float32),
                    rng.uniform(6, 14, pulses).astype(np.float32), TI_ms=TI)
    if not inversion:
        ev = replace(ev, duration=ev.duration[:, 1:], kind=ev.kind[1:], flip=ev.flip[:, 1:],
                     phase=ev.phase[:, 1:], action=ev.action[1:], output_index=ev.output_index[1:])
    if trains > 1:
        scale = np.linspace(1.0, 1.4, trains, dtype=np.float32)[:, None]
        ev = replace(ev, duration=ev.duration * scale, flip=ev.flip * scale,
                     phase=np.repeat(ev.phase, trains, 0))
    return ev


def _maps(cuda, voxels, full=True):
    from torchsim_gb300 import engine

    t1, t2, b1 = draw_tissue(3, voxels)
    rng = np.random.default_rng(5)
    m0 = rng.uniform(0.5, 1.5, voxels).astype(np.float32)
    inv = rng.uniform(0.8, 1.0, voxels).astype(np.float32)
    return engine.tissue_maps(cuda, voxels, t1, t2, m0 if full else None, b1 if full else None,
                              inv if full else None)


@pytest.mark.parametrize("states,voxels,pulses", [
    (1, 5, 3), (2, 33, 1), (7, 1, 31), (10, 6, 30), (11, 13, 61), (13, 97, 64), (16, 8, 33),
    (20, 3, 960), (21, 40, 961), (27, 65, 119), (32, 31, 32), (40, 10, 1931), (64, 4, 90),
    (100, 3, 40), (128, 2, 35)])
@pytest.mark.parametrize("names", [(), ("T1", "T2"), ("M0", "B1", "T1"),
                                   ("inv_efficiency", "T2", "M0")])
def test_agrees_with_the_general_sweep(cuda, states, voxels, pulses, names):
    from torchsim_gb300 import engine
    from torchsim_gb300.sequence import Program

    ev = _events(pulses, TI=12.0 if states % 2 else 0.0)
    maps = _maps(cuda, voxels)
    train, general = Program(ev), Program(ev, unmerged=True)
    for planes in (False, True):
        if names:
            got = engine.forward_tangents(train, maps, states, names, planes=planes)
            want = engine.forward_tangents(general, maps, states, names, planes=planes)
            assert max_rel(got[1].cpu(), want[1].cpu()) <= 2 * JACOBIAN_TOL
            got, want = got[0], want[0]
        else:
            got = engine.forward(train, maps, states, planes=planes)
            want = engine.forward(general, maps, states, planes=planes)
        assert max_rel(got.cpu(), want.cpu()) <= 2 * SIGNAL_TOL


@pytest.mark.parametrize("inversion,trains,full", [(False, 1, True), (True, 3, True), (True, 1, False)])
def test_other_stream_forms(cuda, inversion, trains, full):
    from torchsim_gb300 import engine
    from torchsim_gb300.sequence import Program

    ev = _events(73, trains=trains, inversion=inversion)
    maps = _maps(cuda, 41, full)
    for names in (("T1", "T2"), ("T2", "B1")):
        got = engine.forward_tangents(Program(ev), maps, 18, names)
        want = engine.forward_tangents(Program(ev, unmerged=True), maps, 18, names)
        assert max_rel(got[0].cpu(), want[0].cpu()) <= 2 * SIGNAL_TOL
        assert max_rel(got[1].cpu(), want[1].cpu()) <= 2 * JACOBIAN_TOL
    _, alone = engine.forward_tangents(Program(ev), maps, 18, ("T2", "B1"), with_signal=False)
    assert torch.equal(alone, got[1])


@pytest.mark.parametrize("states", [6, 10, 13, 16, 20, 29, 32, 40])
def test_launch_shapes_give_the_same_bits(cuda, states):
    """A voxel's samples do not depend on how many voxels share its launch,
    hence not on the shape the launch rules pick for them."""
    from torchsim_gb300 import engine
    from torchsim_gb300.sequence import program_for

    ev = _events(100)
    program = program_for(ev)
    t1, t2, b1 = draw_tissue(9, 100000)
    rows = slice(0, 37)
    for names in ((), ("T1", "T2"), ("T1", "T2", "B1")):
        def run(n, names=names):
            maps = engine.tissue_maps(cuda, n, t1[:n], t2[:n], None, b1[:n], None)
            if names:
                return engine.forward_tangents(program, maps, states, names)
            return (engine.forward(program, maps, states),)

        alone = run(37)
        for n in (5000, 25000, 100000):
            for a, b in zip(alone, run(n)):
                assert torch.equal(a, b[rows]), (names, n)


@pytest.mark.parametrize("states,voxels", [(8, 70), (10, 3000), (10, 13000), (16, 3100), (20, 9000),
                                           (20, 25000), (27, 2100), (40, 30), (64, 20)])
def test_normal_equations(cuda, states, voxels):
    """The Gauss-Newton sums of the first voxels against their definition over
    the FP64 oracle's signal and derivatives: FP32 signal and tangent errors
    (1e-5, 1e-4 of their maximum) enter each product once."""
    from torchsim_gb300 import _native
    from torchsim_gb300.sequence import program_for

    ev = _events(150)
    program = program_for(ev)
    maps = _maps(cuda, voxels)
    maps.inv = None
    gen = torch.Generator(device=cuda).manual_seed(1)
    y = torch.randn((voxels, 150), dtype=torch.complex64, device=cuda, generator=gen) * 0.1
    rows = torch.arange(voxels, device=cuda).flip(0).contiguous()
    out = torch.empty((voxels, 10), dtype=torch.float64, device=cuda)
    tissue = maps.struct()
    _native.check(_native.library().tsg_gn_evaluate(
        program.handle, ctypes.byref(tissue), voxels, states, y.data_ptr(), rows.data_ptr(),
        out.data_ptr(), None, torch.cuda.current_stream().cuda_stream))
    n = 12
    host = {k: getattr(maps, k)[:n].cpu().numpy() for k in ("t1", "t2", "m0", "b1")}
    p = packed_from_events(ev, host["t1"], host["t2"], states, m0=host["m0"], b1=host["b1"])
    v = O.forward(p, "f64")
    j = np.stack([O.tangent(p, "f64", t1_ms=1.0), O.tangent(p, "f64", t2_ms=1.0),
                  v / host["m0"][:, None].astype(np.float64)])
    meas = y[rows[:n]].cpu().numpy().astype(np.complex128)
    res = v + meas.real
    cols = [(res**2 + meas.imag**2)]
    cols += [j[a] * j[b] for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))]
    cols += [j[a] * res for a in range(3)]
    got = out[:n].cpu().numpy()
    for k, c in enumerate(cols):
        scale = np.abs(c).sum(1).max()
        assert np.abs(got[:, k] - c.sum(1)).max() <= 3 * JACOBIAN_TOL * scale, k
