"""The CPMG kernel of the complex path (csrc/epg_cpmg.cu) where it can go
wrong: state and echo counts around its shapes' sizes, its sample rows and its
staging chunk, ragged voxel counts, several trains, varied intervals, receiver
phases and frames, every column; and streams next to those it takes. The
general complex kernel (a requested shape selects it) is the comparison; each
is within the stated tolerance of the oracle, so they are within twice that of
each other."""

from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest
import torch

from tests.helpers import draw_tissue, max_rel

pytestmark = pytest.mark.gpu
SIGNAL_TOL, JACOBIAN_TOL = 1e-5, 1e-4
GENERAL = (32, 4, 4)


def _events(echoes, phase=0.0, exc=90.0, trains=1, esp=8.0):
    from torchsim_gb300.sequence import fse_events

    rng = np.random.default_rng(echoes)
    ev = fse_events(rng.uniform(60, 180, echoes).astype(np.float32), esp, phases_deg=phase,
                    exc_phase=exc, exc_flip=85.0)
    if trains > 1:
        scale = np.linspace(1.0, 1.4, trains, dtype=np.float32)[:, None]
        ev = replace(ev, duration=ev.duration * scale, flip=ev.flip * scale,
                     phase=np.repeat(ev.phase, trains, 0))
    return ev


def _check(cuda, ev, states, voxels, names, full=True, offaxis=None):
    from torchsim_gb300 import engine
    from torchsim_gb300.sequence import Program

    t1, t2, b1 = draw_tissue(3, voxels)
    m0 = np.random.default_rng(5).uniform(0.5, 1.5, voxels).astype(np.float32)
    maps = engine.tissue_maps(cuda, voxels, t1, t2, m0 if full else None, b1 if full else None, None)
    off, keep = (engine.offaxis_maps(cuda, voxels, offaxis, None) if offaxis is not None
                 else (None, None))
    prog = Program(ev, phased=True)
    if names:
        got = engine.forward_tangents_complex(prog, maps, states, names, off)
        want = engine.forward_tangents_complex(prog, maps, states, names, off, launch=GENERAL)
        for c, name in enumerate(names):
            assert max_rel(got[1][:, c].cpu(), want[1][:, c].cpu()) <= 2 * JACOBIAN_TOL, name
        got, want = got[0], want[0]
    else:
        got = engine.forward_complex(prog, maps, states, off)
        want = engine.forward_complex(prog, maps, states, off, launch=GENERAL)
    assert float(want.abs().max()) > 1e-3 or states < 2
    assert max_rel(got.cpu(), want.cpu()) <= 2 * SIGNAL_TOL


@pytest.mark.parametrize("echoes,states,voxels", [
    (1, 1, 5), (1, 2, 33), (2, 3, 1), (7, 8, 129), (8, 9, 31), (9, 12, 40), (16, 13, 16),
    (17, 16, 65), (32, 17, 10), (33, 24, 100), (40, 25, 7), (48, 32, 63), (49, 33, 64), (50, 48, 9),
    (64, 49, 5), (64, 64, 33), (64, 128, 8), (65, 128, 3), (65, 65, 3), (66, 66, 2), (255, 10, 20),
    (257, 20, 70), (513, 63, 4)])
@pytest.mark.parametrize("names", [(), ("T1", "T2"), ("M0", "B1", "T1")])
def test_agrees_with_the_general_kernel(cuda, echoes, states, voxels, names):
    _check(cuda, _events(echoes), states, voxels, names)


@pytest.mark.parametrize("names", [(), ("T2", "B1")])
def test_other_stream_forms(cuda, names):
    rng = np.random.default_rng(1)
    ev = _events(40, trains=3)
    _check(cuda, ev, 30, 21, names)
    _check(cuda, replace(ev, duration=ev.duration * rng.uniform(0.0, 2.0, ev.duration.shape).round(2)
                         .astype(np.float32)), 30, 21, names)
    receive = ev.phase.copy()
    receive[:, 2::3] = rng.uniform(-4, 4, receive[:, 2::3].shape)
    _check(cuda, replace(ev, phase=receive), 30, 21, names, full=False)
    for phase, exc in ((90.0, 0.0), (37.0, 127.0), (-180.0, 90.0), (270.0, 0.0)):
        _check(cuda, _events(20, phase, exc), 20, 9, names)
    # Streams that the split does not cover, and a B1phase map.
    _check(cuda, _events(20, 30.0, 90.0), 20, 9, names)
    _check(cuda, _events(20, np.linspace(0, 90, 20).astype(np.float32), 90.0), 20, 9, names)
    _check(cuda, _events(20), 20, 9, names, offaxis=np.full(9, 0.3, np.float32))
