"""The second-order sweeps (csrc/epg_second.cuh) on streams of every op form:
odd and even op counts, samples before the first pulse, several to a pulse and
none for longer than a warp, inversions, spoiling and shifts anywhere, more ops
than one staging chunk, several trains, records in no order; at state counts on
every kind of launch shape (records stored in rows or one by one). Against the
FP64 oracle, at the tolerances of the second-order tests."""

from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.helpers import draw_tissue, max_rel
from tests.test_gpu_frames import _stream

pytestmark = pytest.mark.gpu
SIGNAL_TOL, GRAD_TOL = 1e-5, 1e-4
PER_VOXEL = ("t1_ms", "t2_ms", "m0", "b1")


@pytest.mark.parametrize("events,states,trains,voxels,shuffled", [
    (11, 2, 1, 33, False), (12, 4, 1, 129, True), (13, 4, 2, 5, False), (60, 10, 2, 7, True),
    (61, 10, 1, 40, False), (90, 20, 1, 41, True), (91, 16, 3, 5, False), (70, 33, 1, 9, True),
    (41, 64, 1, 3, False), (2400, 20, 1, 6, False)])
@pytest.mark.parametrize("names", [("T1",), ("T2", "B1"), ("T1", "T2", "B1")])
def test_streams(cuda, events, states, trains, voxels, shuffled, names):
    from torchsim_gb300 import engine
    from torchsim_gb300.sequence import Program

    rng = np.random.default_rng(states + events)
    ev = replace(_stream(events, trains, events + states), phase=np.zeros((trains, events), np.float32))
    if shuffled:
        order = ev.output_index.copy()
        order[order >= 0] = rng.permutation(ev.outputs)
        ev = replace(ev, output_index=order)
    t1, t2, b1 = draw_tissue(18, voxels)
    m0 = rng.uniform(0.5, 1.5, voxels).astype(np.float32)
    prog = Program(ev)
    tissue = engine.tissue_maps(cuda, voxels, t1, t2, m0, b1, None)
    p = O.Packed(t1, t2, ev.duration, ev.kind, ev.flip, ev.action, ev.output_index, states, m0=m0,
                 b1=b1)
    key = {"T1": "t1_ms", "T2": "t2_ms", "B1": "b1"}
    shape = (trains, voxels, ev.outputs)
    want_sig = O.forward(p, "f64").reshape(shape)
    s0 = rng.standard_normal(shape).astype(np.float32)
    sk = rng.standard_normal((trains, voxels, len(names), ev.outputs)).astype(np.float32)
    want = O.adjoint(p, s0.reshape(want_sig.shape) if trains > 1 else s0[0], "f64")
    tangents, values = [], []
    for k, n in enumerate(names):
        tangents.append(O.tangent(p, "f64", **{key[n]: 1.0}).reshape(shape))
        v, c = O.second(p, sk[:, :, k] if trains > 1 else sk[0, :, k], "f64", **{key[n]: 1.0})
        values.append(v)
        want = {g: want[g] + c[g] for g in want}
    up = lambda x: torch.from_numpy((-x).reshape(-1, *x.shape[2:]).astype(np.complex64)).to(cuda)
    ones = torch.ones(voxels, device=cuda)
    for design in (False, True):
        if design:
            mask = sum(engine.DESIGN_BITS[n] for n in names)
            sig, jac, traj = engine.design_forward(prog, tissue, states, mask)
        else:
            directions = [{engine.DIRECTION_OF[n]: ones} for n in names]
            sig, jac, traj, ws = engine.second_forward(prog, tissue, states, directions)
        assert max_rel(sig.real.cpu().numpy().reshape(shape), -want_sig) <= SIGNAL_TOL
        for k, n in enumerate(names):
            assert max_rel(jac[:, k].real.cpu().numpy().reshape(shape), -tangents[k]) <= GRAD_TOL, n
        curvature = {n: torch.zeros(voxels, device=cuda) for n in PER_VOXEL}
        for n in ("flip_rad", "duration_s"):
            curvature[n] = torch.zeros((trains, events), device=cuda)
        if design:
            engine.design_reverse(prog, tissue, states, mask, up(sk), traj, seed_signal=up(s0),
                                  curvature=curvature)
        else:
            got = [{n: torch.zeros(voxels, device=cuda) for n in PER_VOXEL} for _ in names]
            engine.second_reverse(prog, tissue, states, directions, up(sk), traj, ws,
                                  seed_signal=up(s0), curvature=curvature, values=got)
            for k, n in enumerate(names):
                for g in PER_VOXEL:
                    assert max_rel(got[k][g].cpu().numpy(), values[k][g]) <= GRAD_TOL, (n, g)
        # Events of zero duration fold into the op before them on the merged
        # program.
        formed = (ev.duration != 0).reshape(want["duration_s"].shape)
        for g in (*PER_VOXEL, "flip_rad", "duration_s"):
            a, b = curvature[g].cpu().numpy().reshape(want[g].shape), want[g]
            if g == "duration_s":
                a, b = a[formed], b[formed]
            assert max_rel(a, b) <= GRAD_TOL, (design, g)
