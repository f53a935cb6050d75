"""The one-voxel-per-lane CPMG kernel (csrc/epg_echo.cu) against the FP64
oracle where it can go wrong: one to sixty-four echoes, truncation at odd and
even state counts down to one, ragged units; and which trains it takes."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.helpers import max_rel, packed_from_events

SIGNAL_TOL = 1e-5


def _events(echoes, esp=9.0, phase=90.0):
    from torchsim_gb300.sequence import fse_events

    rng = np.random.default_rng(echoes)
    return fse_events(rng.uniform(60, 180, echoes).astype(np.float32), esp, phases_deg=phase)


@pytest.mark.gpu
def test_echo_trains_against_the_oracle(cuda):
    from torchsim_gb300.batching import BatchEntry, SequenceBatch

    rng = np.random.default_rng(0)
    entries = []
    for echoes in (1, 2, 3, 5, 8, 9, 16, 17, 31, 32, 33, 63, 64, 65):
        for states in sorted({1, 2, 3, 4, 6, 7, 9, echoes // 2 + 1, echoes, echoes + 1, 2 * echoes}):
            v = int(rng.integers(1, 140))
            entries.append(BatchEntry(_events(echoes), states,
                                      rng.uniform(200, 3000, v).astype(np.float32),
                                      rng.uniform(10, 300, v).astype(np.float32),
                                      rng.uniform(0.6, 1.4, v).astype(np.float32),
                                      rng.uniform(0.5, 1.5, v).astype(np.float32)))
    batch = SequenceBatch(entries, cuda)
    assert [bool(x) for x in batch.echo] == [e.events.outputs <= 64 for e in entries]
    batch.out.fill_(float("nan"))
    batch.launch((8, 4, 4))
    torch.cuda.synchronize()
    for i, e in enumerate(entries):
        want = O.forward(packed_from_events(e.events, e.t1, e.t2, e.states, m0=e.m0, b1=e.b1), "f64")
        got = batch.signal(i).cpu().numpy()
        assert not got.real.any()
        assert max_rel(got.imag, want) <= SIGNAL_TOL, (e.events.outputs, e.states)


def test_which_trains_the_echo_kernel_takes():
    from torchsim_gb300 import _native
    from torchsim_gb300.batching import compile_ops
    from torchsim_gb300.sequence import mrf_events

    lib = _native.library()

    def takes(ops):
        return bool(lib.tsg_echo_train(ops.ctypes.data, len(ops)))

    for echoes, want in ((1, True), (64, True), (65, False)):
        assert takes(compile_ops(_events(echoes))) is want
    assert not takes(compile_ops(mrf_events(np.full(9, 30.0, np.float32), 8.0)))
    moved = compile_ops(_events(8))
    moved["dt"][5] *= 1.5
    assert not takes(moved)
    swapped = compile_ops(_events(8))
    swapped["record"][[4, 6]] = swapped["record"][[6, 4]]
    assert not takes(swapped)
