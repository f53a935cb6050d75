"""Relaxation times of zero, which the Python simulators clamp but the C entries
take: an op that waits takes all of the magnetisation with it, an op that does
not wait none. The recorded-train sweep against the general sweep of the same
program (asked for by a launch shape that only it has): finite wherever that is,
and within twice the 1e-5 (signal) and 1e-4 (columns) that each is held to
against the oracle."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
V = 70


def _maps(cuda):
    from torchsim_gb300 import engine

    t1 = torch.linspace(200, 2000, V, device=cuda)
    t2 = torch.linspace(20, 150, V, device=cuda)
    t1[3] = t2[11] = t1[40] = t2[40] = 0.0
    t1[5], t2[6], t2[8] = float("inf"), float("inf"), float("nan")
    return engine.TissueMaps(t1, t2, None, torch.linspace(0.8, 1.2, V, device=cuda), None)


def _compare(got, want, bound):
    fine = torch.isfinite(torch.view_as_real(want)).all(-1)
    assert bool(torch.isfinite(torch.view_as_real(got)).all(-1)[fine].all())
    assert (got - want)[fine].abs().max() <= bound * want[fine].abs().max()
    return fine


@pytest.mark.parametrize("lanes,orders", [(1, 10), (5, 2), (10, 2)])
@pytest.mark.parametrize("names", [(), ("T1", "T2")])
@pytest.mark.parametrize("pause", [9.0, 0.0])
def test_recorded_trains(cuda, lanes, orders, names, pause):
    from torchsim_gb300 import engine
    from torchsim_gb300.sequence import Program, mrf_events

    # (A train without an inversion time: its first pulse waits for nothing.)
    rng = np.random.default_rng(1)
    tr = np.full(40, 9.0, np.float32)
    tr[17] = pause
    program = Program(mrf_events(rng.uniform(5, 60, 40).astype(np.float32), tr))
    maps = _maps(cuda)

    def run(warps):
        shape = (lanes, orders, warps)
        if names:
            return engine.forward_tangents(program, maps, 10, names, launch=shape)
        return (engine.forward(program, maps, 10, launch=shape),)

    # Blocks of eight warps are the general sweep's alone.
    for got, want, bound in zip(run(4), run(8), (2e-5, 2e-4)):
        fine = _compare(got, want, bound)
        if got.ndim == 2:
            assert bool(fine[[3, 11, 40]].all()) and not bool(fine[8, 1:].any())
            assert not bool(torch.isfinite(got[8, 1:].real).any())
