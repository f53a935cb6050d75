"""The persistent batched launch on sequences that the echo kernel leaves to it:
CPMG trains of more than 64 echoes (the kernel's echo loop), of varied spacing,
and MRF trains (its op loop), with and without echo-kernel trains beside them, at
every launch shape of the batched tests, against the FP64 oracle."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.helpers import max_rel, packed_from_events

pytestmark = pytest.mark.gpu
SHAPES = [(2, 2, 2), (4, 4, 4), (8, 8, 2), (4, 1, 16), (16, 2, 8)]


def _entries(most_states, beside):
    from torchsim_gb300.batching import BatchEntry
    from torchsim_gb300.sequence import fse_events, mrf_events

    rng = np.random.default_rng(most_states)

    def entry(events, states, voxels):
        return BatchEntry(events, min(states, most_states),
                          rng.uniform(300, 3000, voxels).astype(np.float32),
                          rng.uniform(10, 300, voxels).astype(np.float32),
                          rng.uniform(0.7, 1.3, voxels).astype(np.float32),
                          rng.uniform(0.5, 1.5, voxels).astype(np.float32))

    def train(echoes):
        return fse_events(rng.uniform(100, 180, echoes).astype(np.float32), 9.0, phases_deg=90.0)

    def varied(echoes):
        ev = train(echoes)
        ev.duration *= rng.uniform(0.8, 1.2, ev.duration.shape).astype(np.float32)
        return ev

    entries = [entry(train(65), 130, 1), entry(train(80), 160, 77), entry(train(100), 200, 333),
               entry(train(100), 33, 64), entry(varied(12), 24, 100), entry(varied(70), 100, 41),
               entry(mrf_events(rng.uniform(5, 70, 90).astype(np.float32), 10.0, TI_ms=20.0), 33, 65)]
    if beside:
        entries[2:2] = [entry(train(9), 18, 77), entry(train(64), 128, 130)]
    return entries


def _check(batch):
    for i, e in enumerate(batch.entries):
        want = O.forward(packed_from_events(e.events, e.t1, e.t2, e.states, m0=e.m0, b1=e.b1), "f64")
        got = batch.signal(i).cpu().numpy()
        assert not got.real.any()
        assert max_rel(got.imag, want) <= 1e-5, i


@pytest.mark.parametrize("beside", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_shapes(cuda, shape, beside):
    from torchsim_gb300.batching import SequenceBatch

    entries = _entries(32 * shape[0] if shape[0] < 8 else 256, beside)
    batch = SequenceBatch(entries, cuda)
    assert int((~batch.echo).sum()) == 7 and bool(batch.echo.any()) is beside
    batch.out.fill_(float("nan"))
    batch.launch(shape)
    torch.cuda.synchronize()
    _check(batch)
    for i in (1, 2, len(entries) - 1):
        alone = SequenceBatch([entries[i]], cuda)
        alone.launch(shape)
        torch.cuda.synchronize()
        assert torch.equal(alone.signal(0), batch.signal(i)), i


@pytest.mark.parametrize("beside", [False, True])
def test_autotuner_times_the_persistent_launch(cuda, tmp_path, monkeypatch, beside):
    from torchsim_gb300 import autotune
    from torchsim_gb300.batching import SequenceBatch

    monkeypatch.setenv("TORCHSIM_GB300_CACHE", str(tmp_path / "tuning.json"))
    monkeypatch.setattr(autotune, "_memory", {})
    batch = SequenceBatch(_entries(256, beside), cuda)
    shape, timings = batch.tune(use_cache=False)
    assert shape in batch.candidates() and len(timings) == len(batch.candidates()) > 1
    assert timings[str(shape)] == min(timings.values())
    batch.out.fill_(float("nan"))
    batch.run()
    torch.cuda.synchronize()
    _check(batch)
    assert batch.tune() == (shape, {})
