"""The autotuner's cache never hands a launch shape to work it was not measured
for: a batch's shape goes by the sequences of the persistent launch, and a cached
shape that is no candidate is measured anew. (Launches are planned, not run.)"""

from __future__ import annotations

import numpy as np
import pytest
import torch


@pytest.fixture
def planned(monkeypatch, tmp_path):
    """The autotuner without a GPU: a private cache, and candidates that are run
    and then count as the slower the more orders a lane holds."""
    from torchsim_gb300 import autotune

    monkeypatch.setenv("TORCHSIM_GB300_CACHE", str(tmp_path / "tuning.json"))
    monkeypatch.setattr(autotune, "_memory", {})

    def time_ms(fn, *_):
        fn()
        return 1.0 + fn.__defaults__[0][0]

    monkeypatch.setattr(autotune, "time_ms", time_ms)
    return autotune


def _batch(echoes, voxels=64):
    from torchsim_gb300.batching import BatchEntry, SequenceBatch
    from torchsim_gb300.sequence import fse_events

    tissue = np.full(voxels, 100.0, np.float32)
    batch = SequenceBatch([BatchEntry(fse_events(np.full(e, 150.0, np.float32), 9.0, phases_deg=90.0),
                                      s, tissue, tissue) for e, s in echoes], torch.device("cpu"))
    batch.launch = lambda shape: batch._plan(*shape[:2])
    return batch


def test_batches_of_one_size_and_other_sequences(planned):
    # Three sequences of the same most states and updates: echo trains alone,
    # then with a 70-echo train (the persistent launch) that holds the most
    # states, on no fewer than four orders per lane.
    alone = _batch([(60, 128), (60, 128), (32, 96)])
    mixed = _batch([(70, 128), (50, 128), (32, 96)])
    assert alone.echo.all() and list(mixed.echo) == [False, True, True]
    assert alone.updates() // 10**6 == mixed.updates() // 10**6
    for batch in (alone, mixed, _batch([(64, 128), (56, 128), (32, 96)])):
        shape, _ = batch.tune()
        assert shape in batch.candidates()
        batch.launch(shape)
    assert mixed.tune()[0][0] == 4 and mixed.tune()[1] == {}


def test_a_cached_shape_that_is_no_candidate(planned):
    def run(c):
        if c[0] > 8:
            raise ValueError("not a shape of this kernel")

    assert planned.tune("key", [(16, 2, 2), (4, 2, 2), (8, 2, 2)], run)[0] == (4, 2, 2)
    assert planned.tune("key", [(8, 2, 2)], run)[0] == (8, 2, 2)
    planned._memory.clear()
    assert planned.tune("key", [(4, 2, 2)], run) == ((4, 2, 2), {"(4, 2, 2)": 5.0})
    assert planned.tune("key", iter([(4, 2, 2)]), run) == ((4, 2, 2), {})
