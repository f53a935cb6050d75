"""Batches of few CPMG trains run with the orders over lanes, larger ones with
two voxels per lane: both give the same bits, over truncated and whole trains,
ragged units and angles beyond the paired sine's range (which the oracle tests
of small batches then vouch for). And a small batch takes no longer than on the
persistent kernel, which has the trains it could otherwise run on."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _entry(echoes, states, voxels, rng, b1=(0.6, 1.4), flips=None):
    from torchsim_gb300.batching import BatchEntry
    from torchsim_gb300.sequence import fse_events

    flips = rng.uniform(60, 180, echoes) if flips is None else flips
    return BatchEntry(fse_events(flips.astype(np.float32), 9.0, phases_deg=90.0), states,
                      rng.uniform(200, 3000, voxels).astype(np.float32),
                      rng.uniform(10, 300, voxels).astype(np.float32),
                      rng.uniform(*b1, voxels).astype(np.float32),
                      rng.uniform(0.5, 1.5, voxels).astype(np.float32))


def _entries():
    rng = np.random.default_rng(3)
    entries = []
    for echoes in (1, 2, 3, 4, 5, 7, 8, 9, 16, 31, 32, 33, 63, 64):
        for states in sorted({1, 2, 3, 7, 8, 9, 17, echoes // 2 + 1, echoes, 2 * echoes}):
            entries.append(_entry(echoes, states, int(rng.integers(1, 64)), rng))
    entries.append(_entry(20, 40, 135, rng))
    flips = np.array([0.0, 45.0, -0.7, 180.0, 4e4, 58680.0, 1e6, 120.0, 90.0])
    entries.append(_entry(9, 18, 70, rng, flips=flips))
    entries.append(_entry(20, 40, 70, rng, b1=(900.0, 1200.0)))
    for e, at in ((entries[-1], 5), (entries[-3], 9)):
        e.b1[at] = e.t1[at + 3] = e.m0[at + 4] = np.nan
    return entries


def test_both_kernels_give_the_same_bits(cuda):
    from torchsim_gb300.batching import SequenceBatch

    entries = _entries()
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    rest = _entry(4, 8, 2 * sms * 64, np.random.default_rng(0))
    few, many = SequenceBatch(entries, cuda), SequenceBatch([*entries, rest], cuda)
    assert few.echo.all() and many.echo.all()
    assert few._echo_plan()[2] <= 2 * sms < many._echo_plan()[2]
    for batch in (few, many):
        batch.out.fill_(7.0)
        batch.launch((4, 4, 4))
    torch.cuda.synchronize()
    for i in range(len(entries)):
        a, b = few.signal(i), many.signal(i)
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(), b.nan_to_num()), i


@pytest.mark.parametrize("states", [128, 20])
def test_a_small_batch_is_no_slower_than_the_persistent_kernel(cuda, tmp_path, monkeypatch, states):
    from torchsim_gb300 import autotune
    from torchsim_gb300.batching import SequenceBatch

    monkeypatch.setenv("TORCHSIM_GB300_CACHE", str(tmp_path / "tuning.json"))
    monkeypatch.setattr(autotune, "_memory", {})
    entries = [_entry(64, states, 64, np.random.default_rng(1))]

    def best_us(echo):
        batch = SequenceBatch(entries, cuda)
        batch.echo[:] = echo
        batch.tune(use_cache=False)
        batch.capture()
        times = []
        for _ in range(8):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            begin.record()
            for _ in range(50):
                batch.run()
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end) / 50 * 1e3)
        return min(times)

    # 16 us against 22 (128 states) and 16 (20); 33 and 31 with two voxels per lane.
    assert best_us(True) <= 1.25 * best_us(False)
