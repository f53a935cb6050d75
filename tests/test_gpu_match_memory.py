"""Scratch of a match whose last voxels alone share their atoms among many
candidate lists: the other voxels keep one list each. Results are those of the
voxels matched in smaller calls (each within 2e-6 of the FP64 scores)."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [1, 128, 129])
def test_lists_of_the_last_voxels(cuda, extra):
    from torchsim_gb300 import DictionaryMatcher, _native

    # Whole waves of 128 voxels to each pair of SMs, and a few more.
    pairs = torch.cuda.get_device_properties(cuda).multi_processor_count // 2
    V, A, P = 6 * pairs * 128 + extra, 65_600, 8
    gen = torch.Generator(device=cuda).manual_seed(extra)
    atoms = torch.randn((A, P), device=cuda, generator=gen).to(torch.complex64)
    signals = torch.randn((V, P), dtype=torch.complex64, device=cuda, generator=gen)
    matcher = DictionaryMatcher(dictionary=atoms, top_k=2)
    lib = _native.library()
    one_list = V * lib.tsg_match_candidates() * 8
    assert lib.tsg_match_lists(V, A, 8) > 8
    matcher.match(signals[:100])
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated(cuda)
    torch.cuda.reset_peak_memory_stats(cuda)
    got = matcher.match(signals)
    assert torch.cuda.max_memory_allocated(cuda) - before <= 3 * one_list
    for rows in (slice(0, 300), slice(V - extra - 200, V)):
        want = matcher.match(signals[rows])
        assert (got.scores[rows] - want.scores).abs().max() <= 4e-6
        assert (got.indices[rows] == want.indices).float().mean() >= 0.99
