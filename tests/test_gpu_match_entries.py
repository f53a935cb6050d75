"""The screen and the rescoring as entries of their own (tsg_match_screen,
tsg_match_rescore: one part, never split), on query rows that stay resident and
that stream, partial row tiles and contractions off the tile's width, against
the FP64 scores: rescored scores within 2e-6 of them, so the best atom's score
is within twice that of the best there is."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("voxels,atoms,samples,parts", [
    (1, 3, 8, 1), (64, 65, 20, 2), (129, 500, 64, 2), (300, 4097, 100, 1), (1000, 700, 300, 2)])
def test_screen_and_rescore(cuda, voxels, atoms, samples, parts):
    from torchsim_gb300 import _native

    lib = _native.library()
    stream = torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device=cuda).manual_seed(voxels + atoms)
    d = torch.nn.functional.normalize(torch.randn((atoms, samples), device=cuda, generator=gen), dim=1)
    signals = torch.randn((voxels, samples), dtype=torch.complex64, device=cuda, generator=gen)
    s = signals / torch.linalg.vector_norm(signals, dim=1, keepdim=True)
    scale, k = samples**0.5, -(-samples // 8) * 8

    def padded(x):
        return torch.nn.functional.pad(x, (0, k - samples))

    # Atoms as fp16 values, and their remainders as further columns; the queries
    # once for each, two rows per voxel.
    scaled = padded(d * scale)
    hi = scaled.to(torch.float16)
    rows = torch.cat([hi, (scaled - hi.float()).to(torch.float16)][:parts], dim=1)
    i = torch.arange(atoms, device=cuda)
    at = (i & 1) | (((i >> 1) & 1) << 5) | (((i >> 2) & 15) << 1) | (i & ~63)
    stored = torch.zeros((int(lib.tsg_match_screen_rows(atoms)), parts * k), dtype=torch.float16,
                         device=cuda)
    stored[at] = rows
    query = padded(torch.stack((s.real, s.imag), 1).reshape(2 * voxels, samples) * scale)
    query = query.to(torch.float16).repeat(1, parts)

    m = int(lib.tsg_match_candidates())
    cand_scores = torch.empty((voxels, m), dtype=torch.float32, device=cuda)
    cand = torch.empty((voxels, m), dtype=torch.int32, device=cuda)
    error = torch.zeros(1, dtype=torch.int32, device=cuda)
    _native.check(lib.tsg_match_screen(query.data_ptr(), 2 * voxels, stored.data_ptr(), atoms,
                                       parts * k, cand_scores.data_ptr(), cand.data_ptr(),
                                       error.data_ptr(), stream))
    top = min(3, atoms)
    scores = torch.empty((voxels, top), dtype=torch.float32, device=cuda)
    index = torch.empty((voxels, top), dtype=torch.int64, device=cuda)
    exact = d.to(torch.complex64)
    _native.check(lib.tsg_match_rescore(s.data_ptr(), voxels, exact.data_ptr(), atoms, samples,
                                        cand.data_ptr(), top, scores.data_ptr(), index.data_ptr(),
                                        stream))
    assert int(error.item()) == 0
    want = (s.to(torch.complex128) @ d.to(torch.complex128).mT).abs()
    found = torch.gather(want, 1, index)
    assert (scores - found).abs().max() <= 2e-6
    assert (found - want.topk(top, dim=1).values).abs().max() <= 4e-6
