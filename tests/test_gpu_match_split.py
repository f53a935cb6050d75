"""The matching screen where its work split can go wrong: dictionaries cut
into several lists per voxel, row pairs with one or no live row tile, query
tiles that stay resident and ones that stream, contractions off the tile's
width, chunks of voxels. FP32 rescoring is within 2e-6 of the FP64 scores (the
bound of the exhaustive-search test), so the best atom's FP64 score is within
twice that of the best there is."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(cuda, V, A, P, kind):
    gen = torch.Generator(device=cuda).manual_seed(V + A + P)
    real = torch.randn((A, P), device=cuda, generator=gen)
    zero = torch.zeros_like(real)
    if kind == "complex":
        atoms = torch.complex(real, torch.randn((A, P), device=cuda, generator=gen))
    else:
        atoms = torch.complex(real, zero) if kind == "real" else torch.complex(zero, real)
    truth = torch.randint(0, A, (V,), device=cuda, generator=gen)
    noise = torch.randn((V, P), dtype=torch.complex64, device=cuda, generator=gen)
    turn = torch.polar(torch.rand(V, device=cuda, generator=gen) + 0.5,
                       6.28 * torch.rand(V, device=cuda, generator=gen))
    return atoms, atoms[truth] * turn[:, None] + 0.3 * noise


@pytest.mark.parametrize("V,A,P,kind,chunk", [
    (1, 2100, 8, "real", 65536), (63, 20001, 40, "imaginary", 65536), (65, 9000, 513, "real", 65536),
    (129, 4097, 300, "complex", 65536), (1000, 30000, 100, "complex", 300),
    (10000, 2049, 64, "real", 65536), (9729, 2600, 72, "imaginary", 9729)])
def test_split_screens_find_the_best_atoms(cuda, V, A, P, kind, chunk):
    from torchsim_gb300 import DictionaryMatcher

    atoms, signals = _case(cuda, V, A, P, kind)
    table = torch.arange(2 * A, dtype=torch.float32).reshape(A, 2)
    res = DictionaryMatcher(dictionary=atoms, parameters=table, top_k=3,
                            query_chunk_size=chunk).match(signals)
    d = torch.nn.functional.normalize(atoms.to(torch.complex128), dim=1)
    for rows in torch.arange(V, device=cuda).split(2048):
        s = signals[rows].to(torch.complex128)
        scores = (torch.nn.functional.normalize(s, dim=1) @ d.mH).abs()
        best = scores.topk(3, dim=1).values
        found = torch.gather(scores, 1, res.indices[rows])
        assert (found - best).abs().max() <= 4e-6
        assert (res.scores[rows] - found).abs().max() <= 2e-6
        chosen = atoms[res.indices[rows]].to(torch.complex128)
        power = chosen.abs().square().sum(-1)
        scale = (chosen.conj() * s[:, None]).sum(-1) / power
        assert (res.scales[rows] - scale).abs().max() <= 1e-5 * scale.abs().max()
        density = found * torch.linalg.vector_norm(s, dim=1)[:, None] / power.sqrt()
        assert (res.densities[rows] - density).abs().max() <= 1e-5 * density.max()
    assert torch.equal(res.parameters.cpu(), table[res.indices.cpu()])
