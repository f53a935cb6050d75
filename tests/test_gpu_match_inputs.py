"""Matching with tensors that do not lie in memory as the kernels read them:
dictionaries, signals and parameter tables as transposed, sliced and conjugated
views, against the same values in plain tensors (equal, as the kernels then read
the same bits) and against FP64 scales."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
A, P, V = 700, 24, 130


def _draw(cuda, *shape):
    gen = torch.Generator(device=cuda).manual_seed(sum(shape))
    return torch.randn(shape, dtype=torch.complex64, device=cuda, generator=gen)


def _forms(x):
    """The values of ``x`` (rows, columns) as views of other layouts."""
    rows, columns = x.shape
    wide = x.new_zeros((rows, 2 * columns + 1))
    wide[:, 1::2] = x
    tall = x.new_zeros((2 * rows, columns))
    tall[::2] = x
    forms = {"plain": x.contiguous(), "transposed": x.mT.contiguous().mT, "columns": wide[:, 1::2],
             "rows": tall[::2]}
    if x.is_complex():
        forms["conjugated"] = x.conj().resolve_conj().conj()
        forms["adjoint"] = x.mH.resolve_conj().contiguous().mH
        assert forms["conjugated"].is_conj() and forms["adjoint"].is_conj()
    else:
        forms["negated"] = torch.complex(torch.zeros_like(x), -x).conj().imag
        assert forms["negated"].is_neg()
    for form in forms.values():
        assert torch.equal(form, x)
    return forms


def _check(got, want, atoms, signals):
    for name in ("indices", "scores", "scales", "densities", "parameters"):
        assert torch.equal(getattr(got, name), getattr(want, name)), name
    d = atoms.to(torch.complex128)[got.indices]
    scale = (d.conj() * signals.to(torch.complex128)[:, None]).sum(-1) / d.abs().square().sum(-1)
    assert (got.scales - scale).abs().max() <= 1e-5 * scale.abs().max()


@pytest.mark.parametrize("form", ["transposed", "columns", "rows", "conjugated", "adjoint"])
@pytest.mark.parametrize("which", ["dictionary", "signals"])
def test_complex_views(cuda, which, form):
    from torchsim_gb300 import DictionaryMatcher

    atoms = _draw(cuda, A, P)
    signals = atoms[::5][:V] * _draw(cuda, V, 1) + 0.1 * _draw(cuda, V, P)
    table = torch.arange(2.0 * A, device=cuda).reshape(A, 2)
    want = DictionaryMatcher(dictionary=atoms, parameters=table, top_k=2).match(signals)
    d = _forms(atoms)[form] if which == "dictionary" else atoms
    s = _forms(signals)[form] if which == "signals" else signals
    got = DictionaryMatcher(dictionary=d, parameters=table, top_k=2).match(s)
    _check(got, want, atoms, signals)


@pytest.mark.parametrize("columns,form", [(3, "transposed"), (3, "columns"), (3, "rows"),
                                          (3, "negated"), (1, "one of many")])
def test_table_views(cuda, columns, form):
    from torchsim_gb300 import DictionaryMatcher

    atoms = _draw(cuda, A, P)
    signals = atoms[:V] * _draw(cuda, V, 1)
    table = torch.arange(float(A * columns), device=cuda).reshape(A, columns)
    if form == "one of many":
        view = torch.stack((-table[:, 0], table[:, 0], 0.5 * table[:, 0]), 1)[:, 1]
    else:
        view = _forms(table)[form]
    want = DictionaryMatcher(dictionary=atoms, parameters=table, top_k=1).match(signals)
    got = DictionaryMatcher(dictionary=atoms, parameters=view, top_k=1).match(signals)
    _check(got, want, atoms, signals)
    assert torch.equal(got.parameters, table[got.indices])
