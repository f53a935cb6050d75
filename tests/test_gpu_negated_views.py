"""Protocol and tissue tensors whose negation is still pending (the imaginary
part of a conjugated tensor; a lone one also counts as contiguous): the
device-built MRF stream, its transpose and the fast spin echo's recovery read the
values they stand for, so results equal those of plain tensors."""

from __future__ import annotations

import pytest
import torch

from tests.helpers import draw_tissue

pytestmark = pytest.mark.gpu


def _negated(x):
    view = torch.complex(torch.zeros_like(x), -x).conj().imag
    assert view.is_neg() and torch.equal(view, x)
    return view


@pytest.mark.parametrize("trs", [1, 50])
@pytest.mark.parametrize("tracked", [False, True])
def test_flips_and_repetition_times(cuda, tracked, trs):
    from torchsim_gb300 import MRFSimulator

    t1, t2, b1 = (torch.from_numpy(a).to(cuda) for a in draw_tissue(2, 21))
    flip = torch.linspace(-30, 60, 50, device=cuda)
    tr = torch.linspace(8, 13, trs, device=cuda)

    def run(form):
        f, r = flip.clone(), tr.clone()
        if tracked:
            f.requires_grad_(True), r.requires_grad_(True)
        sig = MRFSimulator(flip=form(f), TR=form(r), states=8).simulate(T1=t1, T2=t2, B1=b1)
        if not tracked:
            return [sig]
        return [sig.detach(), *torch.autograd.grad(sig.real.square().sum(), (f, r))]

    for got, want in zip(run(_negated), run(lambda x: x), strict=True):
        assert torch.equal(got, want)


@pytest.mark.parametrize("voxels", [1, 40])
@pytest.mark.parametrize("diff", [None, ("T1", "T2", "M0")])
def test_echo_train_recovery(cuda, diff, voxels):
    from torchsim_gb300 import fse_sim

    t1, t2, _ = (torch.from_numpy(a).to(cuda) for a in draw_tissue(2, voxels))
    m0 = torch.linspace(0.5, 1.5, voxels, device=cuda)
    flip = torch.linspace(120, 170, 12)

    def run(form):
        out = fse_sim(flip, 8.0, form(t1), t2, M0=form(m0), TR=900.0, states=16, diff=diff)
        return out if diff else [out]

    for got, want in zip(run(_negated), run(lambda x: x), strict=True):
        assert torch.equal(got, want)
