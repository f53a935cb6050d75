"""Gradients that reach the event buffers of an MRF train: only the buffers whose
protocol argument is differentiated require one (flips that move leave the
durations alone, and the other way round), a second backward is defined, and a
protocol tensor may change in place once the signal is there."""

from __future__ import annotations

import pytest
import torch

N = 6
MOVED = [("flip",), ("tr",), ("flip", "tr")]


def _leaves(device, moved):
    flip = torch.linspace(10, 60, N, device=device).requires_grad_("flip" in moved)
    tr = torch.linspace(8, 12, N, device=device).requires_grad_("tr" in moved)
    return flip, tr


@pytest.mark.parametrize("moved", MOVED)
def test_host_built_events(moved):
    from torchsim_gb300.sequence import MrfEvents, mrf_events

    flip, tr = _leaves("cpu", moved)
    events = mrf_events(flip.detach(), tr.detach())
    flip_ev, dur_ev = MrfEvents.apply(flip, tr if tr.requires_grad else None,
                                      torch.from_numpy(events.flip),
                                      torch.from_numpy(events.duration))[:2]
    assert flip_ev.requires_grad is ("flip" in moved)
    assert dur_ev.requires_grad is ("tr" in moved)


@pytest.mark.gpu
@pytest.mark.parametrize("moved", MOVED)
def test_device_built_events(cuda, moved):
    from torchsim_gb300 import MRFSimulator
    from torchsim_gb300.sequence import mrf_stream_with_gradients

    flip, tr = _leaves(cuda, moved)
    _, flip_ev, dur_ev = mrf_stream_with_gradients(flip, tr, 0.0, cuda)
    assert flip_ev.requires_grad is ("flip" in moved)
    assert dur_ev.requires_grad is ("tr" in moved)
    # The gradients are those of all arguments differentiated at once.
    t1, t2 = torch.linspace(300, 1500, 9, device=cuda), torch.linspace(30, 120, 9, device=cuda)

    def grads(names):
        f, r = _leaves(cuda, names)
        sig = MRFSimulator(flip=f, TR=r, states=7).simulate(T1=t1, T2=t2)
        leaves = [x for x in (f, r) if x.requires_grad]
        return dict(zip(names, torch.autograd.grad(sig.real.square().sum(), leaves)))

    both = grads(("flip", "tr"))
    for name, g in grads(moved).items():
        assert torch.equal(g, both[name])


@pytest.mark.gpu
@pytest.mark.parametrize("device", ["cuda", "cpu"])
@pytest.mark.parametrize("moved", [("flip",), ("flip", "tr")])
@pytest.mark.parametrize("route", ["jacobian", "off axis"])
def test_second_backward_of_a_sweep_that_has_none(cuda, route, moved, device):
    """The Jacobian's and the complex path's own backward end the graph; what is
    left of a second derivative is the flips' sign, which does not change."""
    from torchsim_gb300 import MRFSimulator

    flip, tr = _leaves(device, moved)
    t1, t2 = torch.linspace(300, 1500, 9, device=cuda), torch.linspace(30, 120, 9, device=cuda)
    model = MRFSimulator(flip=flip, TR=tr, states=7)
    if route == "jacobian":
        out = model.jacobian(("T1", "T2"), T1=t1, T2=t2)[1]
    else:
        out = model.simulate(T1=t1, T2=t2, B0=torch.linspace(-20, 20, 9, device=cuda))
    leaves = [x for x in (flip, tr) if x.requires_grad]
    first = torch.autograd.grad(out.abs().square().sum(), leaves, create_graph=True)
    assert first[0].requires_grad and bool(first[0].any())
    (second,) = torch.autograd.grad(first[0].square().sum(), [flip])
    assert second.shape == flip.shape and not bool(second.any())


@pytest.mark.gpu
@pytest.mark.parametrize("device", ["cuda", "cpu"])
@pytest.mark.parametrize("second", [False, True])
def test_protocol_tensors_change_in_place_after_the_forward(cuda, device, second):
    from torchsim_gb300 import MRFSimulator

    t1, t2 = torch.linspace(300, 1500, 9, device=cuda), torch.linspace(30, 120, 9, device=cuda)

    def run(change):
        flip, tr = _leaves(device, ("flip", "tr"))
        f, r = flip * torch.tensor([1.0, -1.0], device=device).repeat(N // 2), tr * 1.0
        sig = MRFSimulator(flip=f, TR=r, states=7).simulate(T1=t1, T2=t2)
        if change:
            with torch.no_grad():
                f.mul_(-3.0), r.zero_()
        got = torch.autograd.grad(sig.real.square().sum(), (flip, tr), create_graph=second)
        return torch.autograd.grad(sum((g * g).sum() for g in got), (flip, tr)) if second else got

    for a, b in zip(run(True), run(False)):
        assert bool(b.any()) and torch.equal(a, b)
