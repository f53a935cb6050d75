"""Gradients through a device-built MRF stream (one kernel and its transpose)
against the host-built stream's, over the forms the kernel takes: TRs as a
number, one value or one per pulse, negative flips, strided leaves, longer
trains than its staging chunk, and a second backward."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.helpers import draw_tissue

pytestmark = pytest.mark.gpu


def _grads(cuda, device, flip, tr, n, second):
    from torchsim_gb300 import MRFSimulator

    t1, t2, b1 = (torch.from_numpy(a).to(cuda) for a in draw_tissue(2, 33))
    f = torch.from_numpy(flip).to(device).requires_grad_(True)
    r = tr if isinstance(tr, float) else torch.from_numpy(tr).to(device).requires_grad_(True)
    strided = torch.stack((f, f), 1)[:, 1]  # a view with stride 2
    leaves = [f] if isinstance(tr, float) else [f, r]
    sig = MRFSimulator(flip=strided, TR=r, states=9).simulate(T1=t1, T2=t2, B1=b1)
    gen = torch.Generator(device=cuda).manual_seed(4)
    seed = torch.randn(sig.shape, dtype=torch.complex64, device=cuda, generator=gen)
    got = torch.autograd.grad(sig, leaves, seed, create_graph=second)
    if second:
        got = torch.autograd.grad(sum((g * g).sum() for g in got), leaves)
    return [sig.detach().cpu(), *(g.cpu() for g in got)]


@pytest.mark.parametrize("second", [False, True])
@pytest.mark.parametrize("n,kind", [(2, "each"), (7, "number"), (40, "one"), (255, "each"),
                                    (1025, "each"), (2040, "number")])
def test_device_stream_gradients_equal_the_host_streams(cuda, n, kind, second):
    rng = np.random.default_rng(n)
    flip = rng.uniform(-60, 60, n).astype(np.float32)
    tr = {"number": 9.0, "one": np.array([11.0], np.float32),
          "each": rng.uniform(6, 14, n).astype(np.float32)}[kind]
    for a, b in zip(_grads(cuda, cuda, flip, tr, n, second), _grads(cuda, "cpu", flip, tr, n, second)):
        # The same values through both streams; a lone TR's gradient is summed
        # over the pulses in another order: n float32 terms.
        assert (a - b).abs().max() <= 1e-6 * n**0.5 * b.abs().max()
