"""The fast spin echo's steady state as one kernel (csrc/fse_recovery.cu)
against FSESimulator._post, the tensor form: every column and order, scalar
and per-voxel T1 and M0, odd sizes, complex trains; and the forms it leaves to
the tensor form. Both are FP32 evaluations of the same expression, some ten
roundings deep, so they agree to 1e-5 of the largest value."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.helpers import max_rel

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("rows,echoes", [(1, 1), (33, 7), (1000, 48), (5, 257)])
@pytest.mark.parametrize("names", [None, ("T1", "T2"), ("M0", "T2"), ("B1", "M0", "T1"), ("T2",)])
@pytest.mark.parametrize("form", ["scalar", "maps", "tensor TR", "subclass"])
def test_agrees_with_the_tensor_form(cuda, rows, echoes, names, form):
    from torchsim_gb300.simulators import FSESimulator

    class Doubled(FSESimulator):
        def _post(self, *args):
            out, jac = super()._post(*args)
            return 2 * out, jac

    model = Doubled() if form == "subclass" else FSESimulator()
    gen = torch.Generator(device=cuda).manual_seed(rows + echoes)
    draw = lambda *shape: torch.randn(*shape, dtype=torch.complex64, device=cuda, generator=gen) * 0.3
    kernel = model._kernel_names(names) if names else None
    signal = draw(rows, echoes)
    jac = draw(rows, len(kernel), echoes) if names else None
    held = {"T1": 900.0, "M0": 1.3}
    if form != "scalar":
        held = {"T1": torch.rand(rows, device=cuda, generator=gen) * 2000 + 200,
                "M0": torch.rand(rows, device=cuda, generator=gen) + 0.5}
    protocol = {"ESP": 7.3, "TR": torch.tensor(3000.0) if form == "tensor TR" else 3000.0}
    want = model._post(signal, jac, names, held, protocol, cuda)
    got = model._post_untracked(signal.clone(), None if jac is None else jac.clone(), names, held,
                                protocol, cuda)
    assert max_rel(got[0].cpu(), want[0].cpu()) <= TOL
    if names:
        for c in range(len(names)):
            assert max_rel(got[1][:, c].cpu(), want[1][:, c].cpu()) <= TOL
    else:
        assert got[1] is None
