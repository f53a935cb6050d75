"""Register budgets that no sweep is built for are refused, for a plain recorded
train as for any other program."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.helpers import draw_tissue

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unmerged", [False, True])
@pytest.mark.parametrize("shape,accepted", [((5, 4, 4, 5), True), ((5, 4, 4, 0), True),
                                            ((5, 4, 4, 99), False), ((5, 4, 4, -1), False),
                                            ((10, 2, 4, 5), False)])
def test_register_budgets(cuda, unmerged, shape, accepted):
    from torchsim_gb300 import _native, engine
    from torchsim_gb300.sequence import Program, mrf_events

    program = Program(mrf_events(np.linspace(5, 60, 25).astype(np.float32), 9.0), unmerged=unmerged)
    t1, t2, b1 = draw_tissue(3, 50)
    maps = engine.tissue_maps(cuda, 50, t1, t2, None, b1, None)
    names = ("T1", "T2", "B1")
    if not accepted:
        with pytest.raises(_native.NativeError, match="no sweep kernel"):
            engine.forward_tangents(program, maps, 20, names, launch=shape)
        return
    got = engine.forward_tangents(program, maps, 20, names, launch=shape)
    for a, b in zip(got, engine.forward_tangents(program, maps, 20, names)):
        assert (a - b).abs().max() <= 1e-5 * b.abs().max()
