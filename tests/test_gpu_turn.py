"""The echo kernel's own sine and cosine (csrc/epg_echo.cu) around the limit
of their range (1,024 rad a flip, 1,024 a B1 factor) and beyond it, against the
general sweep of the same train, which calls sincosf on the same angles: each is
within the stated tolerance of the oracle, so they are within twice that of each
other. Voxels beside one that leaves the range keep their bits."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.helpers import draw_tissue, max_rel

pytestmark = pytest.mark.gpu
SIGNAL_TOL = 1e-5
FLIPS = [0.0, 1e-30, -0.7, 45.0, 90.0, 180.0, 270.0, 359.99, 4e4, 58670.0, 58680.0, 1e6, 120.0]


@pytest.mark.parametrize("largest", [1.3, 1023.0, 1025.0, 3e4])
@pytest.mark.parametrize("flips", [FLIPS, FLIPS[:8]])
def test_echo_trains(cuda, flips, largest):
    from torchsim_gb300 import engine
    from torchsim_gb300.batching import BatchEntry, SequenceBatch
    from torchsim_gb300.sequence import Program, fse_events

    ev = fse_events(np.array(flips, np.float32), 9.0, phases_deg=90.0)
    t1, t2, _ = draw_tissue(3, 70)
    b1 = np.linspace(0.5, 1.3, 70).astype(np.float32)

    def run(b1):
        batch = SequenceBatch([BatchEntry(ev, 20, t1, t2, b1)], cuda)
        assert bool(batch.echo[0])
        batch.run()
        return 1j * batch.out.reshape(70, -1).clone()

    tame = run(b1)
    b1[5] = largest
    got = run(b1)
    want = engine.forward(Program(ev), engine.tissue_maps(cuda, 70, t1, t2, None, b1, None), 20)
    assert max_rel(got.cpu(), want.cpu()) <= 2 * SIGNAL_TOL
    others = torch.arange(70, device=cuda) != 5
    assert torch.equal(got[others], tame[others])
