"""A fused solve with many iterations allowed queues no more of them than it
needs (to the next look at the voxels left), and its answer is that of a solve
queued whole."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.helpers import draw_tissue

pytestmark = pytest.mark.gpu
BOUNDS = {"T1": (50.0, 5000.0), "T2": (2.0, 1000.0), "M0": (0.0, 5.0)}


class _Counting:
    """The library, adding up the solve iterations that are queued."""

    def __init__(self, lib):
        self.lib, self.rounds = lib, 0

    def __getattr__(self, name):
        call = getattr(self.lib, name)
        if not name.startswith("tsg_gn_solve"):
            return call

        def counted(*args):
            self.rounds += args[6]._obj.max_iterations + 1 if name == "tsg_gn_solve" else args[8]
            return call(*args)

        return counted


@pytest.mark.parametrize("limit,most", [(8, 9), (31, 32), (40, 41), (400, 64)])
def test_rounds_queued(cuda, monkeypatch, limit, most):
    from torchsim_gb300 import GaussNewton, TrustRegion, _native, engine
    from torchsim_gb300 import recon
    from torchsim_gb300.sequence import Program, mrf_events

    V = 500
    rng = np.random.default_rng(5)
    program = Program(mrf_events(rng.uniform(3, 60, 80).astype(np.float32), 9.0))
    t1, t2, b1 = draw_tissue(4, V)
    maps = engine.tissue_maps(cuda, V, t1, t2, None, b1, None)
    measured = engine.forward(program, maps, 10)
    start = torch.stack((0.9 * maps.t1.double(), 1.1 * maps.t2.double(),
                         torch.full((V,), 0.95, dtype=torch.float64, device=cuda)), 1)

    def solve():
        loop = GaussNewton(TrustRegion(), max_iterations=limit, step_tolerance=1e-4)
        return loop.minimize_program(program, measured, start, BOUNDS, 10, b1=maps.b1)

    counting = _Counting(_native.library())
    monkeypatch.setattr(_native, "library", lambda: counting)
    got = solve()
    assert counting.rounds <= most
    if limit >= 31:
        assert got.iterations < 31 and got.unconverged == 0
    monkeypatch.setattr(recon, "QUEUED_ITERATIONS", 3, raising=False)
    few = solve()
    for name in ("x", "cost", "damping", "steps"):
        assert torch.equal(getattr(got, name), getattr(few, name)), name
    assert (few.iterations, few.unconverged) == (got.iterations, got.unconverged)
