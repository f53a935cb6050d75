"""The complex adjoint on trajectories at 8-byte addresses (the pairs it holds):
the gradients of a 16-byte aligned one, bit for bit, since only the width of the
copies differs. State counts whose default reverse holds two and four orders per
lane, and shapes asked for."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.helpers import draw_tissue

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("states,launch", [(3, None), (9, None), (20, None), (33, None), (64, None),
                                           (20, (5, 4, 0)), (20, (10, 2, 0))])
def test_offset_trajectory(cuda, states, launch):
    from torchsim_gb300 import engine
    from torchsim_gb300.sequence import Program, mrf_events

    rng = np.random.default_rng(states)
    program = Program(mrf_events(rng.uniform(5, 70, 37).astype(np.float32), 9.0,
                                 phases_deg=rng.uniform(-90, 90, 37).astype(np.float32)), phased=True)
    voxels = 77
    t1, t2, b1 = draw_tissue(5, voxels)
    maps = engine.tissue_maps(cuda, voxels, t1, t2, None, b1, None)
    off, keep = engine.offaxis_maps(cuda, voxels, np.linspace(-1, 1, voxels, dtype=np.float32),
                                    np.linspace(-30, 30, voxels, dtype=np.float32))
    gen = torch.Generator(device=cuda).manual_seed(6)
    seed = torch.randn((voxels, program.outputs), dtype=torch.complex64, device=cuda, generator=gen)
    size, _ = engine.complex_adjoint_plan(program, voxels, states, launch)
    buffer = torch.empty(size + 16, dtype=torch.uint8, device=cuda)

    def run(shift):
        trajectory = buffer[shift:shift + size]
        assert trajectory.data_ptr() % 16 == shift
        engine.forward_complex_trajectory(program, maps, states, off, trajectory=trajectory,
                                          launch=launch)
        grads = engine.zero_gradients(engine.COMPLEX_GRAD_NAMES, program, voxels, cuda)
        engine.adjoint_complex(program, maps, states, seed, trajectory, grads, off, launch=launch)
        return grads

    want, got = run(0), run(8)
    del keep
    for name in engine.COMPLEX_GRAD_NAMES:
        assert bool(torch.isfinite(want[name]).all()) and torch.equal(got[name], want[name]), name
