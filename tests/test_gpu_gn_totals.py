"""The summed cost and mean damping that a fused solve reports, iteration by
iteration, against the same solve run one iteration at a time over the voxel
pool with the totals taken by tensor sums. Both sum the same doubles in another
order: n terms of one sign differ by at most n ulp, 40,001 * 2.2e-16 < 1e-11."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.helpers import draw_tissue

pytestmark = pytest.mark.gpu
BOUNDS = {"T1": (50.0, 5000.0), "T2": (2.0, 1000.0), "M0": (0.0, 5.0)}


@pytest.mark.parametrize("voxels", [1, 2, 300, 16385, 40001])
def test_totals_are_those_of_the_pool(cuda, voxels):
    from torchsim_gb300 import GaussNewton, TrustRegion, engine
    from torchsim_gb300.recon import VoxelPool, to_free
    from torchsim_gb300.sequence import Program, mrf_events

    rng = np.random.default_rng(voxels)
    program = Program(mrf_events(rng.uniform(3, 60, 60).astype(np.float32), 9.0))
    t1, t2, b1 = draw_tissue(4, voxels)
    maps = engine.tissue_maps(cuda, voxels, t1, t2, None, b1, None)
    gen = torch.Generator(device=cuda).manual_seed(1)
    measured = engine.forward(program, maps, 10)
    measured = measured + 0.01 * torch.randn(measured.shape, dtype=torch.complex64, device=cuda,
                                             generator=gen)
    loop = GaussNewton(TrustRegion(), max_iterations=6, launch=(5, 2, 4))
    config = loop.config(BOUNDS)
    start = torch.tensor([[600.0, 60.0, 1.0]], dtype=torch.float64, device=cuda)
    u0 = to_free(start, BOUNDS).expand(voxels, 3).contiguous()
    _, _, _, _, costs, dampings = loop._pool_solve(program, measured, u0, maps.b1, config, 10)

    pool = VoxelPool(cuda)
    idx = torch.arange(voxels, device=cuda)
    pool.add(u0, maps.b1, idx, idx)
    want_costs, want_dampings, finished = [], [], 0.0
    for it in range(7):
        if it and pool.n:
            want_dampings.append(float(pool.t["damping"].mean()))
        pool.iterate(program, measured, 10, config, loop.launch)
        finished += float(pool.retire()["cost"].sum())
        want_costs.append(finished + float(pool.t["cost"].sum()))
        if pool.n == 0:
            break
    np.testing.assert_allclose(costs.cpu().numpy(), want_costs, rtol=1e-11)
    np.testing.assert_allclose(dampings.cpu().numpy(), want_dampings, rtol=1e-11)
