"""The voxel counts at which the Gauss-Newton sweep changes its shape follow the
device's number of schedulers: 24, 32 and 40 voxels for each."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("each,lanes", [(24, (5, 1)), (32, (1, 5)), (40, (5, 1))])
def test_lines_per_scheduler(cuda, each, lanes):
    from torchsim_gb300.recon import pool_shape
    from torchsim_gb300.sequence import Program, mrf_events

    program = Program(mrf_events(np.linspace(5, 60, 20).astype(np.float32), 9.0))
    schedulers = 4 * torch.cuda.get_device_properties(cuda).multi_processor_count
    got = tuple(pool_shape(program, schedulers * each + more, 10)[0] for more in (0, 1))
    assert got == lanes
