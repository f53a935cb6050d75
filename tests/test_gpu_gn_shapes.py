"""The Gauss-Newton sweep's shape around the voxel counts where it changes: the
normal equations against those of the general sweep of the same events
(compiled unmerged). Both sum the same products in FP32 runs of at most 32
samples, folded into doubles: 1e-5 of the largest entry of each sum."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from tests.helpers import draw_tissue

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("voxels,lanes", [(14592, 5), (14593, 1), (19456, 1), (19457, 5), (24320, 5),
                                          (24321, 1)])
def test_shapes_change_where_stated(cuda, voxels, lanes):
    from torchsim_gb300 import _native, engine
    from torchsim_gb300.recon import pool_shape
    from torchsim_gb300.sequence import Program, mrf_events

    rng = np.random.default_rng(voxels)
    ev = mrf_events(rng.uniform(3, 60, 40).astype(np.float32), 9.0)
    t1, t2, b1 = draw_tissue(3, voxels)
    maps = engine.tissue_maps(cuda, voxels, t1, t2, None, b1, None)
    measured = engine.forward(Program(ev), maps, 10) * 0.9
    got = []
    for program in (Program(ev), Program(ev, unmerged=True)):
        out = torch.zeros((voxels, 10), dtype=torch.float64, device=cuda)
        tissue = maps.struct()
        _native.check(_native.library().tsg_gn_evaluate(
            program.handle, ctypes.byref(tissue), voxels, 10, measured.data_ptr(), None,
            out.data_ptr(), None, torch.cuda.current_stream().cuda_stream))
        got.append(out)
    assert pool_shape(Program(ev), voxels, 10)[0] == lanes
    assert float(((got[0] - got[1]).abs() / got[1].abs().amax(0)).max()) <= 1e-5
