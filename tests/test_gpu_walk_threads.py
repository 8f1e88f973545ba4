"""The walk's two CTA sizes on both sides of the line between them (80 rays a
channel, a window capacity of 2,048 cells): rows and forward projections have
the same bits."""
import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300.problem import Problem, centred_grid, two_head_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nrays", [(24, 1), (32, 33), (48, 80), (48, 81), (24, 129)])
def test_same_bits(gpu_lib, n, nrays):
    p = Problem(two_head_setup(8, 22.5, n=9), centred_grid(n), nrays)
    rows = torch.from_numpy(np.random.default_rng(n).choice(p.nchannels, 900, replace=False)
                            .astype(np.int32)).cuda()
    x = torch.rand(p.nvoxels, device="cuda")
    small, large = (api.systemMatrixCalculation(p, rows, max_row_nnz=c) for c in (2048, 2049))
    assert small.nnz > 0
    assert torch.equal(small.row_ptr, large.row_ptr)
    assert torch.equal(small.col, large.col)
    assert torch.equal(small.val.view(torch.int32), large.val.view(torch.int32))
    y, z = (api.project_forward(p, rows, x, max_row_nnz=c) for c in (2048, 2049))
    assert torch.equal(y, z)
