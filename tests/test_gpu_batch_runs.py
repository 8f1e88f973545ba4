"""A batch's pass split over launches (by launch shape, the largest problems in
launches of their own): problems of every shape, one that fills the device by
itself and one without rows, in a mixed order, each against the same problem
reconstructed alone.  The sums have the same terms and differ in order only in
the slots' sums (n terms, n * 2^-24 at worst; root of n in practice): 1e-6."""
import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300.problem import Problem, VoxelGrid, centred_grid, two_head_setup

pytestmark = pytest.mark.gpu


def grid_of(n, pitch):
    return VoxelGrid(tuple(-0.5 * k * pitch for k in n), (pitch,) * 3, n)


def member(p, rows):
    rows = torch.from_numpy(np.asarray(rows, np.int32)).cuda()
    g = torch.Generator(device="cuda").manual_seed(rows.numel())
    y = torch.poisson(torch.full((rows.numel(),), 7.0, device="cuda"), generator=g) + 1
    return p, rows, y, torch.ones(p.nvoxels, device="cuda")


def members():
    small = Problem(two_head_setup(4, 45.0, n=7), grid_of((24, 24, 24), 0.002), 20)
    mid = Problem(two_head_setup(4, 45.0, n=7), grid_of((36, 30, 36), 0.002), 60)
    long = Problem(two_head_setup(4, 45.0, n=7), grid_of((150, 24, 150), 0.0008), 60)
    large = Problem(two_head_setup(18, 20.0), centred_grid(16), 4)
    n = 4 * 20 * 32 * torch.cuda.get_device_properties(0).multi_processor_count + 4321
    assert large.nchannels > n  # four groups for every warp of the device, and more
    return [member(long, np.arange(0, long.nchannels, 3)), member(small, np.arange(3001)),
            member(small, []), member(large, np.arange(n)),
            member(mid, np.arange(7, 4000)), member(small, np.arange(5, 6000, 2))]


@pytest.mark.parametrize("order", [(0, 1, 2, 3, 4, 5), (3, 2, 1, 0), (5, 1), (3,), (2, 4)])
def test_runs_match_single(gpu_lib, order):
    every = members()
    ms = [every[i] for i in order]
    a = api.MlemBatch(ms, autotune=False)
    b = api.MlemBatch(ms, autotune=False, use_graph=False)
    a.iterate(3)
    b.iterate(3)
    for k, (p, rows, y, s) in enumerate(ms):
        # (as bits: without rows the image is 0 / 0)
        assert torch.equal(a.image(k).view(torch.int32), b.image(k).view(torch.int32))
        if rows.numel() == 0:
            continue
        R = api.Mlem(p, rows, y, s)
        R.iterate(3)
        x, want = a.image(k).double(), R.image().double()
        assert float((x - want).norm() / want.norm()) <= 1e-6, k
