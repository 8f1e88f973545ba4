"""Candidate pairs of lists on both sides of the length from which a row has a
warp instead of a block (four rows an SM): the pairs of a list are those of its
pieces, one after the other, and the oracle's."""
import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300.problem import Problem, VoxelGrid, two_head_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [0, 1, 2, 3, 700])
@pytest.mark.parametrize("n", [(33, 32, 9), (8, 7, 40), (45, 23, 31)])  # columns: 1056, 56, 1035
def test_long_lists(gpu_lib, oracle, n, more):
    g = VoxelGrid(tuple(-0.0015 * k for k in n), (0.003,) * 3, n)
    p = Problem(two_head_setup(8, 22.5, n=9), g, 5)
    m = 4 * torch.cuda.get_device_properties(0).multi_processor_count + more
    rows = torch.from_numpy(np.random.default_rng(more).integers(0, p.nchannels, m)
                            .astype(np.int32)).cuda()
    cnl, vxl, off = api.getWorkqueue(p, rows)
    parts = [api.getWorkqueue(p, r.contiguous()) for r in rows.split(101)]
    assert cnl.numel() > 0
    assert torch.equal(cnl, torch.cat([q[0] for q in parts]))
    assert torch.equal(vxl, torch.cat([q[1] for q in parts]))
    assert torch.equal(torch.diff(off), torch.cat([torch.diff(q[2]) for q in parts]))
    trig = api.trig_table(p).cpu().numpy()
    pick = np.array([0, 1, 3, 4, m // 2, m - 1])
    ocnl, ovxl, _ = oracle.workqueue(p, rows.cpu().numpy()[pick], trig=trig)
    got = torch.cat([vxl[off[i]:off[i + 1]] for i in pick.tolist()]).cpu().numpy()
    gotc = torch.cat([cnl[off[i]:off[i + 1]] for i in pick.tolist()]).cpu().numpy()
    assert (gotc == ocnl).all() and (got == ovxl).all()
