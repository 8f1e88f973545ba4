"""The grouped layout holds its entries and no more: the device memory a small
or mid-size reconstruction keeps is that of the arrays an iteration reads; and
rows whose sampled groups share more columns than the others, so that the
arrays sized by the sample are too small and the layout is made again."""
import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300.problem import config

pytestmark = pytest.mark.gpu

SLACK = 64 << 20  # the pool's granularity, and arrays that an iteration does not read


def free():
    torch.cuda.synchronize()
    api.trim_memory()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("fmt", [0, 1])
def test_held_memory(gpu_lib, fmt):
    p = config("full")["problem"]
    rows = torch.arange(170000, dtype=torch.int32, device="cuda")
    y, s = torch.ones(rows.numel(), device="cuda"), torch.ones(p.nvoxels, device="cuda")

    def make(r):
        return api.Mlem(p, r, y[:r.numel()], s, value_format=fmt, layout=api.LAYOUT_GROUPED)
    make(rows[:64]).close()  # what a first call loads
    before = free()
    m = make(rows)
    held, stats = before - free(), m.stats()
    assert stats["nnz"] > 2**25 and stats["nnz"] < 2**26
    print(f"{held / stats['nnz']:.2f} bytes held per non-zero, "
          f"{stats['bytes_per_iteration'] / stats['nnz']:.2f} read by an iteration")
    assert held <= stats["bytes_per_iteration"] + SLACK


def test_sample_too_small(gpu_lib):
    p = config("full")["problem"]
    s, cuts = p.setup, 1530
    # one channel per (angle, y sum, z sum), in the order the rows are kept in
    ida, ys, zs = np.meshgrid(np.arange(s.na), np.arange(2 * s.n0y - 1), np.arange(2 * s.n0z - 1),
                              indexing="ij")
    cls = s.channel_id(ida, zs // 2, ys // 2, zs - zs // 2, ys - ys // 2).ravel()
    # groups of 32 rows: one channel 32 times, then 32 channels
    k = np.arange(cuts)
    first = (k + 1) // 2 + 32 * (k // 2)
    pick = np.where((k % 2)[:, None] == 0, first[:, None], first[:, None] + np.arange(32))
    rows = torch.from_numpy(cls[pick.ravel()].astype(np.int32)).cuda()
    A = api.systemMatrixCalculation(p, rows)
    row = torch.repeat_interleave(torch.arange(rows.numel(), device="cuda"), torch.diff(A.row_ptr))
    entry = torch.unique((row // 2) * p.nvoxels + A.col)
    n = torch.bincount(entry // p.nvoxels, minlength=rows.numel() // 2)
    per_cut = ((n + 3) // 4 * 4).view(cuts, 16).sum(1).double()
    assert 2**24 < A.nnz < 2**26
    # every second group is sampled
    assert float(per_cut[::2].mean()) * 1.08 * cuts + 65536 < float(per_cut.sum())
    y = torch.poisson(torch.full((rows.numel(),), 9.0, device="cuda")) + 1
    x = {}
    for layout in (api.LAYOUT_GROUPED, api.LAYOUT_CSC):
        m = api.Mlem(p, rows, y, torch.ones(p.nvoxels, device="cuda"), layout=layout)
        m.iterate(3)
        x[layout] = m.image().double()
    # (sums of the same terms in another order: as the strips' own tests)
    a, b = x[api.LAYOUT_GROUPED], x[api.LAYOUT_CSC]
    assert float((a - b).norm() / b.norm()) <= 1e-6
