"""An infinite image value in a voxel whose entry FP16 rounds to zero: the row
touches the voxel, so its sum is not a number (0 times infinity) and its ratio
0, in the grouped layout's strips as in the column-major layout; a row of the
same strip that does not touch the voxel keeps a ratio."""
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300.problem import Problem, centred_grid, two_head_setup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vanishing(gpu_lib):
    """(problem, rows that have an entry below half of FP16's smallest number
    times the row's largest, such an entry's voxel)."""
    p = Problem(two_head_setup(8, 22.5, n=9), centred_grid(24), 2000)
    rows = torch.arange(0, p.nchannels, 4, dtype=torch.int32, device="cuda")
    A = api.systemMatrixCalculation(p, rows)
    row = torch.repeat_interleave(torch.arange(rows.numel(), device="cuda"), torch.diff(A.row_ptr))
    top = torch.zeros(rows.numel(), device="cuda").scatter_reduce_(0, row, A.val, "amax")
    hit = torch.nonzero((A.val / top[row]).half() == 0).flatten()
    return p, A, rows, row[hit].tolist(), A.col[hit].tolist()


@pytest.mark.parametrize("partners", [0, 1])
def test_infinite_image_at_a_vanishing_value(vanishing, partners):
    p, A, rows, hit_rows, hit_cols = vanishing
    assert len(hit_rows) > 0
    for r, voxel in list(zip(hit_rows, hit_cols))[:4]:
        other = [q for q in (r + 1, r - 1, r + 2, r - 2) if 0 <= q < rows.numel() and
                 voxel not in A.col[A.row_ptr[q]:A.row_ptr[q + 1]].tolist() and
                 A.row_ptr[q + 1] > A.row_ptr[q]][:partners]
        pick = rows[torch.tensor([r] + other, device="cuda")]
        x = torch.rand(p.nvoxels, device="cuda", generator=torch.Generator("cuda").manual_seed(r)) + 1
        x[voxel] = float("inf")
        c = {}
        for layout in (api.LAYOUT_GROUPED, api.LAYOUT_CSC):
            m = api.Mlem(p, pick, torch.full((pick.numel(),), 7.0, device="cuda"),
                         torch.ones(p.nvoxels, device="cuda"), value_format=2, layout=layout)
            m.set_image(x)
            c[layout] = m.correction()
        got, want = c[api.LAYOUT_GROUPED], c[api.LAYOUT_CSC]
        assert torch.equal(got != 0, want != 0)
        assert bool((got == 0).all()) == (len(other) == 0)
        assert torch.isfinite(got).all()
