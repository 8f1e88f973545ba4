"""The grouped layout's strips (rows merged in pairs) where their arithmetic
can go wrong: row counts around a strip, a group and a warp, strips longer
than the pass holds in registers, a short-strip and a long-strip launch shape,
and images or counts that are not finite, which must not reach the rows that
do not touch them.  Against the column-major layout, whose sums have the same
terms: each sum of n terms rounds within n * 2^-24 of it, far below 1e-6 of
the image for the row lengths here (root of n)."""
import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300.problem import Problem, VoxelGrid, centred_grid, config, two_head_setup

pytestmark = pytest.mark.gpu


def recon(p, rows, layout, fmt=0):
    rows = torch.from_numpy(np.asarray(rows, np.int32)).cuda()
    g = torch.Generator(device="cuda").manual_seed(3)
    y = torch.poisson(torch.full((rows.numel(),), 9.0, device="cuda"), generator=g) + 1
    s = torch.ones(p.nvoxels, device="cuda")
    return api.Mlem(p, rows, y, s, layout=layout, value_format=fmt), rows, y


def close(a, b, tol=1e-6):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm()) <= tol


@pytest.mark.parametrize("m", [1, 2, 3, 31, 32, 33, 65, 1000])
def test_row_counts(gpu_lib, m):
    p = Problem(two_head_setup(8, 22.5), centred_grid(24), 30)
    rows = np.sort(np.random.default_rng(m).choice(p.nchannels, m, replace=False))
    if m > 3:
        rows[-2:] = rows[0]  # repeated channels
    a, _, _ = recon(p, rows, api.LAYOUT_GROUPED)
    b, _, _ = recon(p, rows, api.LAYOUT_CSC)
    la, lb = a.iterate(3, loglik=True), b.iterate(3, loglik=True)
    assert close(a.image(), b.image())
    assert abs(la - lb) <= 1e-6 * abs(lb)


def grid_of(n, pitch):
    return VoxelGrid(tuple(-0.5 * k * pitch for k in n), (pitch,) * 3, n)


@pytest.mark.parametrize("n,pitch,rays,longest", [
    ((24, 24, 24), 0.002, 20, 128),        # two chunks per lane
    ((36, 30, 36), 0.002, 60, 256),        # three
    ((60, 40, 60), 0.0016, 100, 512),      # five
    ((150, 24, 150), 0.0008, 60, 640),     # beyond the registers
])
def test_strip_lengths(gpu_lib, n, pitch, rays, longest):
    p = Problem(two_head_setup(4, 45.0, n=7), grid_of(n, pitch), rays)
    rows = np.arange(p.nchannels // 4 * 3)[::3]
    A = api.systemMatrixCalculation(p, torch.from_numpy(rows.astype(np.int32)).cuda())
    assert int(torch.diff(A.row_ptr).max()) > longest // 2
    a, _, _ = recon(p, rows, api.LAYOUT_GROUPED)
    b, _, _ = recon(p, rows, api.LAYOUT_CSC)
    a.iterate(4)
    b.iterate(4)
    assert close(a.image(), b.image())


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_not_finite_stays_in_its_rows(gpu_lib, value):
    p = config("small")["problem"]
    rows = np.arange(0, p.nchannels, 41)
    a, _, y = recon(p, rows, api.LAYOUT_GROUPED)
    b, r, _ = recon(p, rows, api.LAYOUT_CSC)
    A = api.systemMatrixCalculation(p, r)
    x = torch.full((p.nvoxels,), 1.0 / p.nvoxels, device="cuda")
    j = int(A.col[A.nnz // 2])
    x[j] = value  # an image voxel
    for R in (a, b):
        R.set_image(x)
    ca, cb = a.correction(), b.correction()
    assert torch.isfinite(cb).all() and torch.isfinite(ca).all()
    assert close(ca, cb)


def test_infinite_count_stays_in_its_columns(gpu_lib):
    p = config("small")["problem"]
    rows = torch.arange(0, p.nchannels, 41, dtype=torch.int32, device="cuda")
    y = torch.full((rows.numel(),), 5.0, device="cuda")
    y[1234] = float("inf")
    s = torch.ones(p.nvoxels, device="cuda")
    a = api.Mlem(p, rows, y, s, layout=api.LAYOUT_GROUPED)
    b = api.Mlem(p, rows, y, s, layout=api.LAYOUT_CSC)
    ca, cb = a.correction(), b.correction()
    fin = torch.isfinite(cb)
    assert 0 < int((~fin).sum()) < p.nvoxels
    assert torch.equal(fin, torch.isfinite(ca))
    assert close(ca[fin], cb[fin])
