"""Walk windows up to the last byte of an SM's shared memory: a capacity given
by the caller that leaves no room for the walk's guard bands and slab runs, and
a grid of 15,000 cells along y (whose own bands and runs would take most of it).
Rows equal those at the automatic capacity and the oracle's bit for bit; what is
larger than shared memory stays refused."""
import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300._lib import EpetError
from epetreco_gb300.problem import Problem, VoxelGrid, centred_grid, two_head_setup

pytestmark = pytest.mark.gpu

# bytes of a CTA's window and tables, and the tables of 128^3 voxels that every
# layout holds (planes and z terms, in whole 256 bytes)
ROOM, TABLES = 232448 - 4096, 1792 + 1024


def picked(p, n, seed=7):
    rows = np.sort(np.random.default_rng(seed).choice(p.nchannels, n, replace=False))
    return torch.from_numpy(rows.astype(np.int32)).cuda()


def same(A, B):
    return (torch.equal(A.row_ptr, B.row_ptr) and torch.equal(A.col, B.col) and
            torch.equal(A.val.view(torch.int32), B.val.view(torch.int32)))


@pytest.mark.parametrize("nrays", [20, 100])  # 64 and 128 threads a channel
@pytest.mark.parametrize("below", [0, 1, 60, 200])
# (the last fits with the guard bands)
def test_capacity_up_to_shared_memory(gpu_lib, nrays, below):
    p = Problem(two_head_setup(8, 22.5), centred_grid(128), nrays)
    rows = picked(p, 700)
    cap = (ROOM - TABLES) // 8 - below
    want = api.systemMatrixCalculation(p, rows)
    assert want.nnz > 0
    assert same(api.systemMatrixCalculation(p, rows, max_row_nnz=cap), want)
    x = torch.rand(p.nvoxels, device="cuda")
    y = api.project_forward(p, rows, x, max_row_nnz=cap)
    assert torch.equal(y, api.project_forward(p, rows, x))


def test_capacity_beyond_shared_memory_is_refused(gpu_lib):
    p = Problem(two_head_setup(8, 22.5), centred_grid(128), 20)
    with pytest.raises(EpetError):
        api.systemMatrixCalculation(p, picked(p, 10), max_row_nnz=(ROOM - TABLES) // 8 + 32)


def test_grid_long_in_y(gpu_lib, oracle):
    n, pitch = (4, 15000, 4), (0.004, 1e-4, 0.004)
    g = VoxelGrid(tuple(-0.5 * a * b for a, b in zip(n, pitch)), pitch, n)
    p = Problem(two_head_setup(8, 45.0, n=7), g, 30)
    rows = picked(p, 24)
    A = api.systemMatrixCalculation(p, rows)
    trig = api.trig_table(p).cpu().numpy()
    rnd = api.dump_uniforms(p, rows).cpu().numpy()
    orp, ocol, oval = oracle.sm_build_csr(p, rows.cpu().numpy(), p.nrays, rnd, exact=True, trig=trig)
    assert A.nnz > 0
    assert (A.row_ptr.cpu().numpy() == orp).all()
    assert (A.col.cpu().numpy() == ocol).all()
    assert (A.val.cpu().numpy().view(np.uint32) == oval.view(np.uint32)).all()
