"""cooSort and the column-major copy at the edges of their passes and tiles:
item counts around a tile and a chunk, key widths of one, two and more passes
(8- and 9-bit digits), empty columns in every place, against numpy's stable
sorts."""
import numpy as np
import pytest
import torch

from epetreco_gb300 import api

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("rows,cols", [(1, 1), (2, 200), (16, 16), (300, 300), (513, 1 << 17),
                                       (60013, 140608), (2**31 - 1, 2**31 - 1)])
@pytest.mark.parametrize("n", [1, 2, 31, 4095, 4096, 4097, 300001])
def test_coosort_edges(gpu_lib, n, rows, cols):
    rng = np.random.default_rng(n + rows % 1000)
    r = rng.integers(0, rows, n).astype(np.int32)
    c = rng.integers(0, cols, n).astype(np.int32)
    r[rng.random(n) < 0.3] = rows - 1  # repeated keys: the sort is stable
    c[rng.random(n) < 0.3] = 0
    v = np.arange(n, dtype=np.float32)
    dv, dr, dc = dev(v), dev(r), dev(c)
    api.cooSort(dv, dr, dc)
    order = np.lexsort((c, r))
    assert (dr.cpu().numpy() == r[order]).all()
    assert (dc.cpu().numpy() == c[order]).all()
    assert (dv.cpu().numpy() == v[order]).all()


@pytest.mark.parametrize("ncols", [1, 511, 512, 513, 1024, 1025, 300000, 600001])
@pytest.mark.parametrize("m", [1, 700])
def test_csc_empty_columns(gpu_lib, m, ncols):
    rng = np.random.default_rng(ncols)
    used = rng.choice(ncols, max(1, ncols // 3), replace=False)
    lens = rng.integers(0, min(len(used), 60) + 1, m)
    col = np.concatenate([np.sort(rng.choice(used, k, replace=False)) for k in lens] or
                         [np.zeros(0)]).astype(np.int32)
    if len(col) == 0:
        lens[0], col = 1, used[:1].astype(np.int32)
    row = np.repeat(np.arange(m), lens)
    val = rng.random(len(col)).astype(np.float32)
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    A = api.Csr(dev(ptr), dev(col), dev(val), ncols)
    At = api.csr_to_csc(A)
    order = np.argsort(col, kind="stable")
    assert (At.col_ptr.cpu().numpy() == np.searchsorted(col[order], np.arange(ncols + 1))).all()
    assert (At.row.cpu().numpy() == row[order]).all()
    assert (At.val.cpu().numpy() == val[order]).all()
