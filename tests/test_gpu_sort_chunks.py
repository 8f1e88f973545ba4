"""cooSort and the column-major copy where a block sorts several tiles (its
counts carried from one to the next, a tile's items loaded while the one before
is written): item counts around one tile for every block, and several with a
short last chunk, key widths of 8- and 9-bit digits, repeated keys.  Against a
stable sort on the device, every item."""
import pytest
import torch

from epetreco_gb300 import api

pytestmark = pytest.mark.gpu

TILE = 4096


def counts():
    """(blocks of tiles, items more)"""
    return [(1, -1), (1, 0), (1, 1), (2, TILE + 1), (3, -1), (3, 12345), (5, 3 * TILE - 7)]


def items(per_block, more):
    return 2 * torch.cuda.get_device_properties(0).multi_processor_count * TILE * per_block + more


# key bits: 2 + 1 (one pass), 16 (two of 8), 18 (two of 9), 34 (four of 9), 40 (five of 8)
@pytest.mark.parametrize("rows,cols", [(3, 2), (256, 256), (512, 512), (60013, 140608),
                                       (1 << 20, 1 << 20)])
@pytest.mark.parametrize("per_block,more", counts())
def test_coosort(gpu_lib, per_block, more, rows, cols):
    n = items(per_block, more)
    g = torch.Generator(device="cuda").manual_seed(n % 1000 + rows)
    r = torch.randint(0, rows, (n,), device="cuda", generator=g, dtype=torch.int32)
    c = torch.randint(0, cols, (n,), device="cuda", generator=g, dtype=torch.int32)
    r[::3] = rows - 1
    c[::2] = cols - 1  # repeated keys: the sort is stable
    v = torch.arange(n, device="cuda", dtype=torch.int32).view(torch.float32)
    key, order = torch.sort(r.long() * cols + c, stable=True)
    api.cooSort(v, r, c)
    assert torch.equal(v.view(torch.int32), order.int())
    assert torch.equal(r.long() * cols + c, key)


# 9-bit digits: one, two and three passes
@pytest.mark.parametrize("ncols", [500, 140608, 300001])
@pytest.mark.parametrize("per_block,more", counts())
def test_csr_to_csc(gpu_lib, per_block, more, ncols):
    n = items(per_block, more)
    m = 5000
    g = torch.Generator(device="cuda").manual_seed(n % 1000 + ncols)
    col = torch.randint(0, ncols, (n,), device="cuda", generator=g, dtype=torch.int32)
    col[::3] = ncols - 1
    row = torch.randint(0, m, (n,), device="cuda", generator=g).sort().values
    ptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=m), 0)
    val = torch.arange(n, device="cuda", dtype=torch.int32).view(torch.float32)
    At = api.csr_to_csc(api.Csr(ptr, col, val, ncols))
    key, order = torch.sort(col, stable=True)
    assert torch.equal(At.val.view(torch.int32), order.int())
    assert torch.equal(At.row, row[order].int())
    assert torch.equal(At.col_ptr, torch.searchsorted(key, torch.arange(
        ncols + 1, dtype=torch.int32, device="cuda")))
