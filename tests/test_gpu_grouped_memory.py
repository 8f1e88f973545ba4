"""The grouped layout holds its entries and no more: the device memory a small
or mid-size reconstruction keeps is that of the arrays an iteration reads."""
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
