"""Several threads, each on its own stream, with windows and grids of different
sizes at a time: every call gets the shared memory it asked for, and every
result is that of the call alone."""
import threading

import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300.problem import Problem, centred_grid, two_head_setup

pytestmark = pytest.mark.gpu


def together(work, rounds):
    """Runs each of `work` `rounds` times in a thread of its own, on a stream of
    its own; returns the exceptions."""
    errors = []
    start = threading.Barrier(len(work))

    def loop(f):
        try:
            start.wait()
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(rounds):
                    f()
        except Exception as e:  # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=loop, args=(f,)) for f in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    return errors


def test_walk_windows_of_different_sizes(gpu_lib):
    p = Problem(two_head_setup(8, 22.5, n=9), centred_grid(24), 20)
    rows = torch.arange(0, p.nchannels, 811, dtype=torch.int32, device="cuda")
    x = torch.rand(p.nvoxels, device="cuda")
    want = api.project_forward(p, rows, x)
    torch.cuda.synchronize()

    def forward(cap):
        def f():
            assert torch.equal(api.project_forward(p, rows, x, max_row_nnz=cap), want)
        return f
    assert not together([forward(c) for c in (1500, 2000, 6500, 12000, 20000, 26000)], 120)


def test_grouped_layouts_of_different_grids(gpu_lib):
    work = []
    for n in (8, 24, 48, 64, 80):
        p = Problem(two_head_setup(8, 22.5, n=5), centred_grid(n), 4)
        rows = torch.arange(0, p.nchannels, 97, dtype=torch.int32, device="cuda")
        y, s = torch.ones(rows.numel(), device="cuda"), torch.ones(p.nvoxels, device="cuda")

        def make(p=p, rows=rows, y=y, s=s):
            m = api.Mlem(p, rows, y, s, use_graph=False, layout=api.LAYOUT_GROUPED)
            m.iterate(1)
            out = m.image()
            m.close()
            return out
        want = make()
        torch.cuda.synchronize()
        work.append(lambda make=make, want=want: _same(make(), want))
    assert not together(work, 60)


def _same(a, b):
    assert torch.equal(a, b)
