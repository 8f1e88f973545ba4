"""Endpoint rays of lists on both sides of the lengths at which a thread has one,
two and four rows and the stores go through shared memory (8 rays of a warp's
rows at a time): ray counts at and past whole runs, row counts that end inside a
thread's rows, a warp and a block, outputs on and off a 16-byte boundary (off:
stored directly).  Every row equals that of a short list and a sample the
oracle's, bit for bit; the words before and after the output keep what they
held."""
import ctypes as C

import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300._lib import check, lib
from epetreco_gb300.problem import Problem, VoxelGrid, two_head_setup

pytestmark = pytest.mark.gpu

GUARD = 64  # floats on either side of the output


def rows_and_rays():
    """(rows an SM, rows more, rays)"""
    staged = [(1300, more, nrays) for nrays, more in
              ((50, 1), (52, 2), (54, 127), (56, 3), (58, 517), (62, 130), (64, 6), (100, 1))]
    staged += [(3251, 5, 20)]
    direct = [(1300, 0, 50), (1300, 5, 48), (1300, 3, 51), (3249, 2, 20), (3300, 1, 19)]
    two = [(330 + 5 * nrays, more, nrays) for nrays in (2, 7) for more in (-1, 0, 1, 2, 3)]
    one = [(300, more, nrays) for nrays in (3, 8) for more in (-1, 0, 1, 2)]
    return staged + direct + two + one + [(0, 1, 10), (0, 2, 10), (0, 3, 11)]


@pytest.mark.parametrize("shift", [0, 2])  # floats
@pytest.mark.parametrize("per_sm,more,nrays", rows_and_rays())
def test_list_lengths(gpu_lib, oracle, per_sm, more, nrays, shift):
    p = Problem(two_head_setup(8, 45.0, n=13), VoxelGrid((-0.02,) * 3, (0.004,) * 3, (10,) * 3),
                nrays)
    m = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    rows = torch.arange(m, dtype=torch.int32, device="cuda") * 11 % p.nchannels
    if m > 3000:
        rows[1000:1100] = rows[1000]  # repeated channels
        rows[2000:2100] = rows[2000:2100].flip(0)  # descending ones
    n = m * nrays * 6
    buf = torch.full((n + 2 * GUARD + shift,), -7.0, device="cuda")
    out = buf[GUARD + shift:]
    assert out.data_ptr() % 16 == 4 * shift
    check(lib().epet_rays(C.byref(api.problem_struct(p)), C.c_void_p(rows.data_ptr()), m,
                          C.c_void_p(out.data_ptr()),
                          C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert (buf[:GUARD + shift] == -7.0).all() and (buf[GUARD + shift + n:] == -7.0).all()
    got = out[:n].view(m, nrays, 6)
    want = torch.cat([api.rays(p, r.contiguous()) for r in rows.split(max(1, min(19001, m // 2 + 1)))])
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    pick = torch.tensor([k for k in (0, 1, 3, 4, 127, 128, 511, 512, 1050, 2050, m // 2, m - 2, m - 1)
                         if 0 <= k < m], device="cuda")
    some = rows[pick].contiguous()
    trig = api.trig_table(p).cpu().numpy()
    rnd = api.dump_uniforms(p, some).cpu().numpy()
    for i, (c, k) in enumerate(zip(some.tolist(), pick.tolist())):
        w = np.asarray(oracle.rays(p, c, rnd[i], trig=trig), np.float32)
        assert (got[k].cpu().numpy().view(np.uint32) == w.view(np.uint32)).all(), k
