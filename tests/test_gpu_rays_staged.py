"""Endpoint rays of lists long enough for the staged stores (four rows a thread,
a warp's rows written 8 rays at a time through shared memory): ray counts below,
at and past whole runs, row counts that end inside a thread's rows, a warp and a
block, outputs on and off a 16-byte boundary (off: stored directly).  Every row
equals that of a short list (stored directly) and a sample the oracle's, bit for
bit; the words before and after the output keep what they held."""
import ctypes as C

import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300._lib import check, lib
from epetreco_gb300.problem import Problem, VoxelGrid, two_head_setup

pytestmark = pytest.mark.gpu

GUARD = 64  # floats on either side of the output


@pytest.mark.parametrize("shift", [0, 2])  # floats
@pytest.mark.parametrize("nrays,more", [(2, 1), (4, 2), (6, 127), (8, 3), (14, 517), (16, 1),
                                        (18, 130), (22, 6)])
def test_long_lists(gpu_lib, oracle, nrays, more, shift):
    p = Problem(two_head_setup(8, 45.0, n=13), VoxelGrid((-0.02,) * 3, (0.004,) * 3, (10,) * 3),
                nrays)
    m = 800 * torch.cuda.get_device_properties(0).multi_processor_count + more
    rows = torch.arange(m, dtype=torch.int32, device="cuda") * 11 % p.nchannels
    rows[1000:1100] = rows[1000]          # repeated channels
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
    want = torch.cat([api.rays(p, r.contiguous()) for r in rows.split(50021)])
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    pick = torch.tensor([0, 1, 3, 4, 127, 128, 511, 512, 1050, 2050, m // 2, m - 2, m - 1],
                        device="cuda")
    some = rows[pick].contiguous()
    trig = api.trig_table(p).cpu().numpy()
    rnd = api.dump_uniforms(p, some).cpu().numpy()
    for i, (c, k) in enumerate(zip(some.tolist(), pick.tolist())):
        w = np.asarray(oracle.rays(p, c, rnd[i], trig=trig), np.float32)
        assert (got[k].cpu().numpy().view(np.uint32) == w.view(np.uint32)).all(), k
