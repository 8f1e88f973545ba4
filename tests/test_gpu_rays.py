"""Endpoint rays at the edges of their staged stores, against the oracle bit
for bit: ray counts around the staged run of 8 rays (odd ones are stored
directly), row counts around a thread's 4 rows, a warp's and a block's share,
and an output off a 16-byte boundary (8-byte aligned, as the entry point asks);
the words before and after the output keep what they held."""
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
@pytest.mark.parametrize("nrays,m", [(1, 5), (2, 1), (6, 129), (7, 33), (8, 127), (10, 513),
                                     (16, 4), (18, 128), (101, 3)])
def test_rays_match_oracle_and_stay_inside(gpu_lib, oracle, nrays, m, shift):
    p = Problem(two_head_setup(8, 45.0, n=5), VoxelGrid((-0.02,) * 3, (0.004,) * 3, (10,) * 3),
                nrays)
    rows = np.random.default_rng(nrays).integers(0, p.nchannels, m).astype(np.int32)
    d = torch.from_numpy(rows).cuda()
    n = m * nrays * 6
    buf = torch.full((n + 2 * GUARD + shift,), -7.0, dtype=torch.float32, device="cuda")
    out = buf[GUARD + shift:]
    assert out.data_ptr() % 16 == 4 * shift
    check(lib().epet_rays(C.byref(api.problem_struct(p)), C.c_void_p(d.data_ptr()), m,
                          C.c_void_p(out.data_ptr()),
                          C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    got = buf.cpu().numpy()
    assert (got[:GUARD + shift] == -7.0).all() and (got[GUARD + shift + n:] == -7.0).all()
    got = got[GUARD + shift:GUARD + shift + n].reshape(m, nrays, 6)
    trig = api.trig_table(p).cpu().numpy()
    rnd = api.dump_uniforms(p, d).cpu().numpy()
    for i in range(m):
        want = oracle.rays(p, rows[i], rnd[i], trig=trig)
        assert (got[i].view(np.uint32) == np.asarray(want, np.float32).view(np.uint32)).all(), i


@pytest.mark.parametrize("nrays,more", [(2, 0), (2, 1), (10, 517), (7, 3)])
def test_many_rows_as_few_at_a_time(gpu_lib, oracle, nrays, more):
    """Around the row count from which a thread has several rows: the rays of a
    list are those of its pieces, and those of the oracle."""
    p = Problem(two_head_setup(8, 45.0, n=13), VoxelGrid((-0.02,) * 3, (0.004,) * 3, (10,) * 3),
                nrays)
    m = 800 * torch.cuda.get_device_properties(0).multi_processor_count + more
    rows = torch.arange(m, dtype=torch.int32, device="cuda") * 7 % p.nchannels
    got = api.rays(p, rows)
    want = torch.cat([api.rays(p, r.contiguous()) for r in rows.split(30011)])
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    pick = torch.tensor([0, 1, 3, 4, 127, 128, 511, 512, m // 2, m - 2, m - 1], device="cuda")
    some = rows[pick].contiguous()
    trig = api.trig_table(p).cpu().numpy()
    rnd = api.dump_uniforms(p, some).cpu().numpy()
    for i, (c, k) in enumerate(zip(some.tolist(), pick.tolist())):
        w = np.asarray(oracle.rays(p, c, rnd[i], trig=trig), np.float32)
        assert (got[k].cpu().numpy().view(np.uint32) == w.view(np.uint32)).all(), k
