"""Row products whose last warp has groups of lanes past the last row (which take
no part in the others' shuffles): row counts around a group, a warp
and a tile, short to long rows (4 to 32 lanes a row), one vector and two, both
directions.  Against 64-bit sums: a sum of k positive terms rounds within
(k + 1) 2^-24 of it; the words after the output keep what they held."""
import ctypes as C

import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300._lib import check, lib

pytestmark = pytest.mark.gpu

GUARD = 8


def matrix(m, n, mean):
    rng = np.random.default_rng(m + mean)
    lens = np.minimum(rng.integers(1, 2 * mean + 1, m), n)
    col = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens]).astype(np.int32)
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    return api.Csr(torch.from_numpy(ptr).cuda(), torch.from_numpy(col).cuda(),
                   torch.rand(len(col), device="cuda") + 0.1, n)


@pytest.mark.parametrize("mean", [4, 20, 60, 300])
@pytest.mark.parametrize("m", [1, 2, 3, 5, 8, 9, 31, 33, 63, 65, 255])
def test_tails(gpu_lib, m, mean):
    n = 611
    A = matrix(m, n, mean)
    At = api.csr_to_csc(A)
    a, t = A.cstruct(), At.cstruct()
    dense = torch.zeros(m, n, dtype=torch.float64, device="cuda")
    row = torch.repeat_interleave(torch.arange(m, device="cuda"), torch.diff(A.row_ptr))
    dense[row, A.col.long()] = A.val.double()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for trans, M in ((0, dense), (1, dense.t())):
        x = torch.rand(2, M.shape[1], device="cuda") + 0.1
        want = M @ x.double().t()
        bound = ((M != 0).sum(1, keepdim=True) + 1) * 2.0**-24 * want
        y = torch.full((3, M.shape[0] + GUARD), -3.0, device="cuda")
        check(lib().epet_csrmv(trans, C.byref(a), C.byref(t), 1.0, x[0].data_ptr(), 0.0,
                               y[0].data_ptr(), stream))
        pair = x.t().contiguous()
        check(lib().epet_csrmv2(trans, C.byref(a), C.byref(t), 1.0, pair.data_ptr(), 0.0,
                                y[1].data_ptr(), y[2].data_ptr(), stream))
        assert (y[:, M.shape[0]:] == -3.0).all()
        got = y[:, :M.shape[0]].double()
        assert torch.equal(got[0], got[1])
        assert ((got[1:].t() - want).abs() <= bound).all()
