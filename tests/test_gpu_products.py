"""Products with two vectors stored pairwise (one read of the matrix for both):
each result has the bits of its own single-vector product, for ragged and
empty rows, aligned and unaligned streams, both directions, alpha and beta; and
the projector's batches made of them."""
import ctypes as C

import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300._lib import check, lib

pytestmark = pytest.mark.gpu


def matrix(m, n, mean, offset, seed=5):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 2 * mean + 1, m)
    lens[:3] = 0
    lens = np.minimum(lens, n)
    col = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens]).astype(np.int32)
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    nnz = len(col)
    c = torch.zeros(nnz + offset, dtype=torch.int32, device="cuda")
    v = torch.zeros(nnz + offset, device="cuda")
    c[offset:] = torch.from_numpy(col).cuda()
    v[offset:] = torch.rand(nnz, device="cuda")
    return api.Csr(torch.from_numpy(ptr).cuda(), c[offset:], v[offset:], n)


@pytest.mark.parametrize("m", [1, 7, 1003])
@pytest.mark.parametrize("mean,offset", [(5, 0), (20, 1), (90, 0), (400, 3)])
def test_same_bits_as_single_products(gpu_lib, m, mean, offset):
    A = matrix(m, 2500, mean, offset)
    At = api.csr_to_csc(A)
    a, t = A.cstruct(), At.cstruct()
    g = torch.Generator(device="cuda").manual_seed(7)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for trans, n_in, n_out in ((0, A.n, A.m), (1, A.m, A.n)):
        x = torch.rand(2, n_in, device="cuda", generator=g)
        y0 = torch.rand(2, n_out, device="cuda", generator=g)
        pair = x.t().contiguous()
        for alpha, beta in ((1.0, 0.0), (0.5, 2.0)):
            y = y0.clone()
            check(lib().epet_csrmv2(trans, C.byref(a), C.byref(t), alpha, pair.data_ptr(), beta,
                                    y[0].data_ptr(), y[1].data_ptr(), stream))
            for k in range(2):
                one = api.CSRmv(trans, A, x[k], alpha, beta, y0[k].clone(), At=At)
                assert torch.equal(y[k], one)


@pytest.mark.parametrize("batch", [1, 2, 3, 5])
def test_projector_batches(gpu_lib, batch):
    from epetreco_gb300.autograd import Projector
    from epetreco_gb300.problem import config
    p = config("small")["problem"]
    proj = Projector(p, torch.arange(0, p.nchannels, 57, dtype=torch.int32, device="cuda"))
    x = torch.rand(batch, p.nvoxels, device="cuda", requires_grad=True)
    y = proj(x)
    w = torch.rand_like(y)
    (grad,) = torch.autograd.grad((y * w).sum(), x)
    for k in range(batch):
        assert torch.equal(y[k], api.CSRmv(0, proj.A, x[k].detach()))
        assert torch.equal(grad[k], api.CSRmv(1, proj.A, w[k], At=proj.At))


def test_projector_pairs_of_a_large_matrix(gpu_lib):
    """Above the size from which the projector takes its vectors in pairs."""
    from epetreco_gb300.autograd import Projector
    from epetreco_gb300.problem import config
    p = config("small")["problem"]
    proj = Projector(p, torch.arange(p.nchannels, dtype=torch.int32, device="cuda"))
    assert proj.A.nnz >= 1 << 25
    x = torch.rand(3, p.nvoxels, device="cuda", requires_grad=True)
    y = proj(x)
    w = torch.rand_like(y)
    (grad,) = torch.autograd.grad((y * w).sum(), x)
    for k in range(3):
        assert torch.equal(y[k], api.CSRmv(0, proj.A, x[k].detach()))
        assert torch.equal(grad[k], api.CSRmv(1, proj.A, w[k], At=proj.At))
