"""The walk on both sides of the pitch from which its rays' cells are not tested
against the window, against the oracle bit for bit (both sides sum the chords
exactly): oblique lines, off-centre and ragged grids, far heads, wide and thin
crystals."""
import ctypes as C

import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300._lib import check, lib, problem_struct
from epetreco_gb300.problem import Problem, VoxelGrid, two_head_setup

pytestmark = pytest.mark.gpu

# (setup, grid counts, its centre, ray count)
FORMS = {
    "oblique": (dict(na=16, da=22.5, n=13), (45, 23, 41), (0.0, 0.0, 0.0), 40),
    "off_centre": (dict(na=8, da=33.0, n=9), (37, 31, 44), (0.011, -0.006, 0.004), 100),
    "far_heads": (dict(na=8, da=45.0, n=13, pos=0.457), (36, 20, 33), (0.0, 0.004, 0.0), 33),
    "thin": (dict(na=8, da=22.5, n=9, seg=(1e-3, 1e-4, 1e-4)), (44, 9, 47), (0.003, 0.0, 0.0), 129),
}


def error(p):
    v, m = C.c_double(), C.c_double()
    check(lib().epet_selftest_window_error(C.byref(problem_struct(p)), C.byref(v), C.byref(m)))
    return v.value / m.value  # below 1: cells not tested


def problem(form, pitch):
    setup, n, centre, nrays = FORMS[form]
    g = VoxelGrid(tuple(c - 0.5 * pitch * k for c, k in zip(centre, n)), (pitch,) * 3, n)
    return Problem(two_head_setup(**setup), g, nrays)


@pytest.mark.parametrize("side", [1.01, 1.3, 0.99])  # of the limit's pitch
@pytest.mark.parametrize("form", sorted(FORMS))
def test_rows_match_oracle_around_the_limit(gpu_lib, oracle, form, side):
    lo, hi = 1e-4, 4e-3
    for _ in range(40):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if error(problem(form, mid)) > 1.0 else (lo, mid)
    p = problem(form, side * hi)
    assert (error(p) < 1.0) == (side > 1.0)
    na = p.setup.na
    rng = np.random.default_rng(11)
    per = p.nchannels // na
    rows = set(rng.choice(p.nchannels, 40, replace=False).tolist())
    rows |= {a * per + per // 2 + int(k) for a in range(na) for k in rng.integers(-300, 300, 6)}
    rows = np.array(sorted(rows), np.int32)
    d = torch.from_numpy(rows).cuda()
    A = api.systemMatrixCalculation(p, d)
    trig = api.trig_table(p).cpu().numpy()
    rnd = api.dump_uniforms(p, d).cpu().numpy()
    orp, ocol, oval = oracle.sm_build_csr(p, rows, p.nrays, rnd, exact=True, trig=trig)
    assert A.nnz > 0
    assert (A.row_ptr.cpu().numpy() == orp).all()
    assert (A.col.cpu().numpy() == ocol).all()
    assert (A.val.cpu().numpy().view(np.uint32) == oval.view(np.uint32)).all()
