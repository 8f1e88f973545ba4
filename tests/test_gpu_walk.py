"""The walk at the edges of its window arithmetic, against the oracle: grids
one cell thick, ragged and off-centre ones, a pitch so fine that every cell is
tested against the window, lines along z, ray counts around a warp and a CTA;
and grids that hold a crystal, which must be refused.  Patterns and values are
bit-exact (both sides sum the chords exactly)."""
import numpy as np
import pytest
import torch

from epetreco_gb300 import api
from epetreco_gb300._lib import EpetError
from epetreco_gb300.problem import Problem, VoxelGrid, two_head_setup

pytestmark = pytest.mark.gpu


def grid(n, pitch, shift=(0.0, 0.0, 0.0)):
    return VoxelGrid(tuple(-0.5 * a * b + c for a, b, c in zip(n, pitch, shift)), pitch, n)


CASES = {
    "thin_y": (grid((17, 1, 23), (0.003,) * 3), 8, 33),
    "thin_x": (grid((1, 19, 31), (0.002, 0.003, 0.0015)), 8, 31),
    "thin_z": (grid((29, 12, 1), (0.002, 0.002, 0.004)), 8, 1),
    "ragged_off_centre": (grid((37, 21, 44), (0.0021, 0.0033, 0.0017), (0.011, -0.006, 0.004)),
                          16, 129),
    "fine_pitch": (grid((26, 18, 21), (1e-4, 1.3e-4, 0.9e-4), (2e-3, 1e-3, -1e-3)), 8, 40),
    "anisotropic": (grid((60, 7, 5), (0.001, 0.007, 0.011)), 12, 100),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_rows_match_oracle(gpu_lib, oracle, name):
    g, na, nrays = CASES[name]
    p = Problem(two_head_setup(na, 360.0 / na, n=9), g, nrays)
    rng = np.random.default_rng(5)
    per = p.nchannels // na
    centre = per // 2  # the two heads' middle crystals
    rows = set(rng.choice(p.nchannels, 60, replace=False).tolist())
    rows |= {a * per + centre + int(k) for a in range(na) for k in rng.integers(-200, 200, 5)}
    rows = np.array(sorted(rows), np.int32)
    d = torch.from_numpy(rows).cuda()
    A = api.systemMatrixCalculation(p, d)
    trig = api.trig_table(p).cpu().numpy()
    rnd = api.dump_uniforms(p, d).cpu().numpy()
    orp, ocol, oval = oracle.sm_build_csr(p, rows, nrays, rnd, exact=True, trig=trig)
    assert A.nnz > 0
    assert (A.row_ptr.cpu().numpy() == orp).all()
    assert (A.col.cpu().numpy() == ocol).all()
    assert (A.val.cpu().numpy().view(np.uint32) == oval.view(np.uint32)).all()


@pytest.mark.parametrize("pos", [0.02, 0.05])
def test_grid_that_holds_a_crystal_is_refused(gpu_lib, pos):
    p = Problem(two_head_setup(8, 45.0, pos=pos, n=5), grid((60, 20, 60), (0.002,) * 3), 20)
    rows = torch.arange(p.nchannels, dtype=torch.int32, device="cuda")
    with pytest.raises(EpetError):
        api.systemMatrixCalculation(p, rows)
