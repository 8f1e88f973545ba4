"""The walk's windows against the cells that rays visit, in float32 on the CPU
with the kernels' operations: no cell lies further outside a channel's window
than the library's bound on the roundings (epet_selftest_window_error), and
the form without a test of the cells is taken only below the windows' margin.
Rays join corners, edges and faces of the crystals, where the hull ends."""
import ctypes as C
import itertools
import math

import numpy as np
import pytest

from epetreco_gb300._lib import check, lib, problem_struct
from epetreco_gb300.problem import (MeasurementSetup, Problem, VoxelGrid, centred_grid, config,
                                    two_head_setup)

F = np.float32


def bound(p):
    v, m = C.c_double(), C.c_double()
    check(lib().epet_selftest_window_error(C.byref(problem_struct(p)), C.byref(v), C.byref(m)))
    return v.value, m.value


def fma(a, b, c):
    return F(np.float64(a) * np.float64(b) + np.float64(c))


class Channel:
    """Crystal transforms of one channel (crystal_matrix, crystal_apply)."""

    def __init__(self, s, ida, ids):
        a = F(F(F(math.pi) * F(ida)) * F(s.da)) / F(180)
        sn, cs = F(np.sin(a)), F(np.cos(a))
        self.m = []
        for det, (iz, iy) in enumerate(ids):
            ny, nz = (s.n0y, s.n0z) if det == 0 else (s.n1y, s.n1z)
            e0, e1, e2 = F(s.segx), F(s.segy), F(s.segz)
            p1 = (F(iy) - F(0.5) * F(ny - 1)) * e1
            p2 = (F(iz) - F(0.5) * F(nz - 1)) * e2
            X = F(s.pos0x if det == 0 else s.pos1x) - F(0.5) * e0
            Z = p2 - F(0.5) * e2
            self.m.append((cs * e0, sn * e2, cs * X + sn * Z, e1, p1 - F(0.5) * e1,
                           -sn * e0, cs * e2, -sn * X + cs * Z))

    def point(self, det, b):
        t00, t02, t03, t11, t13, t20, t22, t23 = self.m[det]
        b0, b1, b2 = (F(v) for v in b)
        return ((t00 * b0 + t02 * b2) + t03, t11 * b1 + t13, (t20 * b0 + t22 * b2) + t23)


def hull_indices(ch, g, planes, inv):
    """Per slab the hull's extents as positions in voxels (before the margin),
    or None where not every line spans the grid (k_walk, slab_window)."""
    c0 = [ch.point(0, (k & 1, (k >> 1) & 1, k >> 2)) for k in range(8)]
    c1 = [ch.point(1, (k & 1, (k >> 1) & 1, k >> 2)) for k in range(8)]
    a, b = ch.point(0, (0.5,) * 3), ch.point(1, (0.5,) * 3)
    ab = [F(q - r) for q, r in zip(b, a)]
    sa = 2 if abs(ab[2]) > abs(ab[0]) else 0
    h = 2 - sa
    X = planes[sa]
    lines = []
    for i, j in itertools.product((0, 1, 4, 5), repeat=2):
        ds = F(c1[j][sa] - c0[i][sa])
        if ds == 0:
            return None
        li = F(1) / ds
        t = (X - c0[i][sa]) * li
        if not (0 <= t[0] <= 1 and 0 <= t[-1] <= 1):
            return None
        lines.append((t, fma(t, F(c1[j][h] - c0[i][h]), c0[i][h])))
    t = np.stack([x[0] for x in lines])
    v = np.stack([x[1] for x in lines])
    tlo, thi = t.min(0), t.max(0)
    ya, yb = c0[0][1], c0[2][1]
    dya, dyb = F(c1[0][1] - ya), F(c1[2][1] - yb)
    y = np.stack([fma(tlo, dya, ya), fma(thi, dya, ya), fma(tlo, dyb, yb), fma(thi, dyb, yb)])
    out = {}
    for axis, lo, hi in ((h, v.min(0), v.max(0)), (1, y.min(0), y.max(0))):
        o, i = F(g.origin[axis]), inv[axis]
        out[axis] = ((np.minimum(lo[:-1], lo[1:]) - o) * i, (np.maximum(hi[:-1], hi[1:]) - o) * i)
    return sa, out


def outside(ch, g, planes, r0, r1, sa, hull):
    """How far the cells of the ray r0 -> r1, and its points at the cells' entries
    and exits, reach outside the hull's indices, in voxels; None for a ray that
    is tested anyway."""
    dr = [F(b - a) for a, b in zip(r0, r1)]
    if any(d == 0 for d in dr):
        return None
    al = [(planes[d] - r0[d]) / dr[d] for d in range(3)]
    a_in = max(min(x[0], x[-1]) for x in al)
    a_out = min(max(x[0], x[-1]) for x in al)
    if not a_in < a_out or a_in < 0 or a_out > 1:
        return None
    cuts = np.unique(np.concatenate(al + [np.array([a_in, a_out], F)]))
    cuts = cuts[(cuts >= a_in) & (cuts <= a_out)]
    first = cuts[:-1]  # each cell's entry
    idx = []
    for d in range(3):
        if dr[d] > 0:  # alpha(i) <= a < alpha(i + 1)
            i = np.searchsorted(al[d], first, side="right") - 1
        else:          # alpha(i + 1) <= a < alpha(i)
            i = len(al[d]) - 1 - np.searchsorted(al[d][::-1], first, side="right")
        idx.append(np.clip(i, 0, g.n[d] - 1))
    worst = 0.0
    for axis, (lo, hi) in hull.items():
        j = idx[axis].astype(np.float64)
        # (cells of slabs that the hull misses in the other axis count as well)
        lo, hi = lo[idx[sa]].astype(np.float64), hi[idx[sa]].astype(np.float64)
        worst = max(worst, (lo - (j + 1)).max(), (j - hi).max())
        for a in (cuts[:-1], cuts[1:]):
            x = np.float64(r0[axis]) + a.astype(np.float64) * (np.float64(r1[axis]) - r0[axis])
            x = (x - g.origin[axis]) / g.pitch[axis]
            worst = max(worst, (lo - x).max(), (x - hi).max())
    return worst


def grid(n, pitch, centre=(0.0, 0.0, 0.0)):
    return VoxelGrid(tuple(c - 0.5 * a * b for a, b, c in zip(n, pitch, centre)), pitch, n)


CASES = {
    "workload": (two_head_setup(16, 22.5), centred_grid(52)),
    "limit": (two_head_setup(16, 22.5), centred_grid(64, 5.3e-4)),
    "off_centre": (two_head_setup(16, 22.5, n=9), grid((37, 21, 44), (0.0021, 0.0033, 0.0017),
                                                       (0.011, -0.006, 0.004))),
    "far_heads": (two_head_setup(16, 22.5, pos=0.457), centred_grid(64, 1e-3)),
    "thin_crystals": (two_head_setup(16, 22.5, n=9, seg=(1e-5, 1e-5, 1e-5)),
                      centred_grid(48, 6e-4)),
    "steep": (MeasurementSetup(-0.06, 0.06, 8, 3, 401, 3, 401, 11.0, 0.004, 0.001, 0.004),
              grid((40, 60, 40), (0.0015, 0.0015, 0.0015))),
    "tall_grid": (two_head_setup(8, 45.0, n=41), grid((30, 900, 30), (1e-3, 2e-4, 1e-3))),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_no_cell_outside_by_more_than_the_bound(name):
    s, g = CASES[name]
    limit, margin = bound(Problem(s, g, 10))
    assert margin == float(F(1e-3))
    planes = [F(o) + np.arange(n + 1, dtype=F) * F(d) for o, d, n in zip(g.origin, g.pitch, g.n)]
    inv = [F(1) / F(d) for d in g.pitch]
    rng = np.random.default_rng(3)
    worst, rays = 0.0, 0
    for _ in range(150):
        ids = [(int(rng.integers(nz)), int(rng.integers(ny)))
               for nz, ny in ((s.n0z, s.n0y), (s.n1z, s.n1y))]
        ch = Channel(s, int(rng.integers(s.na)), ids)
        hull = hull_indices(ch, g, planes, inv)
        if hull is None:
            continue
        for _ in range(40):
            u = rng.random(6)
            face = rng.random(6)
            u = np.where(face < 0.4, 1e-9, np.where(face < 0.8, 1.0, u))
            r = outside(ch, g, planes, ch.point(0, u[:3]), ch.point(1, u[3:]), *hull)
            if r is not None:
                rays += 1
                worst = max(worst, r)
    print(f"{name}: {worst:.2e} of {limit:.2e} voxel, {rays} rays")
    assert rays > 200
    assert worst <= limit


def test_bound_follows_the_geometry():
    """What the walk takes untested: the workloads' grids, not ten times finer
    ones, and no geometry whose heads need not be apart along a slab axis."""
    for name in ("small", "full"):
        assert bound(config(name)["problem"])[0] < 3e-4
    s = two_head_setup(8, 45.0)
    assert bound(Problem(s, centred_grid(52, 5.5e-4), 10))[0] < 1e-3
    assert bound(Problem(s, centred_grid(52, 4.5e-4), 10))[0] > 1e-3
    assert math.isinf(bound(Problem(two_head_setup(8, 45.0, pos=0.014), centred_grid(4), 10))[0])
    # close heads with steep lines: the hull's slope counts (16 roundings of the
    # largest coordinate, 1.5 times the half height, would be 0.8e-3 of a voxel)
    steep = MeasurementSetup(-0.03, 0.03, 8, 3, 1001, 3, 1001, 45.0, 0.004, 0.001, 0.004)
    assert bound(Problem(steep, centred_grid(8, 0.9e-3), 10))[0] > 1e-3
