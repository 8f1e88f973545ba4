"""The work a user has the library do, as cases that can be timed.

Each case goes through the public entry points (``epetreco_gb300.api`` and
``epetreco_gb300.autograd``): whole reconstructions, iterations of one that is
held, batches, the system-matrix build, the sensitivity image, the projector
with its gradient (matrix-free and stored), the sparse-format conversions and
the products of the reference's own operator surface.  Geometries are the
workloads of ``epetreco_gb300.problem`` or of their ranges: two heads of n x n
crystals, grids of 24 to 64 voxels a side, 8 to 180 angles, 10 to 100 rays per
channel.  ``listed`` names the cases, ``draw`` gives more of the same ranges,
``prepare`` makes inputs from a seed, ``run`` is one pass, ``work`` what a pass
cannot do without, ``exact`` the outputs in 64 bits where plain torch can make
them (the random rays are the library's generator's, so outputs that depend on
a system matrix it built have none).
"""
import math

import torch

from epetreco_gb300 import api, autograd, phantom
from epetreco_gb300.problem import (Problem, VoxelGrid, batch_angle_step, batch_members,
                                    two_head_setup)

GEOMETRY = ("nx", "ny", "nz", "crystals", "angles", "nrays")


def _geometry(nx, ny, nz, crystals, angles, nrays, **more):
    return dict(zip(GEOMETRY, (nx, ny, nz, crystals, angles, nrays)), **more)


def listed():
    return [
        # The workload a CPU can still run: 228,488 channels, 5 iterations, the
        # likelihood read back.  Set-up and launches weigh as much as the work.
        _geometry(32, 32, 32, 13, 8, 10, name="reconstruct_small", kind="reconstruct",
                  counts=1e6, iterations=5, loglik=True, values=0),
        # The headline: 5,140,980 channels, 100 rays, 20 iterations, from the
        # measured rows to the image.
        _geometry(52, 52, 52, 13, 180, 100, name="reconstruct_full", kind="reconstruct",
                  counts=5e8, iterations=20, loglik=False, values=0),
        # The smallest call: one more iteration of a small reconstruction.
        _geometry(24, 24, 24, 13, 8, 20, name="iterate_small", kind="iterate",
                  counts=1e5, iterations=1, loglik=False, values=0),
        # Iterations of the headline's reconstruction, its matrix held.
        _geometry(52, 52, 52, 13, 180, 100, name="iterate_full", kind="iterate",
                  counts=5e8, iterations=20, loglik=False, values=0),
        # 16-bit values, for memory: a mid-size scan.
        _geometry(40, 40, 40, 13, 60, 60, name="iterate_bf16", kind="iterate",
                  counts=1e7, iterations=10, loglik=False, values=1),
        # Sixteen small scans (time frames, bootstrap replicates) at once.
        dict(name="batch_small", kind="batch", problems=16, largest=32, angles=8, iterations=10),
        # Part of a matrix for a caller who keeps the CSR: an odd list of rows on
        # a ragged grid.
        _geometry(51, 47, 49, 13, 120, 100, name="build_rows", kind="build", rows=200003,
                  rays="random"),
        # The sensitivity image of a scanner: every channel.
        _geometry(40, 40, 40, 13, 30, 20, name="sensitivity", kind="sensitivity"),
        # Gradient step on a matrix too large to store: forward and backward.
        _geometry(52, 52, 52, 13, 60, 60, name="project_free", kind="project", rows=150001,
                  batch=1, stored=False),
        # The same on a stored matrix, two images at a time.
        _geometry(40, 40, 40, 13, 60, 40, name="project_stored", kind="project", rows=400009,
                  batch=2, stored=True),
        # The reference's conversions of one chunk of its unsorted elements.
        dict(name="convert_chunk", kind="convert", m=60013, n=140608, mean=330),
        # One iteration out of the reference's own operators on a held matrix.
        dict(name="operators", kind="operators", m=300007, n=140608, mean=430, values=0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _log_int(rng, lo, hi):
    return int(round(_log(rng, lo, hi)))


def draw(rng):
    kind = rng.choice(["reconstruct", "iterate", "batch", "build", "sensitivity", "project",
                       "convert", "operators"])
    if kind == "batch":
        return dict(kind=kind, problems=rng.randint(3, 24), largest=rng.randint(20, 40),
                    angles=rng.choice([4, 8, 12]), iterations=rng.randint(2, 10))
    if kind == "convert":
        return dict(kind=kind, m=_log_int(rng, 500, 90000), n=_log_int(rng, 4000, 260000),
                    mean=rng.randint(20, 400))
    if kind == "operators":
        return dict(kind=kind, m=_log_int(rng, 1000, 400000), n=_log_int(rng, 10000, 260000),
                    mean=rng.randint(20, 480), values=rng.choice([0, 0, 1, 2]))
    nx, ny, nz = (rng.randint(24, 56) for _ in range(3))
    geo = _geometry(nx, ny, nz, rng.randint(7, 13), _log_int(rng, 8, 120), rng.randint(10, 100))
    channels = geo["angles"] * geo["crystals"] ** 4
    if kind in ("reconstruct", "iterate"):
        return dict(geo, kind=kind, counts=float(round(channels * _log(rng, 1.0, 100.0))),
                    iterations=rng.randint(1, 20), loglik=rng.random() < 0.5,
                    values=rng.choice([0, 0, 0, 1, 2]))
    if kind == "sensitivity":
        return dict(geo, kind=kind)
    rows = min(channels, _log_int(rng, 1000, 400000))
    if kind == "build":
        return dict(geo, kind=kind, rows=rows, rays=rng.choice(["random"] * 5 + ["regular"]))
    return dict(geo, kind=kind, rows=rows, batch=rng.randint(1, 3), stored=rng.random() < 0.5)


# ------------------------------------------------------------------- inputs

def _problem(case, **more):
    n = (case["nx"], case["ny"], case["nz"])
    pitch = 0.002
    grid = VoxelGrid(tuple(-0.5 * pitch * k for k in n), (pitch,) * 3, n)
    setup = two_head_setup(case["angles"], batch_angle_step(case["angles"]), n=case["crystals"])
    return Problem(setup, grid, case["nrays"], **more)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _image(p, seed):
    return torch.from_numpy(phantom.phantom_image(p, seed)).cuda()


def _rows(p, count, seed):
    """`count` channels of the setup, ascending, as a measurement's rows are."""
    key = torch.rand(p.nchannels, generator=_generator(seed), device="cuda")
    return torch.topk(key, count).indices.sort().values.to(torch.int32)


def _scan(case, seed):
    p = _problem(case)
    rows, y, _ = phantom.measurement(p, case["counts"], seed=seed, phantom_seed=seed)
    return p, rows, y


def _elements(case, seed):
    """Elements of a system matrix of the shape that scans have, row-major: each
    row a line's runs of neighbouring voxels, drifting from row to row; a few
    rows are empty.  The rows' lengths are the case's, so that the outputs of
    every seed have the same sizes."""
    m, n = case["m"], case["n"]
    g = _generator(11)
    length = torch.rand(m, generator=g, device="cuda")
    length = (case["mean"] * (0.2 + 1.6 * length)).long().clamp(max=n)
    length[torch.rand(m, generator=g, device="cuda") < 0.01] = 0
    g = _generator(seed)
    row = torch.repeat_interleave(torch.arange(m, device="cuda"), length)
    start = torch.cumsum(length, 0) - length
    j = torch.arange(row.numel(), device="cuda") - start[row]
    base = (torch.arange(m, device="cuda") * (n / m)).long()
    base = base + torch.randint(0, max(1, n // 50), (m,), generator=g, device="cuda")
    # runs of 5 voxels, the next run at least as far on (no column twice)
    jump = torch.randint(5, max(6, 5 * n // (2 * case["mean"] + 5)), (m,), generator=g,
                         device="cuda")
    jump = torch.minimum(jump, (n // ((length + 4) // 5).clamp(min=1)).clamp(min=5))
    col = (base[row] + (j // 5) * jump[row] + j % 5) % n
    order = torch.argsort(row * n + col)
    row, col = row[order], col[order]
    val = torch.rand(row.numel(), generator=g, device="cuda") * 2e-3 + 1e-6
    ptr = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(length, 0)
    return row.int(), col.int(), val, ptr


def _vectors(case, seed):
    g = _generator(seed + 1)
    x = torch.rand(case["n"], generator=g, device="cuda") + 0.05
    s = torch.rand(case["n"], generator=g, device="cuda") + 0.5
    y = torch.poisson(20.0 * torch.rand(case["m"], generator=g, device="cuda"), generator=g) + 1
    return x, s, y


def _members(case):
    """The batch's problems: their geometry is the case's, their data the seed's."""
    sizes = (max(8, case["largest"] * 3 // 4), case["largest"])
    return batch_members(case["problems"], grids=sizes, angles=(case["angles"],), rays=(20, 100),
                         counts=(1e5, 1e7))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("reconstruct", "iterate"):
        p, rows, y = _scan(case, seed)
        s = api.sensitivity(p)
        state = dict(case=case, p=p, rows=rows, y=y, s=s)
        if kind == "iterate":
            state["mlem"] = api.Mlem(p, rows, y, s, value_format=case["values"])
            state["start"] = torch.full((p.nvoxels,), 1.0 / p.nvoxels, device="cuda")
        return state
    if kind == "batch":
        problems = []
        for b in _members(case):
            truth = phantom.phantom_image(b.problem, seed + b.phantom_seed, b.n_spheres)
            rows, y, _ = phantom.measurement(b.problem, b.counts, seed=seed + b.poisson_seed,
                                             x_true=truth)
            problems.append((b.problem, rows, y, api.sensitivity(b.problem)))
        start = [torch.full((q[0].nvoxels,), 1.0 / q[0].nvoxels, device="cuda") for q in problems]
        return dict(case=case, batch=api.MlemBatch(problems, autotune=False), start=start)
    if kind == "build":
        p = _problem(case, rays=case["rays"])
        # the caller's own arrays of fixed capacity, as the reference's driver has
        room = 12 * case["rows"] * max(case["nx"], case["ny"], case["nz"])
        return dict(case=case, p=p, rows=_rows(p, case["rows"], seed),
                    col=torch.zeros(room, dtype=torch.int32, device="cuda"),
                    val=torch.zeros(room, device="cuda"))
    if kind == "sensitivity":
        return dict(case=case, p=_problem(case, seed=1251 + seed))
    if kind == "project":
        p = _problem(case)
        rows = _rows(p, case["rows"], seed)
        x = torch.stack([_image(p, seed + k) for k in range(case["batch"])]) + 0.01
        with torch.no_grad():
            y = torch.poisson(1e4 * api.project_forward(p, rows, x[0]),
                              generator=_generator(seed))
        mode = "stored" if case["stored"] else "free"
        return dict(case=case, projector=autograd.Projector(p, rows, mode=mode), y=1e-4 * y,
                    x=x.requires_grad_(True))
    if kind == "convert":
        row, col, val, _ = _elements(case, seed)
        mix = torch.randperm(row.numel(), generator=_generator(seed + 2), device="cuda")
        measured = torch.unique(row)
        return dict(case=case, row=row[mix].contiguous(), col=col[mix].contiguous(),
                    val=val[mix].contiguous(), measured=measured.int())
    row, col, val, ptr = _elements(case, seed)
    x, s, y = _vectors(case, seed)
    A = api.Csr(ptr, col, val, case["n"])
    state = dict(case=case, x=x, s=s, y=y)
    if case["values"]:
        state["A16"] = api.compress(A, case["values"])
        return state
    order = torch.argsort(col, stable=True)
    cptr = torch.searchsorted(col[order].contiguous(),
                              torch.arange(case["n"] + 1, dtype=torch.int32, device="cuda"))
    state["A"] = A
    state["At"] = api.Csc(cptr, row[order].contiguous(), val[order].contiguous(), case["m"])
    return state


# --------------------------------------------------------------------- runs

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "reconstruct":
        mlem = api.Mlem(state["p"], state["rows"], state["y"], state["s"],
                        value_format=case["values"])
        loglik = mlem.iterate(case["iterations"], loglik=case["loglik"])
        return [mlem.image()] + ([loglik] if case["loglik"] else [])
    if kind == "iterate":
        mlem = state["mlem"]
        mlem.set_image(state["start"])
        loglik = mlem.iterate(case["iterations"], loglik=case["loglik"])
        return [mlem.image()] + ([loglik] if case["loglik"] else [])
    if kind == "batch":
        batch = state["batch"]
        for i, x in enumerate(state["start"]):
            batch.member(i).set_image(x)
        batch.iterate(case["iterations"])
        return [batch.image(i) for i in range(len(state["start"]))]
    if kind == "build":
        A = api.systemMatrixCalculation(state["p"], state["rows"])
        state["col"][:A.nnz].copy_(A.col)
        state["val"][:A.nnz].copy_(A.val)
        return [A.row_ptr, state["col"], state["val"]]
    if kind == "sensitivity":
        return list(api.sensitivity(state["p"], return_f64=True))
    if kind == "project":
        x = state["x"]
        ybar = state["projector"](x)
        loss = autograd.poisson_nll(ybar, state["y"])
        (grad,) = torch.autograd.grad(loss, x)
        return [ybar.detach(), grad]
    if kind == "convert":
        val, row, col = state["val"].clone(), state["row"].clone(), state["col"].clone()
        measured = state["measured"]
        api.cooSort(val, row, col)
        csr = api.convertCoo2Csr(row, row.numel(), case["m"])
        ecsr = api.convertCsr2Ecsr(measured, measured.numel(), csr, case["m"])
        At = api.csr_to_csc(api.Csr(ecsr, col, val, case["n"]))
        return [val, row, col, csr, ecsr, At.col_ptr, At.row, At.val]
    x = state["x"]
    if case["values"]:
        return [api.csr16_mv(state["A16"], x)]
    A, At = state["A"], state["At"]
    ybar = api.CSRmv(api.NON_TRANSPOSE, A, x)
    e = torch.empty_like(ybar)
    api.divides(e, state["y"], ybar)
    e = torch.nan_to_num(e, nan=0.0, posinf=0.0)  # empty rows
    c = api.CSRmv(api.TRANSPOSE, A, e, At=At)
    new = torch.empty_like(x)
    api.dividesMultiplies(new, x, c, state["s"])
    norm = api.sum(new)
    api.scales(new, 1.0 / norm)
    return [ybar, c, norm, new]


# --------------------------------------------------------- what is unavoidable

def _per_row(case):
    """Mean entries of a row: grows with the grid's side along the line and with
    the logarithm of the rays (158 at 32 voxels and 10 rays, 429 at 52 and 100)."""
    side = (case["nx"] * case["ny"] * case["nz"]) ** (1 / 3)
    return side * (1.55 + 1.455 * math.log(case["nrays"]))


def _measured(case):
    channels = case["angles"] * case["crystals"] ** 4
    return channels * (1.0 - math.exp(-case["counts"] / channels))


def _walk_flops(case, rows):
    # a crossed cell: the next plane's parameter (4), the length and its sum (4)
    side = (case["nx"] * case["ny"] * case["nz"]) ** (1 / 3)
    return 8.0 * rows * case["nrays"] * 1.45 * side


def work(case):
    kind = case["kind"]
    if kind in ("reconstruct", "iterate"):
        m, V = _measured(case), case["nx"] * case["ny"] * case["nz"]
        value = 2 if case["values"] else 4
        entries = m * _per_row(case)
        iteration = entries * (value + 2) + 8 * m + 12 * V
        flops = 4.0 * entries * case["iterations"]
        if kind == "iterate":
            return dict(bytes=case["iterations"] * iteration, flops=flops)
        return dict(bytes=case["iterations"] * iteration + entries * (value + 2) + 8 * m,
                    flops=flops + _walk_flops(case, m))
    if kind == "batch":
        entries = m = 0.0
        for b in _members(case):
            n = b.problem.grid.n
            one = _geometry(*n, 13, case["angles"], b.problem.nrays, counts=b.counts)
            m += _measured(one)
            entries += _measured(one) * _per_row(one)
        return dict(bytes=case["iterations"] * (6 * entries + 8 * m),
                    flops=case["iterations"] * 4.0 * entries)
    if kind == "build":
        rows = case["rows"]
        return dict(bytes=8.0 * rows * _per_row(case) + 12 * rows, flops=_walk_flops(case, rows))
    if kind == "sensitivity":
        rows = case["angles"] * case["crystals"] ** 4
        return dict(bytes=12.0 * case["nx"] * case["ny"] * case["nz"],
                    flops=_walk_flops(case, rows))
    if kind == "project":
        rows, V = case["rows"], case["nx"] * case["ny"] * case["nz"]
        entries = rows * _per_row(case)
        if case["stored"]:
            return dict(bytes=16.0 * entries + case["batch"] * (8 * V + 20 * rows),
                        flops=4.0 * entries * case["batch"])
        return dict(bytes=case["batch"] * (8.0 * V + 20 * rows),
                    flops=_walk_flops(case, rows) + 4.0 * entries * case["batch"])
    entries = float(case["m"] * case["mean"])
    if kind == "convert":
        return dict(bytes=12.0 * entries + 20.0 * entries + 16 * case["m"] + 8 * case["n"],
                    flops=0.0)
    if case["values"]:
        return dict(bytes=4.5 * entries + 16 * case["m"] + 4 * case["n"], flops=2.0 * entries)
    return dict(bytes=16.0 * entries + 24 * case["m"] + 32 * case["n"], flops=4.0 * entries)


# -------------------------------------------------------------------- exact

def exact(case, seed):
    if case["kind"] == "convert":
        row, col, val, _ = _elements(case, seed)  # row-major: the sorted order
        order = torch.argsort(col, stable=True)
        return [val.double(), None, None, None, None, None, None, val[order].double()]
    if case["kind"] != "operators":
        return None
    row, col, val, _ = _elements(case, seed)
    x, s, y = (v.double() for v in _vectors(case, seed))
    v64 = val.double()
    if case["values"]:
        top = torch.zeros(case["m"], device="cuda").scatter_reduce_(0, row.long(), val, "amax")
        top = torch.where(top > 0, top, torch.ones_like(top))
        kept = (val / top[row.long()]).to(torch.bfloat16 if case["values"] == 1 else torch.float16)
        v64 = kept.double() * top.double()[row.long()]
    ybar = torch.zeros(case["m"], dtype=torch.float64, device="cuda")
    ybar.index_add_(0, row.long(), v64 * x[col.long()])
    if case["values"]:
        return [ybar]
    e = torch.where(ybar > 0, y / ybar, torch.zeros_like(ybar))
    c = torch.zeros(case["n"], dtype=torch.float64, device="cuda")
    c.index_add_(0, col.long(), v64 * e[row.long()])
    new = x * c / torch.where(s == 0, torch.ones_like(s), s)
    norm = new.sum()
    return [ybar, c, float(norm), new / norm]
