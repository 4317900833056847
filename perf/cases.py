"""The workloads that this framework's speed is measured on.

A case is one call sequence that a program using cgxx_b200 makes in earnest:
solves through Handle.solve with every matrix format, preconditioner and
precision, on the structured-grid and geometric-graph systems of the tests and
the benchmark, from a 64 x 64 grid to 160^3; a whole one-off solve from host
arrays; the learned preconditioner's step of a time-stepping program; and the
loss and gradient of the network's training step.

The systems are those of cgxx_b200.generators, built here with torch on the
GPU because they are made many times: variable-coefficient diffusion on
structured grids (5-point Poisson, 7-point and 27-point stencils, coefficient
exp(g) with g a Gaussian random field) and Laplacians of random geometric
graphs. The right-hand side is A x* with x* uniform in [-1, 1], so x* is the
exact solution. The solves run to a relative residual of 1e-13: their
solutions then agree with x* to ten digits, as a program needs that goes on to
difference or differentiate them.
"""
import math

import numpy as np
import torch

import cgxx_b200 as cg
from cgxx_b200 import learned

TOLERANCE = 1e-13
MAX_ITERATIONS = 20000
EPS = 1e-4  # of M^-1 = G G^T + eps D^-1, as in training and the benchmark


def listed():
    return [
        # The smallest solve of the tests and the smoke run: launches and
        # barriers are all of its time.
        {"name": "poisson64_fp64", "kind": "solve", "family": "poisson", "nz": 1, "ny": 64,
         "nx": 64, "format": "crs", "precond": "jacobi", "precision": "fp64"},
        # The CPU-runnable 2-D configuration with an odd edge, read as COO
        # and without preconditioner, as the reference's defaults run it.
        {"name": "poisson257_coo_none", "kind": "solve", "family": "poisson", "nz": 1,
         "ny": 257, "nx": 257, "format": "coo", "precond": "none", "precision": "fp64"},
        # A mid-size 3-D box with three different edges, held as ELL.
        {"name": "diff7_box_ell_fp64", "kind": "solve", "family": "diff7", "nz": 97, "ny": 64,
         "nx": 83, "sigma": 1.0, "corr": 8.0, "format": "ell", "precond": "jacobi",
         "precision": "fp64"},
        # The benchmark's grid in the reference's arithmetic, the default
        # path of every program that only switches libraries.
        {"name": "diff7_160_fp64", "kind": "solve", "family": "diff7", "nz": 160, "ny": 160,
         "nx": 160, "sigma": 1.0, "corr": 8.0, "format": "crs", "precond": "jacobi",
         "precision": "fp64"},
        # One matrix, one solve: what the command-line program does after
        # reading its file (upload, Jacobi set-up, solve, read-back).
        {"name": "diff27_96_oneshot", "kind": "oneshot", "family": "diff27", "nz": 96, "ny": 96,
         "nx": 96, "sigma": 1.0, "corr": 8.0, "format": "crs", "precond": "jacobi",
         "precision": "fp64"},
        # An irregular matrix in FP64: rows of uneven length, scattered
        # columns.
        {"name": "graph1m_fp64", "kind": "solve", "family": "graph", "points": 1000003,
         "degree": 12.0, "format": "crs", "precond": "jacobi", "precision": "fp64"},
        # Mixed precision on the band form's matrices, beyond the sizes that
        # stay in L2 with all their vectors.
        {"name": "diff7_128_mixed", "kind": "solve", "family": "diff7", "nz": 128, "ny": 128,
         "nx": 128, "sigma": 1.0, "corr": 8.0, "format": "crs", "precond": "jacobi",
         "precision": "mixed"},
        # The 27-point workload in mixed precision (no band form).
        {"name": "diff27_128_mixed", "kind": "solve", "family": "diff27", "nz": 128, "ny": 128,
         "nx": 128, "sigma": 1.0, "corr": 8.0, "format": "crs", "precond": "jacobi",
         "precision": "mixed"},
        # A step of a time-stepping program on the grid the network was
        # trained on: new values of the same pattern, set-up, inference,
        # solve, read-back.
        {"name": "diff7_96_learned", "kind": "step", "family": "diff7", "nz": 96, "ny": 96,
         "nx": 96, "sigma": 1.0, "corr": 8.0, "format": "crs", "precond": "learned",
         "precision": "mixed"},
        # The same step at the benchmark's size.
        {"name": "diff7_160_learned", "kind": "step", "family": "diff7", "nz": 160, "ny": 160,
         "nx": 160, "sigma": 1.0, "corr": 8.0, "format": "crs", "precond": "learned",
         "precision": "mixed"},
        # The same step on the geometric-graph workload.
        {"name": "graph2m_learned", "kind": "step", "family": "graph", "points": 2000000,
         "degree": 12.0, "format": "crs", "precond": "learned", "precision": "mixed"},
        # A training step's loss and gradient on the training grid, probes by
        # the training driver's recipe.
        {"name": "train_diff7_96", "kind": "train", "family": "diff7", "nz": 96, "ny": 96,
         "nx": 96, "sigma": 1.0, "corr": 8.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "oneshot", "step", "step", "train"])
    family = rng.choice(["poisson", "diff7", "diff7", "diff27", "graph"]
                        if kind in ("solve", "oneshot") else ["diff7", "diff7", "diff27", "graph"])
    case = {"kind": kind, "family": family}
    # Iterations grow with the edge: the edges' upper ends keep every drawn
    # case below the largest listed one.
    if family == "graph":
        top = {"solve": 1000000, "oneshot": 1000000, "step": 2000000, "train": 250000}[kind]
        case.update(points=_log_int(rng, 5000, top), degree=rng.uniform(8.0, 14.0))
    elif family == "poisson":
        n = _log_int(rng, 48, 640)
        case.update(nz=1, ny=n, nx=max(32, int(n * rng.uniform(0.6, 1.1))))
    else:
        top = {("diff7", "train"): 104, ("diff27", "train"): 72, ("diff7", "step"): 150,
               ("diff27", "step"): 112}.get((family, kind), 140 if family == "diff7" else 112)
        n = _log_int(rng, 20, top)
        case.update(nz=n, ny=max(16, int(n * rng.uniform(0.7, 1.0))),
                    nx=max(16, int(n * rng.uniform(0.7, 1.1))),
                    sigma=rng.uniform(0.5, 1.2), corr=rng.uniform(4.0, 12.0))
    if kind == "step":
        case.update(format="crs", precond="learned", precision="mixed")
    elif kind in ("solve", "oneshot"):
        precision = rng.choice(["fp64", "fp64", "mixed"])
        none = precision == "fp64" and family == "poisson" and rng.random() < 0.5
        case.update(format=rng.choice(["crs", "crs", "ell", "coo"]),
                    precond="none" if none else "jacobi", precision=precision)
    return case


# ---------------------------------------------------------------------------
# Systems: CRS on the GPU, rows sorted by column (ptr int64, rest as stored).

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _field(shape, sigma, corr, gen):
    """exp of a stationary Gaussian field, as generators.diffusion_field."""
    white = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
    k2 = torch.zeros(shape, device="cuda", dtype=torch.float64)
    for ax, n in enumerate(shape):
        k = 2 * math.pi * torch.fft.fftfreq(n, device="cuda", dtype=torch.float64)
        k2 = k2 + (k ** 2).reshape([n if a == ax else 1 for a in range(3)])
    g = torch.fft.ifftn(torch.fft.fftn(white) * torch.exp(-0.25 * corr ** 2 * k2)).real
    g = g - g.mean()
    return torch.exp(g * (sigma / g.std()))


def _grid(case, gen):
    """Cell-centred grid operators of generators.poisson2d and diffusion3d."""
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    N = nz * ny * nx
    family = case["family"]
    if family == "diff27":
        offs = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)]
    elif family == "diff7":
        offs = [(-1, 0, 0), (0, -1, 0), (0, 0, -1), (0, 0, 0), (0, 0, 1), (0, 1, 0), (1, 0, 0)]
    else:
        offs = [(0, -1, 0), (0, 0, -1), (0, 0, 0), (0, 0, 1), (0, 1, 0)]
    kap = (torch.ones((nz, ny, nx), device="cuda", dtype=torch.float64) if family == "poisson"
           else _field((nz, ny, nx), case["sigma"], case["corr"], gen))
    # One layer of cells around the grid, coefficient 0 outside.
    pad = torch.zeros((nz + 2, ny + 2, nx + 2), device="cuda", dtype=torch.float64)
    pad[1:-1, 1:-1, 1:-1] = kap
    lin = torch.arange(N, device="cuda", dtype=torch.int32).reshape(nz, ny, nx)
    vals = torch.empty((N, len(offs)), device="cuda", dtype=torch.float64)
    cols = torch.empty((N, len(offs)), device="cuda", dtype=torch.int32)
    mask = torch.empty((N, len(offs)), device="cuda", dtype=torch.bool)
    diag = torch.zeros((nz, ny, nx), device="cuda", dtype=torch.float64)
    centre = offs.index((0, 0, 0))
    for k, (dz, dy, dx) in enumerate(offs):
        cols[:, k] = (lin + ((dz * ny + dy) * nx + dx)).reshape(-1)
        if k == centre:
            mask[:, k] = True
            continue
        kj = pad[1 + dz:1 + dz + nz, 1 + dy:1 + dy + ny, 1 + dx:1 + dx + nx]
        inside = kj > 0
        w = 1.0 / (abs(dz) + abs(dy) + abs(dx))
        c = torch.where(inside, w * 2.0 * kap * kj / (kap + kj), w * kap)
        diag += c
        vals[:, k] = -c.reshape(-1)
        mask[:, k] = inside.reshape(-1)
    vals[:, centre] = diag.reshape(-1)
    ptr = torch.zeros(N + 1, device="cuda", dtype=torch.int64)
    torch.cumsum(mask.sum(1), 0, out=ptr[1:])
    return N, ptr, cols[mask], vals[mask]


def _graph(case, gen):
    """Laplacian of a random geometric graph plus 1e-3 I, points numbered
    along a Morton curve, as generators.geometric_graph."""
    N, degree = case["points"], case["degree"]
    pts = torch.rand((N, 3), generator=gen, device="cuda", dtype=torch.float64)
    q = (pts * 1024).to(torch.int64).clamp_(max=1023)
    code = torch.zeros(N, device="cuda", dtype=torch.int64)
    for b in range(10):
        for a in range(3):
            code |= ((q[:, a] >> b) & 1) << (3 * b + a)
    pts = pts[torch.sort(code, stable=True).indices]
    r = (3.0 * degree / (4.0 * math.pi * N)) ** (1.0 / 3.0)
    m = max(1, int(1.0 / r))  # cells of edge >= r
    cell = (pts * m).to(torch.int64).clamp_(max=m - 1)
    cid = (cell[:, 0] * m + cell[:, 1]) * m + cell[:, 2]
    order = torch.sort(cid, stable=True).indices
    start = torch.searchsorted(cid[order], torch.arange(m ** 3 + 1, device="cuda"))
    own = torch.arange(N, device="cuda")
    keys, wts = [], []
    for k in range(27):
        near = cell + torch.tensor([k // 9 - 1, k // 3 % 3 - 1, k % 3 - 1], device="cuda")
        ok = ((near >= 0) & (near < m)).all(1)
        nid = torch.where(ok, (near[:, 0] * m + near[:, 1]) * m + near[:, 2], 0)
        count = torch.where(ok, start[nid + 1] - start[nid], 0)
        i = torch.repeat_interleave(own, count)
        ends = torch.cumsum(count, 0)
        at = torch.arange(i.numel(), device="cuda") - (ends - count)[i] + start[nid][i]
        j = order[at]
        d = (pts[i] - pts[j]).square().sum(1).sqrt()
        keep = (d < r) & (i != j)
        keys.append(i[keep] * N + j[keep])
        wts.append(torch.exp(-d[keep] / r))
    keys.append(own * (N + 1))
    wts.append(torch.zeros(N, device="cuda", dtype=torch.float64))
    key, at = torch.sort(torch.cat(keys))
    w = torch.cat(wts)[at]
    rows, cols = key // N, (key % N).to(torch.int32)
    ptr = torch.zeros(N + 1, device="cuda", dtype=torch.int64)
    torch.cumsum(torch.bincount(rows, minlength=N), 0, out=ptr[1:])
    diag = _row_sums(ptr, w) + 1e-3
    vals = torch.where(rows == cols, diag[rows], -w)
    return N, ptr, cols, vals


def _rows_of(ptr):
    return torch.repeat_interleave(torch.arange(ptr.numel() - 1, device="cuda"), ptr[1:] - ptr[:-1])


def _row_sums(ptr, entries):
    """Sum of each row's entries in a fixed order."""
    rows = _rows_of(ptr)
    slot = torch.arange(entries.numel(), device="cuda") - ptr[rows]
    table = torch.zeros((ptr.numel() - 1, int((ptr[1:] - ptr[:-1]).max())), device="cuda",
                        dtype=entries.dtype)
    table[rows, slot] = entries
    return table.sum(1)


def _system(case, seed):
    """(N, ptr, cols, vals, x*) from the seed."""
    gen = _generator(seed)
    N, ptr, cols, vals = (_graph if case["family"] == "graph" else _grid)(case, gen)
    x = torch.rand(N, generator=gen, device="cuda", dtype=torch.float64) * 2.0 - 1.0
    return N, ptr, cols, vals, x


def _pinned(t, dtype):
    a = cg.pinned_empty(t.numel(), dtype)
    torch.from_numpy(np.asarray(a)).copy_(t)
    return a


def _ell(N, ptr, cols, vals):
    """Column-major ELL arrays of generators.to_ell (padding 0)."""
    length = (ptr[1:] - ptr[:-1]).to(torch.int32)
    width = int(length.max())
    rows = _rows_of(ptr)
    at = (torch.arange(cols.numel(), device="cuda") - ptr[rows]) * N + rows
    index = torch.zeros(width * N, device="cuda", dtype=torch.int32)
    data = torch.zeros(width * N, device="cuda", dtype=torch.float64)
    index[at], data[at] = cols, vals
    return width, length, index, data


# ---------------------------------------------------------------------------

def _host_matrix(case, N, ptr, cols, vals):
    """The host arrays of the case's format, page-locked as a program that
    uploads them again and again holds them."""
    if case["format"] == "ell":
        width, length, index, data = _ell(N, ptr, cols, vals)
        return (N, cols.numel(), width, _pinned(length, np.int32), _pinned(index, np.int32),
                _pinned(data, np.float64))
    if case["format"] == "coo":
        return (N, _pinned(_rows_of(ptr).to(torch.int32), np.int32), _pinned(cols, np.int32),
                _pinned(vals, np.float64))
    return (_pinned(ptr.to(torch.int32), np.int32), _pinned(cols, np.int32),
            _pinned(vals, np.float64))


def _upload(h, fmt, arrays):
    {"crs": h.upload_crs, "ell": h.upload_ell, "coo": h.upload_coo}[fmt](*arrays)


def prepare(case, seed):
    N, ptr, cols, vals, x = _system(case, seed)
    kind = case["kind"]
    h = cg.Handle(0)
    state = {"kind": kind, "h": h}
    if kind == "train":
        h.upload_crs(ptr.to(torch.int32).cpu().numpy(), cols.cpu().numpy(), vals.cpu().numpy())
        h.learned_setup()
        net = cg.Gnn(0, learned.init_params(int(seed) % (1 << 31)))
        net.set_probes(3, 4, 3.0, 0)  # the training driver's defaults
        state.update(net=net, seed=_probe_seed(seed))
        return state
    b = _row_sums(ptr, vals * x[cols.to(torch.int64)])
    state.update(
        x=cg.pinned_empty(N, np.float64),
        options=cg.default_options(
            max_iterations=MAX_ITERATIONS, tolerance=TOLERANCE,
            preconditioner={"none": cg.PRECOND_NONE, "jacobi": cg.PRECOND_JACOBI,
                            "learned": cg.PRECOND_LEARNED}[case["precond"]],
            precision=cg.PRECISION_MIXED if case["precision"] == "mixed" else cg.PRECISION_FP64))
    if kind == "oneshot":
        state.update(format=case["format"], arrays=_host_matrix(case, N, ptr, cols, vals),
                     b=_pinned(b, np.float64), jacobi=case["precond"] == "jacobi")
        return state
    if kind == "solve":
        _upload(h, case["format"], _host_matrix(case, N, ptr, cols, vals))
        h.jacobi_from_matrix()
    else:
        h.upload_crs(ptr.to(torch.int32).cpu().numpy(), cols.cpu().numpy(), vals.cpu().numpy())
        weights = "graph12.gnn" if case["family"] == "graph" else "diffusion7.gnn"
        params, _ = learned.load_weights(
            learned.DEFAULT_WEIGHTS.replace("diffusion7.gnn", weights))
        state.update(net=cg.Gnn(0, params), values=vals)
    h.set_vector("K", b.cpu().numpy())
    h.synchronize()
    return state


def run(state):
    h, kind = state["h"], state["kind"]
    if kind == "train":
        loss, grad = state["net"].loss_grad(h, seed=state["seed"])
        return {"loss": loss, "grad": grad}
    if kind == "oneshot":
        _upload(h, state["format"], state["arrays"])
        if state["jacobi"]:
            h.jacobi_from_matrix()
        h.set_vector("K", state["b"])
    elif kind == "step":
        h.update_crs_values_ptr(state["values"].data_ptr())
        h.jacobi_from_matrix()
        h.learned_setup()
        h.learned_factor(state["net"], EPS)
        h.fill_vector("X", 0.0)
    else:
        h.fill_vector("X", 0.0)
    h.solve(state["options"])
    return h.get_vector("X", out=state["x"])


# ---------------------------------------------------------------------------

def _shape(case):
    """(rows, entries) of the case's matrix; a graph's by its mean degree."""
    if case["family"] == "graph":
        return case["points"], case["points"] * (1.0 + 0.95 * case["degree"])
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    N = nz * ny * nx
    if case["family"] == "diff27":
        return N, (3 * nz - 2) * (3 * ny - 2) * (3 * nx - 2)
    faces = N // nx * (nx - 1) + N // ny * (ny - 1) + N // nz * (nz - 1)
    return N, N + 2 * faces


def _iterations(case):
    """Iterations to 1e-13, by fits to measured solves."""
    if case["family"] == "graph":
        its = 8.0 * case["points"] ** (1.0 / 3.0)
    else:
        n = max(case["nz"], case["ny"], case["nx"])
        its = {"poisson": 3.6, "diff7": 5.8, "diff27": 3.7}[case["family"]] * n
    return its * (0.55 if case["precond"] == "learned" else 1.0)


def work(case):
    """Solves: per iteration the distinct values of the symmetric matrix
    (with a 4-byte index each on a graph) once, and x, r and p read and
    written once, in the iteration's precision; the learned factor's BF16
    values on top. Training: the scaled matrix once, and the network's and
    the probes' arithmetic forward and backward."""
    N, nnz = _shape(case)
    half = (nnz + N) / 2.0
    graph = case["family"] == "graph"
    if case["kind"] == "train":
        dense = 3 * 2.0 * 64 * 32 + 2.0 * 4 * 32 + 2.0 * 32 * 10
        sparse = 3 * 2.0 * 32 * nnz
        probes = (3 + 2 + 2 + 3 + 1) * 2.0 * 8 * nnz * 0.75
        return {"bytes": 8.0 * nnz + 20.0 * N, "flops": 3 * (dense * N + sparse) + probes}
    its = _iterations(case)
    width = 8.0 if case["precision"] == "fp64" else 4.0
    per_it = half * (width + (4.0 if graph else 0.0)) + 6 * width * N
    flops = 2.0 * nnz + 12.0 * N
    if case["precond"] == "learned":
        per_it += half * (2.0 + (4.0 if graph else 0.0))
        flops += 4.0 * half
    total = its * per_it + 12.0 * nnz + 16.0 * N
    return {"bytes": total, "flops": its * flops}


# ---------------------------------------------------------------------------

def _probe_seed(seed):
    return (int(seed) * 1000003 + 17) % (1 << 62)


def _rademacher(N, seed):
    """The probes of Gnn.loss_grad (splitmix64 finalizer of seed + golden
    ratio * (t + 1), odd -> +1), in wrapping 64-bit integers."""
    def wrap(v):
        v &= (1 << 64) - 1
        return v - (1 << 64) if v >> 63 else v

    def shift(z, k):  # logical
        return (z >> k) & ((1 << (64 - k)) - 1)

    t = torch.arange(1, N * 8 + 1, device="cuda", dtype=torch.int64)
    z = t * wrap(0x9E3779B97F4A7C15) + wrap(seed)
    z = (z ^ shift(z, 30)) * wrap(0xBF58476D1CE4E5B9)
    z = (z ^ shift(z, 27)) * wrap(0x94D049BB133111EB)
    z = z ^ shift(z, 31)
    return ((z & 1) * 2 - 1).to(torch.float64).reshape(N, 8)


def _exact_train(case, seed):
    """Loss and gradient of the network in 64 bits (no BF16 rounding)."""
    N, ptr, cols, vals, _ = _system(case, seed)
    rows, cols = _rows_of(ptr), cols.to(torch.int64)
    d = vals[rows == cols]
    ah = vals / torch.sqrt(d[rows] * d[cols])
    off, low = rows != cols, rows > cols
    orow, ocol, ow = rows[off], cols[off], ah[off].abs()
    lr, lc, lw = rows[low], cols[low], ah[low].abs()
    zero = torch.zeros(N, device="cuda", dtype=torch.float64)
    feat = torch.stack([zero + 1.0, zero.index_add(0, orow, ow),
                        zero.index_add(0, orow, torch.ones_like(ow)) / 6.0,
                        zero.scatter_reduce(0, orow, ow, "amax")], 1)
    flat = torch.tensor(learned.init_params(int(seed) % (1 << 31)).astype(np.float64),
                        device="cuda", requires_grad=True)
    parts, at = [], 0
    for shp in [(32, 4), (32,)] + 3 * [(32, 64), (32,)] + [(10, 32), (10,)]:
        n = int(np.prod(shp))
        parts.append(flat[at:at + n].reshape(shp))
        at += n

    def spmm(r, c, v, X):
        return torch.zeros_like(X).index_add(0, r, v[:, None] * X[c])

    h = torch.relu(feat @ parts[0].T + parts[1])
    for k in range(3):
        x = torch.cat([h, spmm(orow, ocol, ow, h)], 1)
        h = h + torch.relu(x @ parts[2 + 2 * k].T + parts[3 + 2 * k])
    o = h @ parts[8].T + parts[9]
    gd = torch.nn.functional.softplus(o[:, 1] + 0.5413)
    go = lw * (o[lr, 0] + (o[lr, 2:6] * o[lc, 6:10]).sum(1))
    V = _rademacher(N, _probe_seed(seed))
    for k in range(3):
        s = (V - (2.0 / 3.0) * spmm(rows, cols, ah, V)) * (3.0 if k == 2 else 1.0)
        V = torch.cat([V[:, :4], s[:, 4:]], 1)
    t1 = gd[:, None] * V + spmm(lr, lc, go, V)
    t2 = spmm(rows, cols, ah, t1)
    res = gd[:, None] * t2 + spmm(lc, lr, go, t2) - V
    loss = res.square().sum() / (8.0 * N)
    loss.backward()
    return {"loss": float(loss.detach()), "grad": flat.grad}


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return _system(case, seed)[4]
