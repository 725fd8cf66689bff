"""Performance cases of the HBDIA library: what a user's program has it do.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
what a program holds before the call (matrices on the device, vectors), run()
is one pass through the public entry points, work() the bytes and operations
of a pass and exact() its result in 64 bits without the library.

Matrices are the library's own workloads: the 27-point stencil (centre 26,
neighbours -1), the 7-point Laplacian (6, -1), a banded matrix with dropped
entries, the symmetric positive definite 27-point stencil of the CG solves --
each with off-pattern extras where its workload has them, which end up in the
COO remainder.  Everything random comes from the seed.
"""
import math

import torch

import hbdia_b200 as hb

BANDS = (-4096, -64, -2, -1, 0, 1, 2, 64, 4096)
STORAGE = {"native": hb.STORE_NATIVE, "f32": hb.STORE_F32, "bf16": hb.STORE_BF16_SCALED, "f32_quad": hb.STORE_F32_QUAD}
VALUE_BYTES = {"native": 8, "f32": 4, "bf16": 2, "f32_quad": 4}
# Iterations of a CG solve to 1e-10 on the SPD stencil (its condition number
# depends on the diagonal shift, hardly on the grid): for work() alone.
CG_ITERATIONS = 300


def listed():
    return [
        # The smallest call: a coarse grid's product, launch and latency alone.
        {"name": "spmv_small", "kind": "spmv", "matrix": "stencil27", "nx": 16, "ny": 16, "nz": 16, "extras": 0.005,
         "dtype": "f64", "storage": "native", "bw": 32, "plan": False},
        # A 64^3 stencil product: matrix and vectors fit in the L2 cache.
        {"name": "spmv_f64_64", "kind": "spmv", "matrix": "stencil27", "nx": 64, "ny": 64, "nz": 64, "extras": 0.005,
         "dtype": "f64", "storage": "native", "bw": 32, "plan": False},
        # The headline product: 16.8 M rows, x larger than L2, over device arrays that the caller owns.
        {"name": "spmv_f64_256", "kind": "spmv", "matrix": "stencil27", "nx": 256, "ny": 256, "nz": 256,
         "extras": 0.01, "dtype": "f64", "storage": "native", "bw": 32, "plan": True},
        # A banded matrix with gaps and a ragged last block, values kept in 32 bits.
        {"name": "spmv_banded_f32store", "kind": "spmv", "matrix": "banded", "nx": 7999993, "ny": 1, "nz": 1,
         "extras": 0.002, "dtype": "f64", "storage": "f32", "bw": 32, "plan": False},
        # Values as scaled bfloat16 on an odd grid: blocks straddle grid lines.
        {"name": "spmv_bf16store_odd", "kind": "spmv", "matrix": "stencil27", "nx": 131, "ny": 127, "nz": 125,
         "extras": 0.005, "dtype": "f64", "storage": "bf16", "bw": 32, "plan": False},
        # A single-precision matrix (HBDIA<float>) on an odd grid.
        {"name": "spmv_float_odd", "kind": "spmv", "matrix": "stencil27", "nx": 129, "ny": 121, "nz": 133,
         "extras": 0.01, "dtype": "f32", "storage": "native", "bw": 32, "plan": False},
        # The Laplacian in wider blocks than the default.
        {"name": "spmv_laplace_bw64", "kind": "spmv", "matrix": "stencil7", "nx": 160, "ny": 160, "nz": 160,
         "extras": 0.0, "dtype": "f64", "storage": "native", "bw": 64, "plan": False},
        # Many right-hand sides side by side in memory (row-major), Laplacian 128^3.
        {"name": "spmm_row_k16", "kind": "spmm", "matrix": "stencil7", "nx": 128, "ny": 128, "nz": 128, "extras": 0.0,
         "dtype": "f64", "storage": "native", "k": 16, "layout": "row"},
        # Many right-hand sides, each a contiguous vector (column-major), 27-point 128^3.
        {"name": "spmm_col_k8", "kind": "spmm", "matrix": "stencil27", "nx": 128, "ny": 128, "nz": 128,
         "extras": 0.01, "dtype": "f64", "storage": "native", "k": 8, "layout": "col"},
        # A server's batch: separate vectors of one resident matrix, values in 32 bits.
        {"name": "spmv_list_f32store_k16", "kind": "spmm", "matrix": "stencil27", "nx": 96, "ny": 96, "nz": 96,
         "extras": 0.005, "dtype": "f64", "storage": "f32", "k": 16, "layout": "list"},
        # A whole CG solve to 1e-10, iterations on 32-bit values with FP64 residual updates (the default).
        {"name": "cg_128", "kind": "cg", "nx": 128, "ny": 128, "nz": 128, "extras": 0.0},
        # Uneven matrices computed as one replayed unit.
        {"name": "batch_24", "kind": "batch", "count": 24, "edge_lo": 16, "edge_hi": 96, "edge_seed": 4},
    ]


def draw(rng):
    def edge(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(lo, hi):
        e = edge(lo, hi)
        return {d: max(lo, min(hi, e + rng.randint(-(e // 8), e // 8))) for d in ("nx", "ny", "nz")}

    kind = rng.choice(["spmv", "spmv", "spmv", "spmm", "spmm", "cg", "batch"])
    if kind == "cg":
        return {"kind": "cg", **grid(24, 112), "extras": rng.choice([0.0, 0.005])}
    if kind == "batch":
        lo = rng.randint(12, 32)
        return {"kind": "batch", "count": rng.randint(4, 24), "edge_lo": lo, "edge_hi": rng.randint(lo + 8, 88),
                "edge_seed": rng.randrange(1 << 20)}
    dtype = rng.choice(["f64", "f64", "f64", "f32"])
    if kind == "spmm":
        storage = rng.choice(["native", "f32"]) if dtype == "f64" else "native"
        return {"kind": "spmm", "matrix": rng.choice(["stencil7", "stencil27"]), **grid(16, 128),
                "extras": rng.choice([0.0, 0.005, 0.01]), "dtype": dtype, "storage": storage,
                "k": edge(2, 32), "layout": rng.choice(["row", "col", "list"])}
    storage = rng.choice(["native", "native", "f32", "bf16", "f32_quad"]) if dtype == "f64" else "native"
    matrix = rng.choice(["stencil27", "stencil27", "stencil7", "banded"])
    size = {"nx": edge(4000, 8000000), "ny": 1, "nz": 1} if matrix == "banded" else grid(16, 160)
    bw = rng.choice([32, 32, 32, 64, 16]) if storage == "native" else 32
    return {"kind": "spmv", "matrix": matrix, **size, "extras": rng.choice([0.0, 0.002, 0.01]), "dtype": dtype,
            "storage": storage, "bw": bw, "plan": bool(matrix != "banded" and storage == "native" and bw == 32
                                                       and rng.random() < 0.25)}


# ---------------------------------------------------------------- matrices
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1) % (1 << 62))


def _uniform(shape, gen, dtype=torch.float64):
    return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64).mul_(2.0).sub_(1.0).to(dtype)


def _stencil_mask(case, g):
    """[n, points] neighbour-inside-the-grid mask and the points' offsets, ascending."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = torch.arange(nx * ny * nz, device="cuda")
    x, y, z = r % nx, (r // nx) % ny, r // (nx * ny)
    pts = [(a, b, c) for c in (-1, 0, 1) for b in (-1, 0, 1) for a in (-1, 0, 1)
           if g == 27 or abs(a) + abs(b) + abs(c) <= 1]
    mask = torch.empty((r.numel(), len(pts)), dtype=torch.bool, device="cuda")
    for i, (a, b, c) in enumerate(pts):
        mask[:, i] = (x + a >= 0) & (x + a < nx) & (y + b >= 0) & (y + b < ny) & (z + c >= 0) & (z + c < nz)
    return mask, [(c * ny + b) * nx + a for a, b, c in pts]


def _extras(case, nnz, n, offsets, gen):
    """Off-pattern entries: sorted unique keys row * n + col, and values U(0.1, 1)."""
    m = int(case["extras"] * nnz)
    rows = torch.randint(0, n, (m,), generator=gen, device="cuda")
    cols = torch.randint(0, n, (m,), generator=gen, device="cuda")
    on = torch.isin(cols - rows, torch.tensor(offsets, device="cuda"))
    keys = torch.unique(rows[~on] * n + cols[~on])
    return keys, torch.rand(keys.numel(), generator=gen, device="cuda", dtype=torch.float64) * 0.9 + 0.1


def _join(rows, cols, vals, keys, kvals, n):
    if keys.numel() == 0:
        return rows, cols, vals
    key, order = torch.sort(torch.cat([rows * n + cols, keys]))
    return key // n, key % n, torch.cat([vals, kvals])[order]


def coo(case, seed):
    """The case's matrix as row-sorted COO on the GPU: rows, cols, float64 values, and n."""
    gen = _gen(seed)
    if case["kind"] == "cg":
        return _spd(case, gen)
    if case["matrix"] == "banded":
        n = case["nx"]
        r = torch.arange(n, device="cuda")
        mask = torch.stack([(r + o >= 0) & (r + o < n) for o in BANDS], 1)
        mask &= torch.rand(mask.shape, generator=gen, device="cuda") >= 0.3
        w = torch.rand(mask.shape, generator=gen, device="cuda", dtype=torch.float64).add_(0.5).mul_(mask)
        mid = BANDS.index(0)
        w[:, mid] = torch.where(mask[:, mid], w.sum(1) - w[:, mid] + 1.0, w[:, mid])
        offsets = list(BANDS)
    else:
        g = 27 if case["matrix"] == "stencil27" else 7
        mask, offsets = _stencil_mask(case, g)
        n = mask.shape[0]
        w = torch.full((len(offsets),), -1.0, dtype=torch.float64, device="cuda")
        w[len(offsets) // 2] = float(g - 1)
    at = mask.nonzero()
    rows, cols = at[:, 0], at[:, 0] + torch.tensor(offsets, device="cuda")[at[:, 1]]
    vals = w[at[:, 0], at[:, 1]] if w.dim() == 2 else w[at[:, 1]]
    del at
    keys, kvals = _extras(case, rows.numel(), n, offsets, gen)
    return (*_join(rows, cols, vals, keys, kvals, n), n)


def _grid20(t):
    return torch.round(t * 2.0 ** 20) / 2.0 ** 20


def _spd(case, gen):
    """Symmetric random off-diagonals -(0.5 + u), symmetric extras, diagonal 1.001 * row |sum|.

    The values are multiples of 2^-20, so that sums over them and products with
    a vector of such multiples are exact in any order."""
    mask, offsets = _stencil_mask(case, 27)
    n = mask.shape[0]
    up = mask[:, 14:].nonzero()
    r, c = up[:, 0], up[:, 0] + torch.tensor(offsets[14:], device="cuda")[up[:, 1]]
    v = -_grid20(0.5 + torch.rand(r.numel(), generator=gen, device="cuda", dtype=torch.float64))
    keys, kvals = _extras({"extras": case["extras"] / 2}, 2 * r.numel(), n, offsets, gen)
    a, b = torch.minimum(keys // n, keys % n), torch.maximum(keys // n, keys % n)
    keys = torch.unique(a * n + b)
    r, c, v = torch.cat([r, keys // n]), torch.cat([c, keys % n]), torch.cat([v, -_grid20(kvals[: keys.numel()])])
    rows, cols, vals = torch.cat([r, c]), torch.cat([c, r]), torch.cat([v, v])
    d = torch.arange(n, device="cuda")
    diag = _grid20(torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, rows, vals.abs()).mul_(1.001))
    key, order = torch.sort(torch.cat([rows * n + cols, d * n + d]))
    return key // n, key % n, torch.cat([vals, diag])[order], n


def _matrix(case, parts, bw=32):
    """The matrix converted on the device (on the host where only the host converter builds it)."""
    import numpy as np
    rows, cols, vals, n = parts
    dt = np.float32 if case.get("dtype") == "f32" else np.float64
    m = hb.HBDIA(rows.to(torch.int32).cpu().numpy(), cols.to(torch.int32).cpu().numpy(),
                 vals.to(torch.float32 if dt == np.float32 else torch.float64).cpu().numpy(), n, n, dtype=dt)
    storage = case.get("storage", "native")
    if case["kind"] == "cg":
        m.convertToHBDIAFormat(bw, 2)
    elif storage == "f32_quad":
        m.convertToHBDIAFormat(bw, 2, upload=False)
        m.prepareForGPU(STORAGE[storage])
    else:
        m.convertOnDevice(bw, 2, storage=STORAGE[storage])
    return m


def _layout_plan(case, seed):
    """The stencil's HBDIA device arrays, built with torch, under a LayoutPlan (threshold 2)."""
    import numpy as np
    g = 27 if case["matrix"] == "stencil27" else 7
    f32 = case["dtype"] == "f32"
    dt = torch.float32 if f32 else torch.float64
    mask, offsets = _stencil_mask(case, g)
    n, p = mask.shape
    w = torch.full((p,), -1.0, dtype=dt, device="cuda")
    w[p // 2] = float(g - 1)
    nnz = int(mask.sum())
    nb = -(-n // 32)
    pad = torch.zeros((nb * 32, p), dtype=torch.bool, device="cuda")
    pad[:n] = mask
    pad = pad.view(nb, 32, p)
    keep = pad.sum(1) >= 2
    lone = (pad & ~keep[:, None, :]).view(nb * 32, p).nonzero()
    at = keep.nonzero()
    off = torch.tensor(offsets, device="cuda")
    offs = off[at[:, 1]].to(torch.int32)
    values = pad.permute(0, 2, 1)[keep].to(dt).mul_(w[at[:, 1]][:, None])
    start = torch.zeros(nb + 1, dtype=torch.int32, device="cuda")
    start[1:] = keep.sum(1).cumsum(0)
    keys, kvals = _extras(case, nnz, n, offsets, _gen(seed))
    r, c, v = _join(lone[:, 0], lone[:, 0] + off[lone[:, 1]], w[lone[:, 1]].double(), keys, kvals, n)
    row_ptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    row_ptr[1:] = torch.bincount(r, minlength=n).cumsum(0)
    arrays = {"values": values, "offsets": offs, "blockStart": start, "cooRow": r.to(torch.int32),
              "cooCol": c.to(torch.int32), "cooVal": v.to(dt), "cooRowPtr": row_ptr}
    del mask, pad, at, lone
    torch.cuda.synchronize()
    return hb.LayoutPlan(dtype=np.float32 if f32 else np.float64, numRows=n, numCols=n, blockWidth=32, numBlocks=nb,
                         totalOffsets=offs.numel(), numCoo=r.numel(), keep=arrays,
                         **{k: t.data_ptr() if t.numel() else 0 for k, t in arrays.items()}), n


def _batch_edges(case):
    import random
    r = random.Random(case["edge_seed"])
    return [r.randint(case["edge_lo"], case["edge_hi"]) for _ in range(case["count"])]


def _batch_member(edge):
    return {"kind": "spmv", "matrix": "stencil27", "nx": edge, "ny": edge, "nz": edge, "extras": 0.005,
            "dtype": "f64", "storage": "native"}


def _vectors(case, seed, n):
    """The right-hand sides of a product, in the case's layout."""
    dt = torch.float32 if case.get("dtype") == "f32" else torch.float64
    gen = _gen(seed + 500)
    if case["kind"] == "spmv":
        return _uniform(n, gen, dt)
    X = _uniform((case["k"], n), gen, dt)
    return {"row": lambda: X.t().contiguous(), "col": lambda: X, "list": lambda: [X[j].clone() for j in
                                                                                range(case["k"])]}[case["layout"]]()


# ---------------------------------------------------------------- the contract
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        edges = _batch_edges(case)
        parts = [_batch_member(e) for e in edges]
        mats = [_matrix(p, coo(p, seed + 7919 * i)) for i, p in enumerate(parts)]
        xs = [_vectors(p, seed + 7919 * i, e ** 3) for (i, p), e in zip(enumerate(parts), edges)]
        ys = [torch.zeros_like(x) for x in xs]
        batch = hb.Batch(mats)
        batch.bind([x.data_ptr() for x in xs], [y.data_ptr() for y in ys])
        state = {"kind": kind, "batch": batch, "x": xs, "y": ys}
    elif kind == "cg":
        parts = coo(case, seed)
        b = _product(*parts[:3], _grid20(_uniform(parts[3], _gen(seed + 500))), parts[3])  # exact: A * solution
        m = _matrix(case, parts)
        state = {"kind": kind, "m": m, "b": b, "x": torch.zeros_like(b), "stream": torch.cuda.Stream()}
    else:
        if case.get("plan"):
            m, n = _layout_plan(case, seed)
        else:
            parts = coo(case, seed)
            n = parts[3]
            m = _matrix(case, parts, case.get("bw", 32))
            del parts
        x = _vectors(case, seed, n)
        y = [torch.zeros_like(t) for t in x] if isinstance(x, list) else torch.zeros_like(x)
        state = {"kind": kind, "m": m, "x": x, "y": y, "n": n, "k": case.get("k", 1), "layout": case.get("layout"),
                 "plan": bool(case.get("plan"))}
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return state


def run(state):
    stream = torch.cuda.current_stream().cuda_stream
    kind = state["kind"]
    if kind == "batch":
        state["batch"].run(stream)
        return state["y"]
    if kind == "cg":
        with torch.cuda.stream(state["stream"]):  # a stream that can be captured; the call returns when the solve is done
            state["x"].zero_()
        hb.cg_solve(state["m"], state["b"].data_ptr(), state["x"].data_ptr(), stream=state["stream"].cuda_stream)
        return state["x"]
    m, x, y, k, n = state["m"], state["x"], state["y"], state["k"], state["n"]
    if kind == "spmv" and state["plan"]:
        m.spmv(x.data_ptr(), y.data_ptr(), stream)
    elif kind == "spmv":
        hb.spmv_device(m, x.data_ptr(), y.data_ptr(), stream)
    elif state["layout"] == "row":
        hb.spmm_device(m, x.data_ptr(), k, y.data_ptr(), k, k, stream)
    elif state["layout"] == "col":
        hb.spmm_device_colmajor(m, x.data_ptr(), n, y.data_ptr(), n, k, stream)
    else:
        hb.spmv_list_device(m, [t.data_ptr() for t in x], [t.data_ptr() for t in y], stream)
    return y


def _nnz(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case.get("matrix") == "banded":
        return 0.7 * sum(max(0, nx - abs(o)) for o in BANDS)
    if case.get("matrix") == "stencil7":
        return 7 * nx * ny * nz - 2 * (nx * ny + ny * nz + nx * nz)
    return (3 * nx - 2) * (3 * ny - 2) * (3 * nz - 2)


def _spmv_work(case, value, vec, k=1):
    """Every value once, one offset per 32 values, x in and y out; extras: row, column, value."""
    n, nnz = case["nx"] * case["ny"] * case["nz"], _nnz(case)
    extras = case["extras"] * nnz
    return {"bytes": nnz * (value + 4 / 32) + 2 * k * vec * n + extras * (8 + vec), "flops": 2 * k * (nnz + extras)}


def work(case):
    if case["kind"] == "batch":
        parts = [_spmv_work(_batch_member(e), 8, 8) for e in _batch_edges(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if case["kind"] == "cg":
        # per iteration: the 32-bit values, p and q of the product, x, r and p of the updates
        n = case["nx"] * case["ny"] * case["nz"]
        w = _spmv_work(case, 4, 8)
        return {"bytes": CG_ITERATIONS * (w["bytes"] + 6 * 8 * n), "flops": CG_ITERATIONS * (w["flops"] + 10 * n)}
    vec = 4 if case["dtype"] == "f32" else 8
    return _spmv_work(case, min(vec, VALUE_BYTES[case["storage"]]), vec, case.get("k", 1))


def _product(rows, cols, vals, x, n):
    y = torch.zeros(n, dtype=torch.float64, device="cuda")
    step = 1 << 26
    for i in range(0, rows.numel(), step):
        y.index_add_(0, rows[i:i + step], vals[i:i + step] * x[cols[i:i + step]])
    return y


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for i, e in enumerate(_batch_edges(case)):
            p = _batch_member(e)
            rows, cols, vals, n = coo(p, seed + 7919 * i)
            out.append(_product(rows, cols, vals, _vectors(p, seed + 7919 * i, n), n))
        return out
    if kind == "cg":
        return _grid20(_uniform(case["nx"] * case["ny"] * case["nz"], _gen(seed + 500)))
    rows, cols, vals, n = coo(case, seed)
    if case["dtype"] == "f32":
        vals = vals.float().double()
    x = _vectors(case, seed, n)
    if kind == "spmv":
        return _product(rows, cols, vals, x.double(), n)
    layout = case["layout"]
    columns = [x[:, j] if layout == "row" else x[j] for j in range(case["k"])]
    ys = [_product(rows, cols, vals, c.double().contiguous(), n) for c in columns]
    if layout == "list":
        return ys
    return torch.stack(ys, 1 if layout == "row" else 0)
