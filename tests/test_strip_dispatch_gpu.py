"""Which kernel runs: the strip kernel on large regular layouts under AUTO, the
others where they are set or a knob of theirs is, the same y from all of them;
partial matrices' column windows, rectangular matrices and caller-owned arrays
among the layouts."""
import numpy as np
import pytest

from conftest import bits_equal
from test_partition_gpu import _emulated

pytestmark = pytest.mark.gpu

OFFS = np.array([-700, -40, -2, -1, 0, 1, 2, 40, 700])


def _rows(rounds):
    """Rows that give every warp of the strip kernel this many strips."""
    import torch
    return int(rounds * torch.cuda.get_device_properties(0).multi_processor_count * 16) * 128 - 51


def _banded(nr, nc, seed, offs=OFFS):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(nr, dtype=np.int64), len(offs))
    cols = rows + np.tile(offs, nr)
    keep = (cols >= 0) & (cols < nc)
    rows, cols = rows[keep], cols[keep]
    er, ec = rng.integers(0, nr, nr // 200), rng.integers(0, nc, nr // 200)
    ok = ~np.isin(ec - er, offs)
    key = np.unique(er[ok] * nc + ec[ok])
    rows, cols = np.concatenate([rows, key // nc]), np.concatenate([cols, key % nc])
    o = np.argsort(rows, kind="stable")
    return rows[o].astype(np.int32), cols[o].astype(np.int32), rng.uniform(-1, 1, len(rows))


def _run(lib, m, x, kern):
    m.setKernel(kern)
    yv = lib.HBDIAVector(np.full(m.getNumRows(), np.nan, x.dtype))
    xv = lib.HBDIAVector(x)
    lib.hbdiaSpMV(m, xv, yv, True, False)
    m.synchronize()
    return yv.toHost(), m.selectedKernel(xv.getDeviceDataPtr())


@pytest.mark.parametrize("storage,dtype,bw", [("STORE_NATIVE", "f8", 32), ("STORE_NATIVE", "f4", 32), ("STORE_F32", "f8", 32),
                                              ("STORE_BF16_SCALED", "f8", 32), ("STORE_F32_QUAD", "f8", 32), ("STORE_BF16_QUAD", "f8", 32),
                                              ("STORE_NATIVE", "f8", 64), ("STORE_NATIVE", "f4", 128), ("STORE_F32", "f8", 96)])
def test_kernel_choice(lib, storage, dtype, bw):
    n = _rows(8)
    rows, cols, vals = _banded(n, n, bw)
    m = lib.HBDIA(rows, cols, vals.astype(dtype), n, n, dtype=np.dtype(dtype))
    m.convertToHBDIAFormat(bw, 2, upload=False)
    m.prepareForGPU(getattr(lib, storage))
    x = np.random.default_rng(1).uniform(-1, 1, n).astype(dtype)
    y, k = _run(lib, m, x, lib.KERNEL_AUTO)
    assert k == lib.KERNEL_STRIP
    quad = storage.endswith("QUAD")
    for kern in (lib.KERNEL_STRIP, lib.KERNEL_PIPE, lib.KERNEL_QUAD, lib.KERNEL_WARP, lib.KERNEL_ROWWISE):
        z, k = _run(lib, m, x, kern)
        want = kern if kern == lib.KERNEL_STRIP else lib.KERNEL_QUAD if quad else kern if bw == 32 else lib.KERNEL_ROWWISE
        assert k == want
        assert bits_equal(z, y), kern
    m.setTuning(lib.TUNE_PREFETCH, 0)  # a knob of the other kernels: they run
    z, k = _run(lib, m, x, lib.KERNEL_AUTO)
    assert k == (lib.KERNEL_STRIP if bw != 32 else lib.KERNEL_PIPE if storage == "STORE_NATIVE" else lib.KERNEL_QUAD)
    assert bits_equal(z, y)


def test_small_layouts(lib):
    n = 4000
    rows, cols, vals = _banded(n, n, 3)
    for bw, auto in ((32, lib.KERNEL_PIPE), (64, lib.KERNEL_ROWWISE), (48, lib.KERNEL_ROWWISE)):
        m = lib.HBDIA(rows, cols, vals, n, n)
        m.convertToHBDIAFormat(bw, 2)
        x = np.random.default_rng(1).uniform(-1, 1, n)
        y, k = _run(lib, m, x, lib.KERNEL_AUTO)
        assert k == auto
        z, k = _run(lib, m, x, lib.KERNEL_STRIP)  # runs where it can read the layout
        assert k == (auto if bw == 48 else lib.KERNEL_STRIP) and bits_equal(z, y)
        z, k = _run(lib, m, x, lib.KERNEL_AUTO)
        assert k == auto and bits_equal(z, y)


@pytest.mark.parametrize("storage,dtype,bw,n,K", [
    ("STORE_NATIVE", "f8", 32, 40000, 1), ("STORE_NATIVE", "f8", 32, 40077, 9), ("STORE_NATIVE", "f4", 32, 50001, 6), ("STORE_NATIVE", "f8", 64, 40045, 7),
    ("STORE_NATIVE", "f8", 96, 60200, 4), ("STORE_NATIVE", "f4", 64, 50033, 31), ("STORE_F32", "f8", 32, 40045, 4), ("STORE_F32", "f8", 64, 40064, 8),
    ("STORE_F32_QUAD", "f8", 32, 40045, 10), ("STORE_F32_QUAD", "f8", 32, 400031, 32), ("STORE_BF16_SCALED", "f8", 32, 40045, 7),
    ("STORE_BF16_QUAD", "f8", 32, 40127, 13), ("STORE_BF16_SCALED", "f8", 32, 400000, 30)])
def test_strip_set_equals_oracle(lib, orc, storage, dtype, bw, n, K):
    """The strip kernel on every layout it can read: lists of every rest, strips
    whose tiles differ, more than 32 offsets, stored zeros under an infinite or
    NaN x, long COO rows."""
    import oracle
    from test_strip_gpu import _matrix
    rows, cols, vals, x = _matrix(n, K, K + bw)
    vals, x = vals.astype(dtype), x.astype(dtype)
    m = lib.HBDIA(rows, cols, vals, n, n, dtype=np.dtype(dtype))
    m.convertToHBDIAFormat(bw, 2, upload=False)
    m.prepareForGPU(getattr(lib, storage))
    ref = orc.convert(rows, cols, vals, n, n, bw, 2)
    if storage == "STORE_NATIVE":
        want = ref.spmv(x)
    else:
        L = ref.layout()
        want = ref.spmv_with_values(L.data.astype(np.float32).astype(np.float64) if "F32" in storage else
                                    oracle.bf16_block_scaled(L.data, L.block_start, bw), x)
    y, k = _run(lib, m, x, lib.KERNEL_STRIP)
    assert k == lib.KERNEL_STRIP
    assert np.isfinite(want).all() and bits_equal(y, want)


@pytest.mark.parametrize("shape", [(1.0, 0.8), (0.9, 1.0)])
@pytest.mark.parametrize("dtype,bw", [("f8", 32), ("f4", 64)])
def test_rectangular(lib, shape, dtype, bw):
    """More rows than columns leave strips without blocks at the end."""
    n = _rows(8)
    nr, nc = int(n * shape[0]), int(n * shape[1])
    rows, cols, vals = _banded(nr, nc, 5)
    m = lib.HBDIA(rows, cols, vals.astype(dtype), nr, nc, dtype=np.dtype(dtype))
    m.convertToHBDIAFormat(bw, 2)
    x = np.random.default_rng(1).uniform(-1, 1, max(nr, nc)).astype(dtype)
    y, k = _run(lib, m, x, lib.KERNEL_AUTO)
    assert k == lib.KERNEL_STRIP
    z, k = _run(lib, m, x, lib.KERNEL_ROWWISE)
    assert bits_equal(z, y)
    assert np.isfinite(y).all()


@pytest.mark.parametrize("storage", ["STORE_F32", "STORE_F32_QUAD"])
def test_partial_windows(lib, storage):
    """Two ranks' partial matrices, x read through each one's column window."""
    n = 2 * _rows(3)
    offs = np.array([-3000, -700, -40, -2, -1, 0, 1, 2, 40, 700, 3000])
    rows, cols, vals = _banded(n, n, 9, offs)
    x = np.random.default_rng(2).uniform(-1, 1, n)
    ya, ranks = _emulated(lib, rows, cols, vals, n, 2, 32, 2, x, storage=getattr(lib, storage))
    for m, w0, win, rb, nl in ranks:
        assert m.selectedKernel(win.data_ptr()) == lib.KERNEL_STRIP
    yb, ranks = _emulated(lib, rows, cols, vals, n, 2, 32, 2, x, lib.KERNEL_WARP, storage=lib.STORE_F32)
    for m, w0, win, rb, nl in ranks:
        assert m.selectedKernel(win.data_ptr()) == lib.KERNEL_WARP
    for a, b in zip(ya, yb):
        assert bits_equal(a, b)


def test_layout_plans(lib):
    """Over the caller's arrays the choice is the matrix's own; a value array
    off a 16-byte boundary is left to the kernels that load single values."""
    import torch
    n = _rows(8)
    rows, cols, vals = _banded(n, n, 4)
    m = lib.HBDIA(rows, cols, vals, n, n)
    m.convertToHBDIAFormat(32, 2)
    L = m.layout()
    dev = {k: torch.from_numpy(np.ascontiguousarray(L[k])).cuda() for k in ("offsets", "block_start", "coo_row", "coo_col", "coo_val", "coo_row_ptr")}
    x = torch.rand(n, dtype=torch.float64, device="cuda")
    ys = []
    for shift, want in ((0, lib.KERNEL_STRIP), (1, lib.KERNEL_PIPE)):
        buf = torch.zeros(len(L["data"]) + shift, dtype=torch.float64, device="cuda")
        buf[shift:] = torch.from_numpy(L["data"]).cuda()
        torch.cuda.synchronize()
        p = lib.LayoutPlan(numRows=n, numCols=n, blockWidth=32, numBlocks=L["num_blocks"], totalOffsets=len(L["offsets"]),
                           numCoo=len(L["coo_row"]), values=buf.data_ptr() + 8 * shift, offsets=dev["offsets"].data_ptr(),
                           blockStart=dev["block_start"].data_ptr(), cooRow=dev["coo_row"].data_ptr(), cooCol=dev["coo_col"].data_ptr(),
                           cooVal=dev["coo_val"].data_ptr(), cooRowPtr=dev["coo_row_ptr"].data_ptr(), keep=(dev, buf))
        assert p.selectedKernel(x.data_ptr()) == want
        y = torch.zeros(n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        p.spmv(x.data_ptr(), y.data_ptr(), 0)
        torch.cuda.synchronize()
        ys.append(y)
    assert torch.equal(ys[0], ys[1])


def test_uneven_shares(lib):
    """Strips whose tiles differ that recur with a period of the warps' stride:
    64^2 planes, 2 strips of 32, on the same warps every time."""
    from hbdia_b200 import generate_stencil27
    nz = -(-_rows(5) // 4096)
    n = 64 * 64 * nz
    rows, cols, vals = generate_stencil27(64, 64, nz, extra_fraction=0.002)
    x = np.random.default_rng(1).uniform(-1, 1, n)
    m = lib.HBDIA(rows, cols, vals, n, n)
    m.convertToHBDIAFormat(32, 2)
    y, k = _run(lib, m, x, lib.KERNEL_AUTO)
    assert k == lib.KERNEL_PIPE
    z, k = _run(lib, m, x, lib.KERNEL_STRIP)
    assert k == lib.KERNEL_STRIP and bits_equal(z, y)


def test_autotuner_tells_sizes_apart(lib):
    """A small matrix's choice is not taken by a large one of the same class that
    the strip kernel can serve."""
    import torch
    lib.autotune_clear()
    got = []
    for n in (4000, _rows(8), _rows(9)):
        rows, cols, vals = _banded(n, n, 3)
        m = lib.HBDIA(rows, cols, vals, n, n)
        m.convertToHBDIAFormat(64, 2)
        x, y = torch.rand(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        r = m.autotune(x.data_ptr(), y.data_ptr())
        m.synchronize()
        got.append((r.kernel, r.fromCache))
        assert m.selectedKernel(x.data_ptr()) == r.kernel
    assert got == [(lib.KERNEL_ROWWISE, 0), (lib.KERNEL_STRIP, 0), (lib.KERNEL_STRIP, 1)]
    lib.autotune_clear()


def test_layout_plan_of_short_lists(lib):
    """Lists that are mostly tails of the pipelined kernel's groups reach the strip
    kernel at the same size through a layout plan as through a matrix."""
    import torch
    n, offs = _rows(3), np.array([-700, -40, -1, 0, 1, 40, 700])
    rows, cols, vals = _banded(n, n, 6, offs)
    m = lib.HBDIA(rows, cols, vals, n, n)
    m.convertToHBDIAFormat(32, 2)
    L = m.layout()
    dev = {k: torch.from_numpy(np.ascontiguousarray(L[k])).cuda() for k in ("data", "offsets", "block_start", "coo_row", "coo_col", "coo_val",
                                                                            "coo_row_ptr")}
    x = torch.rand(n, dtype=torch.float64, device="cuda")
    y, z = torch.zeros_like(x), torch.zeros_like(x)
    torch.cuda.synchronize()
    p = lib.LayoutPlan(numRows=n, numCols=n, blockWidth=32, numBlocks=L["num_blocks"], totalOffsets=len(L["offsets"]), numCoo=len(L["coo_row"]),
                       values=dev["data"].data_ptr(), offsets=dev["offsets"].data_ptr(), blockStart=dev["block_start"].data_ptr(),
                       cooRow=dev["coo_row"].data_ptr(), cooCol=dev["coo_col"].data_ptr(), cooVal=dev["coo_val"].data_ptr(),
                       cooRowPtr=dev["coo_row_ptr"].data_ptr(), keep=dev)
    assert p.selectedKernel(x.data_ptr()) == m.selectedKernel(x.data_ptr()) == lib.KERNEL_STRIP
    p.spmv(x.data_ptr(), y.data_ptr(), 0)
    lib.spmv_device(m, x.data_ptr(), z.data_ptr(), 0)
    torch.cuda.synchronize()
    assert torch.equal(y, z)
