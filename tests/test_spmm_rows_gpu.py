"""The row-major SpMM on blocks whose width is a multiple of 32: every column
equals the SpMV of that column bit for bit, for column counts around each of
its lane groupings and above one pass, odd and padded leading dimensions,
unaligned blocks, a ragged last tile, a block of more than 32 offsets, stored
zeros under an infinite X, and COO rows with many entries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(n, seed):
    rng = np.random.default_rng(seed)
    offs = np.array([-700, -33, -2, -1, 0, 1, 2, 3, 40, 699])
    rows = np.repeat(np.arange(n, dtype=np.int64), len(offs))
    cols = rows + np.tile(offs, n)
    keep = (cols >= 0) & (cols < n) & (rng.random(len(rows)) > 0.1)
    rows, cols = rows[keep], cols[keep]
    vals = rng.uniform(0.1, 1.0, len(rows))
    vals[rng.random(len(rows)) < 0.05] = 0.0
    bad = rng.choice(n, 20, replace=False)  # columns of stored zeros only
    vals[np.isin(cols, bad)] = 0.0
    er = np.concatenate([rng.integers(0, n, n // 20), np.full(50, 70), np.repeat(np.arange(128, 160), 40)])
    ec = np.concatenate([rng.integers(0, n, n // 20 + 50), np.tile(900 + 3 * np.arange(40), 32) + np.repeat(np.arange(32), 40)])
    ok = ~np.isin(ec - er, offs) & ~np.isin(ec, bad)
    key = np.unique(er[ok] * n + ec[ok])
    rows, cols = np.concatenate([rows, key // n]), np.concatenate([cols, key % n])
    vals = np.concatenate([vals, rng.uniform(0.1, 1.0, len(key))])
    o = np.argsort(rows, kind="stable")
    return rows[o].astype(np.int32), cols[o].astype(np.int32), vals[o], bad


@pytest.mark.parametrize("storage,dtype,bw", [("STORE_NATIVE", "f8", 32), ("STORE_NATIVE", "f4", 32), ("STORE_F32", "f8", 32),
                                              ("STORE_BF16_SCALED", "f8", 32), ("STORE_NATIVE", "f8", 64), ("STORE_NATIVE", "f4", 96)])
def test_row_major_columns_equal_spmv(lib, storage, dtype, bw):
    import torch
    n = 3000 + 17
    rows, cols, vals, bad = _matrix(n, bw)
    dt = np.dtype(dtype)
    td = torch.float64 if dtype == "f8" else torch.float32
    m = lib.HBDIA(rows, cols, vals.astype(dt), n, n, dtype=dt)
    m.convertToHBDIAFormat(bw, 2, upload=False)
    m.prepareForGPU(getattr(lib, storage))
    gen = torch.Generator(device="cuda").manual_seed(3)
    X = torch.rand((n, 72), generator=gen, device="cuda", dtype=td) * 2 - 1
    X[torch.from_numpy(bad).cuda()] = float("inf")
    want = torch.empty((72, n), device="cuda", dtype=td)
    for j in range(72):
        lib.spmv_device(m, X[:, j].contiguous().data_ptr(), want[j].data_ptr(), 0)
    torch.cuda.synchronize()
    assert torch.isfinite(want).all()
    want = want.t().contiguous()
    for k in (1, 2, 3, 4, 5, 6, 8, 9, 12, 16, 17, 20, 24, 31, 32, 33, 36, 64):
        for ldx, ldy, shift in ((k, k, 0), (k + 1, k + 3, 0), (k + 4, k + 8, 0), (k + 4, k + 4, 1)):
            A = torch.full((n * ldx + shift,), float("nan"), device="cuda", dtype=td)
            B = torch.full((n * ldy + shift,), float("nan"), device="cuda", dtype=td)
            A[shift:].view(n, ldx)[:, :k] = X[:, :k]
            es = A.element_size()
            lib.spmm_device(m, A.data_ptr() + es * shift, ldx, B.data_ptr() + es * shift, ldy, k, 0)
            torch.cuda.synchronize()
            Y = B[shift:].view(n, ldy)
            assert torch.equal(Y[:, :k], want[:, :k]), (k, ldx, ldy, shift)
            assert torch.isnan(Y[:, k:]).all(), (k, ldx, ldy, shift)
