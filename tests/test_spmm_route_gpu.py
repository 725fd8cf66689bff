"""Row-major SpMM on both sides of every limit that decides between lanes that
share rows of X and one lane per row: each column equals that column's SpMV,
bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHORT = np.array([-700, -40, -2, -1, 0, 1, 2, 40, 700])
LONG = np.array([-900, -850, -800, -45, -44, -43, -3, -2, -1, 0, 1, 2, 3, 43, 44, 45, 800, 850, 900])


def _banded(lib, n, offs, dtype, bw, storage):
    rng = np.random.default_rng(n + bw)
    rows = np.repeat(np.arange(n, dtype=np.int64), len(offs))
    cols = rows + np.tile(offs, n)
    keep = (cols >= 0) & (cols < n)
    rows, cols = rows[keep], cols[keep]
    er, ec = rng.integers(0, n, n // 100), rng.integers(0, n, n // 100)
    ok = ~np.isin(ec - er, offs)
    key = np.unique(er[ok] * n + ec[ok])
    rows, cols = np.concatenate([rows, key // n]), np.concatenate([cols, key % n])
    vals = rng.uniform(-1, 1, len(rows))
    vals[rng.random(len(rows)) < 0.05] = 0.0
    o = np.argsort(rows, kind="stable")
    m = lib.HBDIA(rows[o].astype(np.int32), cols[o].astype(np.int32), vals[o].astype(dtype), n, n, dtype=np.dtype(dtype))
    m.convertToHBDIAFormat(bw, 2, upload=False)
    m.prepareForGPU(getattr(lib, storage))
    return m


@pytest.mark.parametrize("n,offs,dtype,bw,storage", [
    (60001, SHORT, "f8", 32, "STORE_NATIVE"), (230001, LONG, "f8", 32, "STORE_NATIVE"), (560001, SHORT, "f8", 32, "STORE_NATIVE"),
    (230001, LONG, "f8", 32, "STORE_F32"), (1200001, LONG, "f8", 32, "STORE_F32"), (90001, SHORT, "f4", 32, "STORE_NATIVE"),
    (230001, SHORT, "f4", 32, "STORE_NATIVE"), (810001, SHORT, "f4", 32, "STORE_NATIVE"), (60001, LONG, "f4", 32, "STORE_NATIVE"),
    (60001, SHORT, "f8", 64, "STORE_NATIVE"), (300001, SHORT, "f8", 64, "STORE_NATIVE"), (510001, LONG, "f8", 96, "STORE_NATIVE"),
    (70001, LONG, "f4", 64, "STORE_NATIVE"), (60001, LONG, "f4", 64, "STORE_NATIVE")])
def test_columns_equal_spmv(lib, n, offs, dtype, bw, storage):
    import torch
    m = _banded(lib, n, offs, dtype, bw, storage)
    td = torch.float64 if dtype == "f8" else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(3)
    X = torch.rand((n, 19), generator=gen, device="cuda", dtype=td) * 2 - 1
    want = torch.empty((19, n), device="cuda", dtype=td)
    m.setKernel(lib.KERNEL_ROWWISE)
    for j in range(19):
        lib.spmv_device(m, X[:, j].contiguous().data_ptr(), want[j].data_ptr(), 0)
    torch.cuda.synchronize()
    want = want.t().contiguous()
    for k in (1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 12, 16, 17, 19):
        for ld in (k, k + 1, k + 4):
            A = torch.full((n, ld), float("nan"), device="cuda", dtype=td)
            B = torch.full((n, ld), float("nan"), device="cuda", dtype=td)
            A[:, :k] = X[:, :k]
            torch.cuda.synchronize()
            lib.spmm_device(m, A.data_ptr(), ld, B.data_ptr(), ld, k, 0)
            torch.cuda.synchronize()
            assert torch.equal(B[:, :k], want[:, :k]), (k, ld)
            assert torch.isnan(B[:, k:]).all(), (k, ld)
