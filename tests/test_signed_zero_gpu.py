"""Sums that underflow to -0: y = dia + coo turns them into +0 at every row of
a matrix with a COO remainder, rows without remainder entries included, and
leaves them -0 in a matrix without one.  All kernels give the oracle's signs."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


def _matrix(n, coo, big, small, seed):
    """Three diagonals of -small; x is small but for one row in 50.  coo: off-pattern entries in one row of 300."""
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n, dtype=np.int64), 3)
    cols = rows + np.tile([-1, 0, 1], n)
    keep = (cols >= 0) & (cols < n)
    rows, cols = rows[keep], cols[keep]
    vals = np.full(len(rows), -big)
    if coo:
        er = np.arange(0, n, 300)
        ec = (er + n // 2) % n
        rows, cols, vals = np.concatenate([rows, er]), np.concatenate([cols, ec]), np.concatenate([vals, -big * np.ones(len(er))])
        o = np.argsort(rows, kind="stable")
        rows, cols, vals = rows[o], cols[o], vals[o]
    x = np.where(rng.random(n) < 0.02, 1.0, small)
    return rows.astype(np.int32), cols.astype(np.int32), vals, x


def _scale(dtype):
    # a stored value and an x whose product underflows (the value within float's range)
    return (1e-30, 1e-30) if dtype == "f4" else (1e-30, 1e-300)


# rows at which the three-offset layouts run the large-matrix kernels, and small ones
@pytest.mark.parametrize("coo", [True, False])
@pytest.mark.parametrize("storage,dtype,bw,n", [
    ("STORE_NATIVE", "f8", 32, 4001), ("STORE_NATIVE", "f8", 32, 700000), ("STORE_NATIVE", "f4", 32, 700000),
    ("STORE_NATIVE", "f8", 64, 700000), ("STORE_NATIVE", "f4", 128, 700000), ("STORE_F32", "f8", 32, 4001), ("STORE_F32", "f8", 32, 1500000),
    ("STORE_F32_QUAD", "f8", 32, 1500000), ("STORE_F32_QUAD", "f8", 32, 4001), ("STORE_BF16_SCALED", "f8", 32, 2200000), ("STORE_BF16_SCALED", "f8", 32, 4001)])
def test_spmv_sign_of_zero(lib, orc, storage, dtype, bw, n, coo):
    import oracle
    big, small = _scale(dtype)
    n = n if coo else n // bw * bw  # (a ragged last block's lone entries are a remainder)
    rows, cols, vals, x = _matrix(n, coo, big, small, n)
    vals, x = vals.astype(dtype), x.astype(dtype)
    ref = orc.convert(rows, cols, vals, n, n, bw, 2)
    if storage == "STORE_NATIVE":
        want = ref.spmv(x)
    else:
        L = ref.layout()
        stored = L.data.astype(np.float32).astype(np.float64) if "F32" in storage else oracle.bf16_block_scaled(L.data, L.block_start, bw)
        want = ref.spmv_with_values(stored, x)
    assert np.signbit(want[want == 0]).all() if not coo else not np.signbit(want[want == 0]).any()
    assert (want == 0).sum() > n // 2
    m = lib.HBDIA(rows, cols, vals, n, n, dtype=np.dtype(dtype))
    m.convertToHBDIAFormat(bw, 2, upload=False)
    m.prepareForGPU(getattr(lib, storage))
    for kern in (lib.KERNEL_AUTO, lib.KERNEL_QUAD, lib.KERNEL_PIPE, lib.KERNEL_WARP, lib.KERNEL_STAGED, lib.KERNEL_ROWWISE):
        m.setKernel(kern)
        yv = lib.HBDIAVector(np.full(n, np.nan, dtype))
        lib.hbdiaSpMV(m, lib.HBDIAVector(x), yv, True, False)
        m.synchronize()
        assert bits_equal(yv.toHost(), want), kern


@pytest.mark.parametrize("coo", [True, False])
@pytest.mark.parametrize("dtype,bw", [("f8", 32), ("f4", 32), ("f8", 64), ("f8", 16)])
def test_spmm_sign_of_zero(lib, orc, dtype, bw, coo):
    import torch
    n = 3017 if coo else 3008
    big, small = _scale(dtype)
    rows, cols, vals, x = _matrix(n, coo, big, small, 7)
    vals = vals.astype(dtype)
    m = lib.HBDIA(rows, cols, vals, n, n, dtype=np.dtype(dtype))
    m.convertToHBDIAFormat(bw, 2)
    ref = orc.convert(rows, cols, vals, n, n, bw, 2)
    X = np.stack([np.roll(x, 37 * j) for j in range(20)], 1).astype(dtype)
    want = np.stack([ref.spmv(np.ascontiguousarray(X[:, j])) for j in range(20)], 1)
    assert (want == 0).any() and np.signbit(want[want == 0]).all() != coo
    Xt = torch.from_numpy(X).cuda()
    for k in (1, 2, 3, 4, 5, 8, 9, 12, 16, 20):
        A = Xt[:, :k].contiguous()
        Y = torch.full((n, k), float("nan"), dtype=A.dtype, device="cuda")
        C = Xt[:, :k].t().contiguous()
        Z = torch.full((k, n), float("nan"), dtype=A.dtype, device="cuda")
        torch.cuda.synchronize()
        lib.spmm_device(m, A.data_ptr(), k, Y.data_ptr(), k, k, 0)
        lib.spmm_device_colmajor(m, C.data_ptr(), n, Z.data_ptr(), n, k, 0)
        m.synchronize()
        assert bits_equal(Y.cpu().numpy(), want[:, :k]), k
        assert bits_equal(Z.cpu().numpy().T.copy(), want[:, :k]), k
