"""BF16 values with a block scale of zero, infinity or NaN: a product counts by
its widened value (stored * scale), so 0 * infinity is NaN in every kernel and
a scale of zero skips a product even under an infinite x."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


def _same(a, b):
    na, nb = np.isnan(a), np.isnan(b)
    return np.array_equal(na, nb) and bits_equal(np.where(na, 0, a), np.where(nb, 0, b))


@pytest.mark.parametrize("storage", ["STORE_BF16_SCALED", "STORE_BF16_QUAD"])
@pytest.mark.parametrize("n", [2200000 + 45, 5000])  # the first runs the kernel of large layouts
def test_block_maximum_outside_float(lib, orc, storage, n):
    import oracle
    rng = np.random.default_rng(n)
    rows = np.repeat(np.arange(n, dtype=np.int64), 5)
    cols = rows + np.tile([-40, -1, 0, 1, 700], n)
    keep = (cols >= 0) & (cols < n)
    rows, cols = rows[keep], cols[keep]
    vals = rng.uniform(0.1, 1.0, len(rows))
    vals[rng.random(len(rows)) < 0.1] = 0.0
    blk = rows // 32
    for b, v in ((20, 1e39), (41, 1e-60), (62, -1e300), (64, 1e-310), (149, 1e60)):  # scales inf and 0
        at = np.flatnonzero(blk == b)
        vals[at] = np.where(vals[at] == 0, 0.0, v)
    rows, cols = rows.astype(np.int32), cols.astype(np.int32)
    x = rng.uniform(-1, 1, n)
    ref = orc.convert(rows, cols, vals, n, n, 32, 2)
    L = ref.layout()
    with np.errstate(all="ignore"):
        want = ref.spmv_with_values(oracle.bf16_block_scaled(L.data, L.block_start, 32), x)
    assert np.isnan(want).sum() >= 5 * 32 - 5
    m = lib.HBDIA(rows, cols, vals, n, n)
    m.convertToHBDIAFormat(32, 2, upload=False)
    m.prepareForGPU(getattr(lib, storage))
    for kern in (lib.KERNEL_AUTO, lib.KERNEL_QUAD, lib.KERNEL_WARP):
        m.setKernel(kern)
        yv = lib.HBDIAVector(np.zeros(n))
        lib.hbdiaSpMV(m, lib.HBDIAVector(x), yv, True, False)
        m.synchronize()
        assert _same(yv.toHost(), want), kern


@pytest.mark.parametrize("n", [2200000, 5024])
def test_caller_scales(lib, n):
    """A caller's scales: zero, infinite and NaN ones beside ordinary ones."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(3)
    offs = torch.tensor([-2, -1, 0, 1, 2, 3, 64, 100], device="cuda")
    nb, K = -(-n // 32), offs.numel()
    stored = torch.randint(0, 3, (nb, K, 32), generator=gen, device="cuda").to(torch.bfloat16)
    scales = torch.full((nb,), 2.0, device="cuda")
    scales[10], scales[21], scales[32], scales[44:48] = 0.0, float("inf"), float("nan"), 0.0
    arrays = {"values": stored, "scales": scales, "offsets": offs.to(torch.int32).repeat(nb),
              "blockStart": (torch.arange(nb + 1, device="cuda") * K).to(torch.int32)}
    x = torch.randint(-2, 3, (n,), generator=gen, device="cuda").double()
    x[32 * 10 + 5], x[32 * 45 + 7], x[32 * 21 + 3] = float("inf"), float("inf"), 0.0
    torch.cuda.synchronize()
    plan = lib.LayoutPlan(storage=lib.STORE_BF16_SCALED, numRows=n, numCols=n, blockWidth=32, numBlocks=nb, totalOffsets=nb * K, numCoo=0,
                          keep=arrays, **{k: t.data_ptr() for k, t in arrays.items()})
    v = (stored.double() * scales.double()[:, None, None]).permute(0, 2, 1).reshape(nb * 32, K)[:n]
    r = torch.arange(n, device="cuda")
    want = torch.zeros(n, dtype=torch.float64, device="cuda")
    for k in range(K):
        c = r + offs[k]
        ok = (c >= 0) & (c < n) & (v[:, k] != 0)
        want[ok] += v[ok, k] * x[c[ok]]
    want = want.cpu().numpy()
    assert np.isfinite(want[32 * 44:32 * 48]).all() and np.isnan(want[32 * 32:32 * 33]).any()
    y = torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    plan.spmv(x.data_ptr(), y.data_ptr(), 0)
    torch.cuda.synchronize()
    assert _same(y.cpu().numpy(), want)
    for k in (1, 2, 3, 4, 8, 16) if n < 10000 else (2,):
        X = x[:, None].repeat(1, k).contiguous()
        Y = torch.zeros((n, k), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        plan.spmm(X.data_ptr(), k, Y.data_ptr(), k, k, 0)
        torch.cuda.synchronize()
        for j in range(k):
            assert _same(Y[:, j].contiguous().cpu().numpy(), want), (k, j)
