"""The strip SpMV (four 32-row tiles per warp, values streamed through shared
memory), which large regular layouts run: y equals the oracle's bit for bit
for every value storage and block width it takes, at list lengths around its
group of 4 and its limit of 32, with ragged last strips, strips whose tiles
differ (some with more than 32 offsets), stored zeros of either sign under an
infinite or NaN x, and COO rows that cross its 32- and 64-entry chunks."""
import numpy as np
import pytest

from conftest import bits_equal

pytestmark = pytest.mark.gpu


def _matrix(n, K, seed):
    rng = np.random.default_rng(seed)
    offs = np.unique(np.concatenate([[0], rng.permutation(np.r_[-40:41, 700:720, -3000:-2990])[:3 * K]]))
    offs = np.sort(rng.permutation(offs)[:K]).astype(np.int64)
    rows = np.repeat(np.arange(n, dtype=np.int64), K)
    cols = rows + np.tile(offs, n)
    keep = (cols >= 0) & (cols < n)
    # 5 % of the strips lose the first offset of one tile
    lost = rng.random(-(-n // 128)) < 0.05
    k = np.tile(np.arange(K), n)
    keep &= ~(lost[rows // 128] & ((rows // 32) % 4 == 1) & (k == 0))
    rows, cols = rows[keep], cols[keep]
    vals = rng.uniform(0.1, 1.0, len(rows))
    vals[rng.random(len(rows)) < 0.05] = 0.0
    bad = rng.choice(n, 50, replace=False)  # columns of stored zeros only
    at = np.isin(cols, bad)
    vals[at] = np.where(rng.random(at.sum()) < 0.5, 0.0, -0.0)
    # off-pattern entries: scattered ones, one row of 70, runs of three, and one tile with 40 more offsets
    er = np.concatenate([rng.integers(0, n, n // 100), np.full(70, 640), np.repeat(np.arange(1280, 1300), 3),
                         np.repeat(np.arange(2560, 2592), 40)])
    ec = np.concatenate([rng.integers(0, n, n // 100 + 70 + 60), np.tile(20000 + 3 * np.arange(40), 32) + np.repeat(np.arange(32), 40)])
    ok = ~np.isin(ec - er, offs) & ~np.isin(ec, bad)
    key = np.unique(er[ok] * n + ec[ok])
    rows, cols = np.concatenate([rows, key // n]), np.concatenate([cols, key % n])
    vals = np.concatenate([vals, rng.uniform(0.1, 1.0, len(key))])
    o = np.argsort(rows, kind="stable")
    x = rng.uniform(-1, 1, n)
    x[bad] = np.tile([np.inf, -np.inf, np.nan, np.inf, -np.inf], 10)
    return rows[o].astype(np.int32), cols[o].astype(np.int32), vals[o], x


# Rows from which the layouts below run the strip kernel on 148 SMs: native values (fewer where lists are short);
# wide blocks; and FP32 / BF16 storage, whose lists count too
NATIVE, SHORT, HALF = 9472 * 128, 4736 * 128, 1184 * 128
def _fp32(K): return max(HALF, -(-32 * 1024 // K) * 128 * 21 // 20)
def _bf16(K): return max(3552 * 128, -(-48 * 1024 // K) * 128 * 21 // 20)


@pytest.mark.parametrize("storage,dtype,bw,n,K", [
    ("STORE_NATIVE", "f8", 32, SHORT + 77, 3), ("STORE_NATIVE", "f8", 32, NATIVE, 9),
    ("STORE_NATIVE", "f4", 32, SHORT + 1, 6), ("STORE_NATIVE", "f8", 64, HALF + 45, 7),
    ("STORE_NATIVE", "f8", 96, HALF + 200, 4), ("STORE_NATIVE", "f4", 64, HALF + 33, 5),
    ("STORE_F32", "f8", 32, _fp32(4) + 45, 4), ("STORE_F32", "f8", 32, _fp32(31) + 96, 31),
    ("STORE_F32", "f8", 64, _fp32(8) + 64, 8), ("STORE_F32_QUAD", "f8", 32, _fp32(10) + 45, 10),
    ("STORE_F32_QUAD", "f8", 32, _fp32(32) + 31, 32), ("STORE_BF16_SCALED", "f8", 32, _bf16(7) + 45, 7),
    ("STORE_BF16_QUAD", "f8", 32, _bf16(13) + 127, 13)])
def test_strip_equals_oracle(lib, storage, dtype, bw, n, K):
    import oracle
    rows, cols, vals, x = _matrix(n, K, K + bw)
    dt = np.dtype(dtype)
    vals, x = vals.astype(dt), x.astype(dt)
    m = lib.HBDIA(rows, cols, vals, n, n, dtype=dt)
    m.convertToHBDIAFormat(bw, 2, upload=False)
    m.prepareForGPU(getattr(lib, storage))
    ref = oracle.Restated().convert(rows, cols, vals, n, n, bw, 2)
    if storage == "STORE_NATIVE":
        yref = ref.spmv(x)
    else:
        L = ref.layout()
        stored = L.data.astype(np.float32).astype(np.float64) if "F32" in storage else \
            oracle.bf16_block_scaled(L.data, L.block_start, bw)
        yref = ref.spmv_with_values(stored, x)
    yv = lib.HBDIAVector(np.full(n, np.nan, dt))
    lib.hbdiaSpMV(m, lib.HBDIAVector(x), yv, True, False)
    m.synchronize()
    assert np.isfinite(yref).all()
    assert bits_equal(yv.toHost(), yref)


def test_strip_reads_unaligned_layouts_elsewhere(lib):
    """A caller's value array 8 bytes off a 16-byte boundary is served by the
    kernels that load single values: the same y."""
    import torch
    n = NATIVE
    rows, cols, vals, x = _matrix(n, 3, 5)
    m = lib.HBDIA(rows, cols, vals, n, n)
    m.convertToHBDIAFormat(32, 2)
    L = m.layout()
    dev = {k: torch.from_numpy(np.ascontiguousarray(L[k])).cuda() for k in
           ("offsets", "block_start", "coo_row", "coo_col", "coo_val", "coo_row_ptr")}
    xt = torch.from_numpy(x).cuda()
    ys = []
    for shift in (0, 1):
        buf = torch.zeros(len(L["data"]) + shift, dtype=torch.float64, device="cuda")
        buf[shift:] = torch.from_numpy(L["data"]).cuda()
        p = lib.LayoutPlan(numRows=n, numCols=n, blockWidth=32, numBlocks=L["num_blocks"], totalOffsets=len(L["offsets"]),
                           numCoo=len(L["coo_row"]), values=buf.data_ptr() + 8 * shift, offsets=dev["offsets"].data_ptr(),
                           blockStart=dev["block_start"].data_ptr(), cooRow=dev["coo_row"].data_ptr(),
                           cooCol=dev["coo_col"].data_ptr(), cooVal=dev["coo_val"].data_ptr(),
                           cooRowPtr=dev["coo_row_ptr"].data_ptr(), keep=(dev, buf))
        y = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
        p.spmv(xt.data_ptr(), y.data_ptr(), 0)
        torch.cuda.synchronize()
        ys.append(y)
    assert torch.equal(ys[0].view(torch.int64), ys[1].view(torch.int64))
    assert torch.isfinite(ys[0]).all()
