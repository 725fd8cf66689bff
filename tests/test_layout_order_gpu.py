"""Layout plans whose offset lists do not ascend: every column is bounded by its
own offset, not by the list's first and last.  The lists here begin and end
with offsets near 0 and hold far ones between them, with non-zero values at the
columns outside [0, n); x lies in a larger buffer with NaN on both sides.
Values are small integers, so sums are exact in any order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BIG, SMALL = 9472 * 128 + 4096 + 17, 20000 + 45  # the first runs the kernels of large layouts


def _plan(lib, n, bw, dtype, sort):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n + bw)
    td = torch.float64 if dtype == "f8" else torch.float32
    offs = torch.tensor([-3, n // 3, 5, -(n // 2), 0, 1, -n + 7, 2, 40, -1, 3], device="cuda")
    if sort:
        offs = offs.sort().values
    K, nb = offs.numel(), -(-n // bw)
    vals = torch.randint(1, 4, (nb, K, bw), generator=gen, device="cuda").to(td)
    r = torch.arange(nb * bw, device="cuda").view(nb, bw)
    vals[(r >= n)[:, None, :].expand(nb, K, bw)] = 0
    arrays = {"values": vals, "offsets": offs.to(torch.int32).repeat(nb), "blockStart": (torch.arange(nb + 1, device="cuda") * K).to(torch.int32)}
    torch.cuda.synchronize()
    plan = lib.LayoutPlan(dtype=np.dtype(dtype).type, numRows=n, numCols=n, blockWidth=bw, numBlocks=nb, totalOffsets=nb * K, numCoo=0,
                          keep=arrays, **{k: t.data_ptr() for k, t in arrays.items()})
    return plan, vals.permute(0, 2, 1).reshape(nb * bw, K)[:n], offs, td


def _want(v, offs, X):
    import torch
    n = v.shape[0]
    r = torch.arange(n, device="cuda")
    Y = torch.zeros((n, X.shape[1]), dtype=torch.float64, device="cuda")
    for k in range(offs.numel()):
        c = r + offs[k]
        ok = (c >= 0) & (c < n)
        Y[ok] += v[ok, k].double()[:, None] * X[c[ok]].double()
    return Y


@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("n,bw,dtype", [(BIG, 32, "f8"), (BIG, 32, "f4"), (BIG, 64, "f8"), (SMALL, 32, "f8"), (SMALL, 32, "f4"), (SMALL, 64, "f4"),
                                        (SMALL, 16, "f8")])
def test_any_offset_order(lib, n, bw, dtype, sort):
    import torch
    plan, v, offs, td = _plan(lib, n, bw, dtype, sort)
    gen = torch.Generator(device="cuda").manual_seed(5)
    for k in (1,) if n == BIG else (1, 2, 3, 4, 8, 9, 16, 24):
        buf = torch.full((3 * n, k), float("nan"), dtype=td, device="cuda")
        X = buf[n:2 * n]
        X.copy_(torch.randint(-3, 4, (n, k), generator=gen, device="cuda"))
        Y = torch.full((n, k), float("nan"), dtype=td, device="cuda")
        torch.cuda.synchronize()
        if k == 1:
            plan.spmv(X.data_ptr(), Y.data_ptr(), 0)
            torch.cuda.synchronize()
            assert torch.equal(Y.double(), _want(v, offs, X))
            Y.fill_(float("nan"))
            torch.cuda.synchronize()
        plan.spmm(X.data_ptr(), k, Y.data_ptr(), k, k, 0)
        torch.cuda.synchronize()
        assert torch.equal(Y.double(), _want(v, offs, X)), k
