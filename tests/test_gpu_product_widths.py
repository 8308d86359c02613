"""SELL-32 products at the edges of the rule that chooses between slices ahead and one at a time (csrc/kernels_blas.cu):
half a million rows, 4.5, 8 and 16 entries per row, the fill of the last wave.  The reference is the sum in torch FP64;
each row may be off by the rounding of its own sum, (terms + 2) * 2^-53 times the sum of its terms' absolute values on
either side."""
import numpy as np
import pytest

EPS = 2.0**-53


def _band(torch, n, w, odd=0):
    """n rows of w diagonals (the last `odd` rows without their outer ones)."""
    off = torch.arange(-(w // 2), w - w // 2, device="cuda")
    col = torch.arange(n, device="cuda")[:, None] + off[None, :]
    keep = (col >= 0) & (col < n)
    if odd:
        keep[n - odd:, 0] = False
    ptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    ptr[1:] = torch.cumsum(keep.sum(1), 0).int()
    val = torch.randn(n, w, device="cuda", dtype=torch.float64, generator=torch.Generator("cuda").manual_seed(n + w))
    return ptr, col[keep].int().contiguous(), val[keep].contiguous(), keep, col.clamp(0, n - 1), val


@pytest.mark.gpu
@pytest.mark.parametrize("n,w", [(1, 1), (33, 3), (20001, 7), (524287, 5), (524288, 5), (524289, 4), (600001, 1), (600001, 8),
                                 (600001, 9), (600001, 16), (1000003, 16), (1000003, 20), (524288, 27)])
@pytest.mark.parametrize("sigma", [0.0, 0.25])
def test_product(cuda, pkg, n, w, sigma):
    torch = cuda
    ptr, col, val, keep, at, full = _band(torch, n, w, odd=min(5, n - 1) if w > 1 else 0)
    x = torch.randn(n, device="cuda", dtype=torch.float64, generator=torch.Generator("cuda").manual_seed(1))
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    A = pkg.Matrix(pkg.Context(), ptr, col, val)
    assert A.format == "sell"
    A.spmv(x, y, sigma)
    terms = torch.where(keep, full * x[at], 0.0)
    want = terms.sum(1) + sigma * x
    size = terms.abs().sum(1) + abs(sigma) * x.abs()
    assert torch.all((y - want).abs() <= 2 * (w + 2) * EPS * size)
    A.close()


@pytest.mark.gpu
def test_rows_of_one_entry_take_their_share_of_the_time(cuda, pkg):
    """A product is bound by its bytes: with one entry per row instead of seven they are 36 instead of 108 per row."""
    torch = cuda
    n, ms = 3000000, {}
    for w in (1, 7):
        ptr, col, val = _band(torch, n, w)[:3]
        x = torch.ones(n, device="cuda", dtype=torch.float64)
        y = torch.empty_like(x)
        torch.cuda.synchronize()
        A = pkg.Matrix(pkg.Context(), ptr, col, val)
        A.time_spmv(x, y, 0.25, 20)
        ms[w] = min(A.time_spmv(x, y, 0.25, 40) for _ in range(5))
        A.close()
    assert ms[1] < 0.55 * ms[7], ms
