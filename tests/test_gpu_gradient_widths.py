"""Gradients of the values at the edges of the rule that chooses between a thread per row and one per entry
(csrc/adjoint_host.c), and over every row length that a warp's code is made for (csrc/adjoint.cu: up to 8 entries at a
time).  The reference is the same sum in torch FP64; each gradient may be off by the rounding of its own sum,
(m + 2) * 2^-53 times the sum of its terms' absolute values on either side."""
import numpy as np
import pytest

EPS = 2.0**-53


def _matrix(torch, n, lens, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    ptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    ptr[1:] = torch.cumsum(lens, 0).int()
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    first = ptr[:-1].long()
    col = (rows + torch.arange(rows.numel(), device="cuda") - first[rows]) % n
    return ptr, col.int().contiguous(), torch.randn(rows.numel(), device="cuda", dtype=torch.float64, generator=g), rows


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,lens", [
    (1, 3, "1"), (97, 2, "1..8"), (4097, 3, "1..8"), (20001, 5, "0..9"), (1000, 3, "17"),
    (7999, 30, "39"), (7999, 29, "39"), (8000, 30, "39"),  # few long rows: 1150 products per row
    (2097152, 3, "1"), (2097153, 3, "1"), (2097153, 2, "2"), (2097153, 3, "2"),  # many rows of one or two entries
])
def test_gradients(cuda, pkg, n, m, lens):
    torch = cuda
    at = torch.arange(n, device="cuda")
    if ".." in lens:
        lo, hi = (int(v) for v in lens.split(".."))
        lens = lo + (at // 32 + at % 3) % (hi - lo + 1)  # (rows of other lengths within a warp, and from warp to warp)
    else:
        lens = torch.full((n,), int(lens), device="cuda")
    lens = lens.clamp(max=n)
    ptr, col, val, rows = _matrix(torch, n, lens, n + m)
    g = torch.Generator("cuda").manual_seed(m)
    X, Y = (torch.randn(m, n, device="cuda", dtype=torch.float64, generator=g) for _ in range(2))
    w = torch.rand(m, device="cuda", dtype=torch.float64, generator=g)
    torch.cuda.synchronize()
    A = pkg.Matrix(pkg.Context(), ptr, col, val)
    A.set_format("sell")
    dval, _, _ = A.adjoint_gradients(X, Y, w)
    want, size = torch.zeros_like(dval), torch.zeros_like(dval)
    for j in range(m):
        t = w[j] * Y[j][rows] * X[j][col.long()]
        want -= t
        size += t.abs()
    assert torch.all((dval - want).abs() <= 2 * (m + 2) * EPS * size)
    A.close()


@pytest.mark.gpu
def test_rows_of_one_entry_take_their_share_of_the_time(cuda, pkg):
    """The sums are bound by the FP64 pipe: 2 operations per row and shift with one entry per row, 8 with seven."""
    torch = cuda
    n, m, us = 1000000, 32, {}
    X, Y = (torch.ones(m, n, device="cuda", dtype=torch.float64) for _ in range(2))
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    for k in (1, 7):
        ptr, col, val, _ = _matrix(torch, n, torch.full((n,), k, device="cuda"), k)
        torch.cuda.synchronize()
        A = pkg.Matrix(pkg.Context(), ptr, col, val)
        assert A.format == "sell"
        best = np.inf
        for _ in range(6):
            start.record()
            A.adjoint_gradients(X, Y, want=("val",))
            end.record()
            torch.cuda.synchronize()
            best = min(best, start.elapsed_time(end))
        us[k] = best
        A.close()
    assert us[1] < 0.75 * us[7], us
