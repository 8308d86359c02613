"""HYB products where the longest rows take a block each, and where they do not, at the bounds: rows of 512, 513 and
a few batches of a block (1024 entries), one to many block rows per block, long rows in a matrix whose other rows keep
the warps busy longer (no block rows), y += A x and the residual check beside y = A x.  A row's terms are summed in
some fixed order: the bound is 1e-15 x (row length) x largest product."""
import numpy as np
import pytest


def _matrix(n, lens, seed):
    rng = np.random.default_rng(seed)
    L = np.minimum(np.asarray(lens, dtype=np.int64), n)
    ptr = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(L, out=ptr[1:])
    rows = np.repeat(np.arange(n), L)
    col = ((rows * 13 + (np.arange(rows.size) - ptr[rows].astype(np.int64)) * 7) % n).astype(np.uint32)
    return ptr, col, rng.standard_normal(rows.size), rows, L


CASES = {
    "one long row": (5000, lambda r, n: np.where(np.arange(n) == n - 1, 4097, 3)),
    "at the bound": (2049, lambda r, n: np.where(np.arange(n) % 97 == 5, 513, np.where(np.arange(n) % 89 == 3, 512, 8))),
    "batches": (6000, lambda r, n: np.where(np.arange(n) % 500 == 7, 1023 + np.arange(n) // 500 % 3, r.integers(0, 40, n))),
    "many": (9001, lambda r, n: np.where(r.random(n) < 0.1, r.integers(513, 3000, n), 1)),
    "warps only": (3000, lambda r, n: r.integers(513, 640, n)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CASES))
def test_hyb_block_rows(cuda, pkg, name):
    torch = cuda
    n, lens = CASES[name]
    rng = np.random.default_rng(len(name))
    ptr, col, val, rows, L = _matrix(n, lens(rng, n), n)
    x = rng.standard_normal(n)
    want = np.zeros(n, dtype=np.longdouble)
    np.add.at(want, rows, val.astype(np.longdouble) * x[col].astype(np.longdouble))
    bound = 1e-15 * (L + 1) * max(np.max(np.abs(val)), 1.0) * np.max(np.abs(x))
    A = pkg.Matrix(pkg.Context(), ptr, col, val)
    A.set_format("hyb")
    xd = torch.from_numpy(x).cuda()
    for sigma in (0.0, -1.25):
        y = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
        A.spmv(xd, y, sigma)
        assert np.all(np.abs(y.cpu().numpy() - (want + np.longdouble(sigma) * x).astype(np.float64)) <= bound)
    got = pkg.mult(pkg.workloads.Csr(ptr, col, val), x, np.ones(n))  # (the host call takes the same default form)
    assert np.all(np.abs(got - (want + 1).astype(np.float64)) <= bound + 2.0**-52 * np.abs(want).astype(np.float64))
    res = torch.empty(1, dtype=torch.float64, device="cuda")
    b = torch.ones(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    pkg.true_residuals_noalloc(A, xd[None, :], b, torch.zeros(1, dtype=torch.float64, device="cuda"), res)
    torch.cuda.synchronize()
    exact = float(np.linalg.norm((1 - want).astype(np.float64)) / np.sqrt(n))
    assert abs(float(res[0]) - exact) <= 1e-13 * exact
    A.close()
