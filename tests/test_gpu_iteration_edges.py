"""The fused iteration and the SELL-32 product at the sizes where their kernels change path.

Iteration: one to several passes of the shift update (64 shifts each), more shifts than a block has threads in the
scalar stages, fewer rows than a warp, blocks of 128..1024 threads.  The reference is the oracle; the bar is the
repository's (1e-8 of each solution's largest value).  Product: row lengths around the entries that the slice pipeline
keeps ahead (7 and 8) up to the 64 of a SELL-32 row, empty rows, n around whole slices, blocks and waves; a row is
summed in stored order with FMAs, so that 1e-15 of (row length x largest product) bounds any rounding."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("dims,m,mode", [
    ((3, 2, 2), 2, "incremental"), ((3, 3, 3), 1, "incremental"), ((9, 8, 7), 65, "incremental"),
    ((8, 8, 8), 130, "incremental"), ((8, 8, 8), 300, "incremental"), ((8, 9, 8), 300, "deferred"),
    ((31, 30, 29), 5, "incremental"), ((60, 61, 62), 3, "deferred"), ((41, 37, 1), 9, "incremental"),
    ((211, 198, 1), 6, "deferred"),
])
def test_iteration_edges(cuda, pkg, oracle, dims, m, mode):
    a = pkg.workloads.stencil_cd3d(*dims)
    b = np.random.default_rng(m).standard_normal(a.n)
    sigma = np.linspace(0.02, 1.5, m)
    want = oracle.solve(a, b, sigma, seed=0, tol=1e-10, max_iter=2000)
    got = pkg.solve(a, b, sigma, seed=0, tol=1e-10, max_iter=2000, shift_mode=mode)
    assert got.status == 0
    scale = np.max(np.abs(want.x), axis=1)
    assert np.all(np.max(np.abs(got.x - want.x), axis=1) <= 1e-8 * scale)


@pytest.mark.gpu
@pytest.mark.parametrize("n,lens", [
    (1, [1]), (31, [7]), (33, [8, 0, 7]), (64, [64]), (255, [9, 1]), (257, [8]), (1000, [0, 3, 15, 16, 17]),
    (116737, [7, 7, 7, 9]), (250001, [5]), (524287, [3, 6]), (524288, [5, 5, 6]), (600001, [0, 4, 5, 12]),
    (700003, [7, 8, 5, 9]),
])
@pytest.mark.parametrize("sigma", [0.0, 0.75])
def test_sell_product_edges(cuda, pkg, n, lens, sigma):
    torch = cuda
    rng = np.random.default_rng(n)
    L = np.minimum(np.resize(lens, n), n).astype(np.int64)
    ptr = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(L, out=ptr[1:])
    rows = np.repeat(np.arange(n), L)
    col = ((rows * 7 + (np.arange(rows.size) - ptr[rows].astype(np.int64)) * 101) % n).astype(np.uint32)
    val = rng.standard_normal(rows.size)
    x = rng.standard_normal(n)
    want = np.zeros(n, dtype=np.longdouble)
    np.add.at(want, rows, val.astype(np.longdouble) * x[col].astype(np.longdouble))
    want += np.longdouble(sigma) * x
    A = pkg.Matrix(pkg.Context(), ptr, col, val)
    A.set_format("sell")
    y = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    A.spmv(torch.from_numpy(x).cuda(), y, sigma)
    bound = 1e-15 * (L + 1) * max(np.max(np.abs(val)), 1.0) * np.max(np.abs(x))
    assert np.all(np.abs(y.cpu().numpy() - want.astype(np.float64)) <= bound)
    A.close()
