"""Gradients from given solutions at the edges of their kernels: row lengths around the entries held in registers
(8, up to the 64 of a SELL-32 row), empty rows, odd n, one and many shifts, with and without weights, padded leading
dimensions, and a matrix that takes the thread-per-entry path.  The reference is the same sums in torch FP64; each
output may be off by the rounding of its own sum, (terms + 2) * 2^-53 times the sum of its terms' absolute values on
either side."""
import numpy as np
import pytest

EPS = 2.0**-53


def _csr(n, lens, seed):
    rng = np.random.default_rng(seed)
    ptr = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(lens, out=ptr[1:])
    col = np.concatenate([np.sort(rng.choice(n, size=k, replace=False)) for k in lens] or [np.zeros(0)])
    return ptr, col.astype(np.uint32), rng.standard_normal(int(ptr[-1]))


def _lens(kind, n, rng):
    if kind == "mixed":  # all within SELL-32, around multiples of the 8 entries in registers
        return np.tile([7, 8, 9, 7, 8, 8, 16, 9], n // 8 + 1)[:n]
    if kind == "gaps":
        return np.where(np.arange(n) % 11 == 3, 0, 5)
    if kind == "widest":
        return np.full(n, 64)
    return np.minimum(n - 1, np.where(rng.random(n) < 0.05, 200, 3))  # "irregular": not SELL-32


@pytest.mark.gpu
@pytest.mark.parametrize("kind,n,m,weights,pad", [
    ("mixed", 33, 1, True, 0), ("mixed", 1000, 5, False, 7), ("gaps", 257, 3, True, 1), ("widest", 129, 2, True, 0),
    ("mixed", 90001, 33, True, 31), ("irregular", 700, 6, True, 3),
])
def test_gradients_match_torch(cuda, pkg, kind, n, m, weights, pad):
    torch = cuda
    rng = np.random.default_rng(n + m)
    ptr, col, val = _csr(n, _lens(kind, n, rng), n)
    A = pkg.Matrix(pkg.Context(), ptr, col, val)
    if kind != "irregular":
        A.set_format("sell")  # (the form that takes the thread-per-row path, whatever the padding)
    assert (A.format == "sell") == (kind != "irregular")
    X, Y = (torch.from_numpy(rng.standard_normal((m, n + pad))).cuda()[:, :n] for _ in range(2))
    w = torch.from_numpy(rng.uniform(0.5, 2.0, m)).cuda() if weights else None
    dval, db, ds = A.adjoint_gradients(X, Y, w)
    lam = Y if w is None else w[:, None] * Y
    rows = torch.repeat_interleave(torch.arange(n), torch.from_numpy(np.diff(ptr.astype(np.int64)))).cuda()
    terms = lam[:, rows] * X[:, torch.from_numpy(col.astype(np.int64)).cuda()]
    for got, want, size, count in (
        (dval, -terms.sum(0), terms.abs().sum(0), m),
        (db, lam.sum(0), lam.abs().sum(0), m),
        (ds, -(lam * X).sum(1), (lam * X).abs().sum(1), n),
    ):
        assert torch.all((got - want).abs() <= 2 * (count + 2) * EPS * size)
    A.close()
