"""Which batches share one persistent launch (csrc/batch.c): with fewer than 8 workers, or where no family that could
join has more than 8192 rows.  The families of a shared launch report its one device time; on the workers a family's
solve is the one it gets alone, bit for bit.  Either way every x_j agrees with the other route's."""
import numpy as np
import pytest


def _family(pkg, n, m, seed):
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    keep = np.stack([i > 0, i >= 0, i < n - 1], axis=1)
    col = np.stack([i - 1, i, i + 1], axis=1)[keep].astype(np.uint32)
    val = np.broadcast_to([-1.1, 2.05, -0.9], (n, 3))[keep].copy()
    ptr = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(keep.sum(axis=1), out=ptr[1:])
    return pkg.workloads.Family(f"n{n}", pkg.workloads.Csr(ptr, col, val), rng.standard_normal(n),
                                0.05 * np.arange(1, m + 1), 0, 1e-10, 10000, {})


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,workers,shared", [((500, 8192), 8, True), ((8193, 500), 8, False), ((8193, 500), 7, True),
                                                  ((300, 301), 16, True), ((9000, 8193, 40), 0, False)])
def test_route(cuda, pkg, sizes, workers, shared):
    fams = [_family(pkg, n, 6 + i, n) for i, n in enumerate(sizes)]
    kw = dict(tol=1e-10, max_iter=10000)
    res, _ = pkg.batch_solve(fams, workers=workers, **kw)
    alone, _ = pkg.batch_solve(fams, workers=workers, persistent=False, **kw)
    assert all(r.status == 0 for r in res + alone)
    assert (len({r.solve_ms for r in res}) == 1) == shared
    for r, a in zip(res, alone):
        scale = np.max(np.abs(a.x))
        # (both stop at 1e-10 of |b|; sigma >= 0.05 above a spectrum of at least 0.05 bounds |x| / |b| and the error)
        assert np.max(np.abs(r.x - a.x)) <= 1e-8 * scale
        if not shared:
            assert r.k == a.k and np.array_equal(r.x, a.x)
