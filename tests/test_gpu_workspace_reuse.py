"""Contexts, workspaces and the memory pool reused between calls: the same bits on a fresh, a reused and a released
library state, on several host threads at once, and on a solver that ran another family (a longer one, another seed)
before; the statistics of a solve that come back in one block."""
import threading

import numpy as np
import pytest


def _problem(pkg, dims, m, seed=0):
    a = pkg.workloads.stencil_cd3d(*dims)
    return a, np.random.default_rng(seed).standard_normal(a.n), np.linspace(0.01, 0.9, m)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["incremental", "deferred"])
def test_same_bits_whatever_ran_before(cuda, pkg, mode):
    a, b, sigma = _problem(pkg, (17, 13, 11), 7)
    kw = dict(tol=1e-10, max_iter=1000, shift_mode=mode)
    pkg.release()
    first = pkg.solve(a, b, sigma, **kw)
    assert first.status == 0 and first.refined == 0
    pkg.solve(*_problem(pkg, (30, 31, 9), 20), tol=1e-12, max_iter=3000)
    again = pkg.solve(a, b, sigma, **kw)
    pkg.release()
    released = pkg.solve(a, b, sigma, **kw)
    results = [None] * 6

    def work(i):
        results[i] = pkg.solve(a, b, sigma, **kw)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(results))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    for r in [again, released] + results:
        assert r.k == first.k and np.array_equal(r.x, first.x) and np.array_equal(r.conv_k, first.conv_k)
        assert np.array_equal(r.active, first.active)
        for key in ("alpha", "beta", "omega", "rr"):
            assert np.array_equal(r.extra["hist"][key], first.extra["hist"][key])


@pytest.mark.gpu
def test_solver_runs_again_after_a_longer_solve(cuda, pkg):
    torch = cuda
    a, b, sigma = _problem(pkg, (25, 24, 23), 30)
    A = pkg.Matrix(pkg.Context(), a.ptr, a.col, a.val)
    s = pkg.Solver(A, 30, tol=1e-10, max_iter=1000, shift_mode="deferred", refine=False, true_residuals=True)
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()  # noqa: E731
    x = torch.empty((30, a.n), dtype=torch.float64, device="cuda")
    easy = sigma + 3.0
    one = s.run(dev(b), dev(easy), seed=4, x=x)
    x1 = x.clone()
    s.run(dev(b), dev(sigma), seed=0, x=x)  # more iterations and flushes
    two = s.run(dev(b), dev(easy), seed=4, x=x)
    assert two.k == one.k and torch.equal(x, x1) and np.array_equal(two.active, one.active)
    assert two.max_true_residual <= 1.01e-10
    n, live = a.n, 30
    assert two.flush_ms > 0 and two.flush_bytes <= 8.0 * n * (2 * (two.k + 1) + two.flushes + 1 + 4.0 * live * (two.flushes + 1))
    assert two.flush_bytes >= 8.0 * n * (2 * (two.k - 1) + 3.0 * 1)
    s.close()
    A.close()
