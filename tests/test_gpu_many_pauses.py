"""Deferred solves that pause far more often than their chunks of iterations would end: basis blocks of three
iterations, alone or with chunks of 200.  A solve that goes on is not taken for one that hangs."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("use_graph", [True, False, "loop"])
@pytest.mark.parametrize("chunk", [0, 200])
@pytest.mark.parametrize("capped", [False, True])
def test_small_blocks(cuda, pkg, use_graph, chunk, capped):
    a = pkg.workloads.stencil_cd2d(300, 300)
    b = np.random.default_rng(3).standard_normal(a.n)
    sigma = np.array([0.004, 0.1])
    kw = dict(seed=0, tol=1e-11, max_iter=330 if capped else 1000, shift_mode="deferred", refine=False)
    want = pkg.solve(a, b, sigma, **kw)
    got = pkg.solve(a, b, sigma, basis_block=3, graph_chunk=chunk, use_graph=use_graph, **kw)
    assert want.k > 300  # (over a hundred pauses)
    assert got.status == want.status == (4 if capped else 0)
    assert abs(got.k - want.k) <= 0.02 * want.k
    assert np.max(np.abs(got.x[1] - want.x[1])) <= 1e-8 * np.max(np.abs(want.x[1]))
    if not capped:
        assert np.max(np.abs(got.x - want.x)) <= 1e-8 * np.max(np.abs(want.x))
