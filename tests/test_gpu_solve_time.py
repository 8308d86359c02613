"""stats.solve_ms is the device time of the whole solve, its true-residual corrections among it: no less than the same
solve takes without them."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("form,mode", [("fused", "incremental"), ("fused", "deferred"), ("plain", "auto")])
def test_corrections_add_to_the_time(cuda, pkg, form, mode):
    a = pkg.workloads.stencil_cd3d(20)
    b = np.full(a.n, 1.0 / np.sqrt(a.n))
    sigma = np.array([0.01, 0.02, 0.4])
    # a tolerance below what the true residuals reach: every solve ends with corrections
    kw = dict(seed=0, tol=2e-15, max_iter=400, form=form, shift_mode=mode)
    pkg.solve(a, b, sigma, refine=True, **kw)
    bare = min(pkg.solve(a, b, sigma, refine=False, **kw).solve_ms for _ in range(3))
    for _ in range(3):
        r = pkg.solve(a, b, sigma, refine=True, **kw)
        assert r.refined >= 1
        assert r.solve_ms > bare, (r.solve_ms, bare)
