"""A solve that fails leaves the caller's device array of solutions as it was.  In the deferred shift mode the rows go
there without a second copy, so the kernel that writes them looks whether a flush failed; the failure is made through
the library's test hook (the next flush sets its error flag), and the flushes themselves run as ever."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("refine", [False, True])
@pytest.mark.parametrize("where", ["first", "last"])
def test_failed_flush_leaves_x(cuda, pkg, refine, where):
    torch = cuda
    a = pkg.workloads.stencil_cd3d(12)
    m = 5
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()  # noqa: E731
    b, sigma = dev(np.random.default_rng(0).standard_normal(a.n)), dev(np.linspace(0.01, 0.5, m))
    # (at most 20 iterations per basis block: "last": the only flush is the one at the end)
    kw = dict(tol=1e-10, shift_mode="deferred", flush="tensor", refine=refine,
              **(dict(basis_block=20) if where == "first" else dict(max_iter=12)))
    x = torch.full((m, a.n), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    A = pkg.Matrix(pkg.Context(), a.ptr, a.col, a.val)
    pkg.lib().hbk_flush_tc_test_error(1)
    try:
        with pytest.raises(pkg.HbicgError, match="flush"):
            pkg.Solver(A, m, **kw).run(b, sigma, seed=0, x=x)
    finally:
        pkg.lib().hbk_flush_tc_test_error(0)
    assert torch.all(x == 7.0)
    r = pkg.Solver(A, m, **kw).run(b, sigma, seed=0, x=x)
    assert r.flushes == (0 if where == "last" else r.flushes) and (where == "last" or r.flushes > 1)
    assert not torch.any(x == 7.0)
    A.close()
