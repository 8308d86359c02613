"""Timed workloads of the shifted solver: what a program has it do, through the package's public calls.

Kinds (the "kind" of a case):
  solve     a shifted family (A + sigma_j I) x_j = b with matrix, workspace and right-hand side resident on the GPU
            (Matrix and Solver kept, Solver.run per pass): a parameter sweep, a time step, a frequency response
  call      the drop-in entry point shifted_lopbicg_dynamic on host arrays: matrix and b in, every x_j out
  batch     many small uneven families in one batch_solve call, host arrays in and out
  train     forward and backward of the differentiable solve (shifted_solve): a loss over the solutions, gradients
            with respect to the matrix values, the right-hand side and the shifts
  gradients the gradients alone from solutions already at hand (Matrix.adjoint_gradients)
  spmv      one product y = A x + sigma x (Matrix.spmv)

Matrices: convection-diffusion stencils in two and three dimensions ("stencil", sides nx, ny, nz; nz = 0 is the
5-point one) and rows of power-law length (n rows).  Solves run at the package's default tolerance of 1e-12;
"refine" says whether the true residuals are checked and corrected after the solve (the package's default) or not
(what the reference's entry points do).  Every value is FP64, the only type that the library computes in.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

pkg = load_package()
DEV = "cuda"


def listed():
    return [
        # the smallest call: a coarse grid as in unit tests, reduced models and coarsest levels; latency is all there is
        dict(name="solve_8", kind="solve", nx=8, ny=8, nz=8, m=6, lo=0.01, hi=0.05, refine=True),
        # the reference's small configuration: 32^3, 16 shifts
        dict(name="solve_32", kind="solve", nx=32, ny=32, nz=32, m=16, lo=0.01, hi=0.15, refine=True),
        # an ordinary two-dimensional family with ragged sides
        dict(name="solve_2d", kind="solve", nx=331, ny=293, nz=0, m=24, lo=0.01, hi=1.0, refine=False),
        # an ordinary three-dimensional family: 128^3, 32 shifts
        dict(name="solve_128", kind="solve", nx=128, ny=128, nz=128, m=32, lo=1e-3, hi=1.0, refine=False),
        # the largest: 256^3, 64 shifts, the benchmark's shape
        dict(name="solve_256", kind="solve", nx=256, ny=256, nz=256, m=64, lo=1e-4, hi=1.0, refine=False),
        # irregular sparsity: power-law row lengths (network and circuit matrices)
        dict(name="solve_powerlaw", kind="solve", n=60000, m=16, lo=0.5, hi=4.0, refine=True),
        # one drop-in call from a C program's host buffers
        dict(name="call_48", kind="call", nx=47, ny=48, nz=50, m=12, lo=0.01, hi=0.5),
        # many small families at once: a sweep over matrices
        dict(name="batch_16", kind="batch", count=16, n_lo=4000, n_hi=80000, m_lo=8, m_hi=40),
        # one step of fitting a matrix, a source or shifts through the solve
        dict(name="train_56", kind="train", nx=56, ny=57, nz=55, m=16, lo=0.01, hi=1.0),
        # the backward pass's gradients at the differentiable benchmark's size
        dict(name="gradients_128", kind="gradients", nx=128, ny=128, nz=128, m=32),
        # the product alone, structured and irregular: power iterations, residual checks, other Krylov methods
        dict(name="spmv_stencil", kind="spmv", nx=255, ny=254, nz=256),
        dict(name="spmv_powerlaw", kind="spmv", n=2000000),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sides(rng, n_lo, n_hi, flat):
    """Sides of a grid of about n points, n log-uniform, each side off the cube's (or square's) by up to an eighth."""
    n = _log(rng, n_lo, n_hi)
    s = n ** (1 / 2 if flat else 1 / 3)
    side = lambda: max(3, int(round(s * rng.uniform(0.9, 1.1))))  # noqa: E731
    return side(), side(), 0 if flat else side()


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "call", "batch", "train", "gradients", "spmv", "spmv"])
    if kind in ("solve", "call", "train"):
        if kind == "solve" and rng.random() < 0.15:
            return dict(kind=kind, n=int(_log(rng, 2000, 60000)), m=rng.randint(1, 16), lo=0.5, hi=4.0,
                        refine=rng.random() < 0.5)
        top = 3e6 if kind == "solve" else 2e5
        nx, ny, nz = _sides(rng, 300, top, rng.random() < 0.3)
        if nz == 0:  # (two-dimensional grids are worse conditioned: ordinary sizes only)
            nx, ny = min(nx, 400), min(ny, 400)
        m = int(round(_log(rng, 1, 48)))
        c = dict(kind=kind, nx=nx, ny=ny, nz=nz, m=m, lo=0.01, hi=round(rng.uniform(0.1, 1.0), 3))
        if kind == "solve":
            c["refine"] = m * nx * ny * max(nz, 1) < 1e6 and rng.random() < 0.5
        return c
    if kind == "batch":
        m_lo = rng.randint(4, 16)
        return dict(kind=kind, count=rng.randint(3, 20), n_lo=int(_log(rng, 1000, 8000)),
                    n_hi=int(_log(rng, 15000, 80000)), m_lo=m_lo, m_hi=m_lo + rng.randint(0, 16))
    if kind == "gradients":
        nx, ny, nz = _sides(rng, 1e4, 2e6, rng.random() < 0.3)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, m=rng.randint(1, 32))
    if rng.random() < 0.5:
        return dict(kind=kind, n=int(_log(rng, 5e4, 2e6)))
    nx, ny, nz = _sides(rng, 5e4, 1.6e7, rng.random() < 0.3)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz)


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _dims(case):
    return [d for d in (case["nx"], case["ny"], case["nz"]) if d]


def _coefficients(ndim):
    """diagonal, west, east, the other axes: the repository's convection-diffusion stencils."""
    return 2.0 * ndim, -1.2, -0.8, -1.0


def _stencil(dims):
    """CSR (int32 ptr, int32 col, float64 val) on the GPU, natural order, ascending columns."""
    n = math.prod(dims)
    diag, west, east, other = _coefficients(len(dims))
    idx = torch.arange(n, device=DEV)
    coords, stride, rem = [], [1], idx
    for d in dims:
        coords.append(rem % d)
        rem = rem // d
        stride.append(stride[-1] * d)
    slow = range(1, len(dims))
    entries = [(-stride[a], other, coords[a] > 0) for a in reversed(slow)]
    entries += [(-1, west, coords[0] > 0), (0, diag, coords[0] >= 0), (1, east, coords[0] < dims[0] - 1)]
    entries += [(stride[a], other, coords[a] < dims[a] - 1) for a in slow]
    mask = torch.stack([e[2] for e in entries], dim=1)
    ptr = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    ptr[1:] = torch.cumsum(mask.sum(dim=1), 0).int()
    off = torch.tensor([e[0] for e in entries], dtype=torch.int32, device=DEV)
    col = (idx.int()[:, None] + off[None, :])[mask]
    val = torch.tensor([e[1] for e in entries], dtype=torch.float64, device=DEV).expand(n, -1)[mask]
    return ptr, col.contiguous(), val.contiguous()


def _powerlaw(n, seed):
    """CSR with Zipf row lengths (mean about 16, at most 4000), a third of the columns near the diagonal, diagonal
    1.1 x the row's absolute sum: the repository's irregular workload, drawn on the GPU."""
    g = _gen(seed)
    u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    length = torch.clamp((2.0 / u).round(), 1, 4000).long()
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), length)
    tot = rows.numel()
    near = torch.rand(tot, generator=g, device=DEV) < 0.3
    cols = torch.where(near, torch.clamp(rows + torch.randint(-64, 65, (tot,), generator=g, device=DEV), 0, n - 1),
                       torch.randint(0, n, (tot,), generator=g, device=DEV))
    key = torch.unique((rows * n + cols)[cols != rows])
    vals = torch.randn(key.numel(), generator=g, device=DEV, dtype=torch.float64)
    # (row sums in fixed point: the same matrix on every run, whatever order the additions take)
    total = torch.zeros(n, dtype=torch.int64, device=DEV).index_add_(0, key // n, (vals.abs() * 2.0**30).round().long())
    total = total.double() / 2.0**30
    at = torch.arange(n, device=DEV)
    key, order = torch.sort(torch.cat([key, at * n + at]))
    vals = torch.cat([vals, torch.where(total > 0, 1.1 * total, 1.0)])[order]
    ptr = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0).int()
    return ptr, (key % n).int(), vals.contiguous()


def _csr(case, seed):
    return _powerlaw(case["n"], seed) if "n" in case else _stencil(_dims(case))


def _sigma(case):
    """m shifts from lo to hi, geometric."""
    m, lo, hi = case["m"], case["lo"], case["hi"]
    return lo * (hi / lo) ** (np.arange(m) / max(m - 1, 1))


def _normal(seed, *shape):
    return torch.randn(*shape, generator=_gen(seed), device=DEV, dtype=torch.float64)


def _rhs(n, seed):
    b = _normal(seed + 1, n)
    return b / torch.linalg.vector_norm(b)


class _HostFamily:
    def __init__(self, a, b, sigma):
        self.a, self.b, self.sigma, self.seed = a, b, sigma, 0


def _families(case, seed):
    """2-D and 3-D grids in turn, sides, shifts and right-hand sides from the seed, as host arrays."""
    rng = np.random.default_rng(seed)
    shapes = np.random.default_rng(case["count"])  # (the same families for every seed, with other right-hand sides)
    out = []
    for f in range(case["count"]):
        n = math.exp(shapes.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))
        dims = [int(round(n ** (1 / 2)))] * 2 if f % 2 == 0 else [int(round(n ** (1 / 3)))] * 3
        a = pkg.workloads.stencil_cd2d(*dims) if f % 2 == 0 else pkg.workloads.stencil_cd3d(*dims)
        sigma = np.sort(shapes.uniform(0.01, 1.0, int(shapes.integers(case["m_lo"], case["m_hi"] + 1))))
        out.append((dims, _HostFamily(a, rng.standard_normal(a.n), sigma)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "batch":
        s["families"] = [f for _, f in _families(case, seed)]
        return s
    ptr, col, val = _csr(case, seed)
    n = ptr.numel() - 1
    if kind == "call":
        pin = lambda t: t.cpu().pin_memory()  # noqa: E731
        s.update(ptr=pin(ptr), col=pin(col), val=pin(val), b=pin(_rhs(n, seed)), sigma=torch.from_numpy(_sigma(case)))
        s.update(x=torch.zeros(case["m"], n, dtype=torch.float64).pin_memory(), r=torch.empty_like(s["b"]).pin_memory())
        return s
    if kind == "train":
        leaf = lambda t: t.requires_grad_(True)  # noqa: E731
        s.update(ptr=ptr, col=col, val=leaf(val), b=leaf(_rhs(n, seed)), sigma=leaf(torch.from_numpy(_sigma(case)).to(DEV)))
        s.update(w=torch.rand(case["m"], generator=_gen(seed + 2), device=DEV, dtype=torch.float64), c=_rhs(n, seed + 3))
        return s
    torch.cuda.synchronize()  # the library works on a stream of its own
    s["matrix"] = pkg.Matrix(pkg.Context(), ptr, col, val)
    if kind == "solve":
        s.update(solver=pkg.Solver(s["matrix"], case["m"], refine=case["refine"]), b=_rhs(n, seed), sigma=torch.from_numpy(_sigma(case)).to(DEV))
        s["x"] = torch.empty(case["m"], n, dtype=torch.float64, device=DEV)
    elif kind == "gradients":
        s.update(x=_normal(seed + 1, case["m"], n), y=_normal(seed + 2, case["m"], n))
        s["w"] = torch.rand(case["m"], generator=_gen(seed + 3), device=DEV, dtype=torch.float64)
    else:
        s.update(x=_normal(seed + 1, n), y=torch.empty(n, dtype=torch.float64, device=DEV), sigma=0.25)
    return s


# -------------------------------------------------------------------- runs
def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "solve":
        s["solver"].run(s["b"], s["sigma"], seed=0, x=s["x"])
        return s["x"]
    if kind == "call":
        s["r"].copy_(s["b"])  # (the entry point takes b in r and x = 0, and overwrites both)
        s["x"].zero_()
        pkg.dropin_raw("dynamic", s["ptr"], s["col"], s["val"], s["x"], s["r"], s["sigma"])
        return s["x"]
    if kind == "batch":
        results, _ = pkg.batch_solve(s["families"], tol=1e-11, max_iter=10000)
        return [r.x for r in results]
    if kind == "train":
        leaves = s["val"], s["b"], s["sigma"]
        x = pkg.shifted_solve(s["ptr"], s["col"], *leaves, tol=1e-11)
        grads = torch.autograd.grad(s["w"] @ (x @ s["c"]), leaves)
        return dict(x=x, val=grads[0], b=grads[1], sigma=grads[2])
    if kind == "gradients":
        return s["matrix"].adjoint_gradients(s["x"], s["y"], s["w"])
    return s["matrix"].spmv(s["x"], s["y"], s["sigma"])


# -------------------------------------------------------- what a pass needs
def _size(case):
    """Rows and nonzeros."""
    if "n" in case:
        return case["n"], 16 * case["n"]  # (about: the lengths are drawn)
    dims = _dims(case)
    n = math.prod(dims)
    return n, n + sum(2 * n // d * (d - 1) for d in dims)


def _iterations(case):
    """About how many iterations the solve takes to 1e-12, from the condition number of a stencil (fitted)."""
    if "n" in case:
        return 600
    dims = _dims(case)
    low = sum(2 - 2 * math.cos(math.pi / (d + 1)) for d in dims) + case["lo"]
    return int((35 if len(dims) == 2 else 10.5) * (4 * len(dims) / low) ** 0.37)


def _solve_work(n, nnz, m, iters):
    """Two products and the seed's vectors per iteration, every x_j and p_j formed from the basis or updated as it
    goes (2 operations per element and shift for each of x and p, per iteration), every x_j written once."""
    product = 12 * nnz + 4 * (n + 1) + 16 * n
    return dict(bytes=iters * (2 * product + 13 * 8 * n) + 8 * n * m,
                flops=iters * (4 * nnz + 22 * n + 8 * n * m))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = dict(bytes=0, flops=0)
        shapes = np.random.default_rng(case["count"])
        for f in range(case["count"]):
            n = int(math.exp(shapes.uniform(math.log(case["n_lo"]), math.log(case["n_hi"]))))
            m = len(shapes.uniform(0.01, 1.0, int(shapes.integers(case["m_lo"], case["m_hi"] + 1))))
            side = round(n ** (1 / (2 + f % 2)))
            iters = _iterations(dict(nx=side, ny=side, nz=side * (f % 2), lo=0.02))
            for k, v in _solve_work(n, (5 + 2 * (f % 2)) * n, m, iters).items():
                total[k] += v
        return total
    n, nnz = _size(case)
    product = 12 * nnz + 4 * (n + 1) + 16 * n
    if kind == "spmv":
        return dict(bytes=product, flops=2 * nnz + 2 * n)
    m = case["m"]
    gradients = dict(bytes=16 * m * n + 4 * (n + 1) + 12 * nnz + 8 * n, flops=2 * nnz * m + n * m + 4 * n * m)
    if kind == "gradients":
        return gradients
    w = _solve_work(n, nnz, m, _iterations(case))
    if kind == "train":
        return {k: 2 * w[k] + gradients[k] for k in w}
    return w


# ------------------------------------------------------- 64-bit references
def _stencil_solve(dims, b, sigma, transposed=False):
    """Every x_j by a direct method: sine transforms along the symmetric axes, then one tridiagonal system along x
    for each pair of modes, by elimination (diagonally dominant, so without pivoting)."""
    diag, west, east, other = _coefficients(len(dims))
    if transposed:
        west, east = east, west
    nx, rest = dims[0], dims[1:]
    f = b.reshape(*reversed(dims))  # (nz, ny, nx)
    shift = torch.full(tuple(reversed(rest)), diag, dtype=torch.float64, device=DEV)
    sines = []
    for a, d in enumerate(rest):
        i = torch.arange(1, d + 1, dtype=torch.float64, device=DEV)
        sines.append(math.sqrt(2.0 / (d + 1)) * torch.sin(math.pi / (d + 1) * (i[:, None] * i[None, :] % (2 * d + 2))))
        axis = len(rest) - 1 - a
        shape = [1] * len(rest)
        shape[axis] = d
        shift = shift + (2 * other * torch.cos(math.pi * i / (d + 1))).reshape(shape)
        f = torch.tensordot(f, sines[a], dims=([axis], [0])).movedim(-1, axis)
    f = f.reshape(-1, nx).t().contiguous()
    shift = shift.reshape(-1)
    out = torch.empty(len(sigma), b.numel(), dtype=torch.float64, device=DEV)
    up = torch.empty_like(f)
    for j, sg in enumerate(sigma):
        x = torch.empty_like(f)
        up[0] = east / (shift + sg)
        x[0] = f[0] / (shift + sg)
        for i in range(1, nx):
            inv = 1.0 / (shift + sg - west * up[i - 1])
            up[i] = east * inv
            x[i] = (f[i] - west * x[i - 1]) * inv
        for i in range(nx - 2, -1, -1):
            x[i] -= up[i] * x[i + 1]
        x = x.t().reshape(*reversed(dims))
        for a in range(len(rest)):
            axis = len(rest) - 1 - a
            x = torch.tensordot(x, sines[a], dims=([axis], [0])).movedim(-1, axis)
        out[j] = x.reshape(-1)
    return out


def _rows(ptr):
    return torch.repeat_interleave(torch.arange(ptr.numel() - 1, device=DEV), (ptr[1:] - ptr[:-1]).long())


def _product(ptr, col, val, x):
    a = torch.sparse_csr_tensor(ptr.long(), col.long(), val, size=(ptr.numel() - 1,) * 2)
    return a @ x


def _dominant_solve(ptr, col, val, b, sigma):
    """Every x_j of a strictly diagonally dominant matrix by Jacobi's iteration (a contraction by 1/1.1 in the
    maximum norm), until it is down to rounding."""
    rows = _rows(ptr)
    on = rows == col
    d = torch.zeros_like(b).index_add_(0, rows[on], val[on])[:, None] + sigma[None, :]
    off = torch.where(on, torch.zeros_like(val), val)
    x = b[:, None] / d
    for _ in range(400):
        x = (b[:, None] - _product(ptr, col, off, x)) / d
    return x.t().contiguous()


def _gradients(ptr, col, x, lam):
    """dval, db, dsigma from solutions x and weighted adjoint solutions lam."""
    rows, dval = _rows(ptr), torch.zeros(col.numel(), dtype=torch.float64, device=DEV)
    for j in range(x.shape[0]):
        dval -= lam[j][rows] * x[j][col.long()]
    return dval, lam.sum(0), -(lam * x).sum(1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [_stencil_solve(dims, torch.from_numpy(f.b).to(DEV), f.sigma).cpu() for dims, f in _families(case, seed)]
    if kind == "gradients":
        s = prepare(case, seed)
        ptr, col, _ = _csr(case, seed)
        return _gradients(ptr, col, s["x"], s["w"][:, None] * s["y"])
    ptr, col, val = _csr(case, seed)
    n = ptr.numel() - 1
    if kind == "spmv":
        x = _normal(seed + 1, n)
        return _product(ptr, col, val, x) + 0.25 * x
    b, sigma = _rhs(n, seed), _sigma(case)
    if "n" in case:
        return _dominant_solve(ptr, col, val, b, torch.from_numpy(sigma).to(DEV))
    x = _stencil_solve(_dims(case), b, sigma)
    if kind != "train":
        return x
    s = prepare(case, seed)
    lam = s["w"][:, None] * _stencil_solve(_dims(case), s["c"], sigma, transposed=True)
    dval, db, dsigma = _gradients(ptr, col, x, lam)
    return dict(x=x, val=dval, b=db, sigma=dsigma)
