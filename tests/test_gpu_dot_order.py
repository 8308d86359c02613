"""The order in which a solve's dot products are summed (csrc/kernels_fused.cu): a matter of n and the number of SMs,
not of how the kernels are launched.  One iteration restated here in that order, with fused multiply-adds where the
kernels have them; alpha, omega, beta and (r, r) then agree bit for bit, as every operation is the same one.

Another order is as accurate, but moves the residual below the tolerance at which the solve stops, and with it the
ninth digit of results that cancel (the shift gradients)."""
import numpy as np
import pytest

NT = 256
SPLIT = 134217729.0  # 2^27 + 1


def _fma(a, b, c):
    """a b + c rounded once: the product's error by Dekker's splitting, the sum's by Knuth's."""
    a, b, c = np.broadcast_arrays(np.float64(a), np.float64(b), np.float64(c))
    p = a * b
    ah, bh = a * SPLIT, b * SPLIT
    ah, bh = ah - (ah - a), bh - (bh - b)
    al, bl = a - ah, b - bh
    e = al * bl - (((p - ah * bh) - al * bh) - ah * bl)
    s = p + c
    t = s - p
    return s + (((p - (s - t)) + (c - t)) + e)


def _tree(v):
    """256 values: the 32 lanes of each of 8 warps, then the 8 sums."""
    for width in (32, NT // 32):
        v = v.reshape(-1, width)
        while v.shape[1] > 1:
            h = v.shape[1] // 2
            v = v[:, :h] + v[:, h:]
        v = v[:, 0]
    return v[0]


def _dot(x, y, sets):
    n = len(x)
    steps = -(-n // (sets * NT))
    at = np.arange(steps * sets * NT).reshape(steps, sets, NT)
    acc = np.zeros((sets, NT))
    for k in range(steps):
        here = at[k] < n
        i = np.where(here, at[k], 0)
        acc = np.where(here, _fma(x[i], y[i], acc), acc)
    part = np.array([_tree(a) for a in acc])
    thread = np.zeros(NT)
    for i in range(0, sets, NT):
        p = part[i:i + NT]
        thread[:len(p)] = thread[:len(p)] + p
    return _tree(thread)


def _band(n, off, val):
    """CSR of a matrix with constant diagonals (ascending offsets) and its product in stored order."""
    i = np.arange(n)[:, None]
    col = i + np.array(off)[None, :]
    keep = (col >= 0) & (col < n)
    ptr = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(keep.sum(axis=1), out=ptr[1:])

    def product(x):
        acc = np.zeros(n)
        for o, v in zip(off, val):
            lo, hi = max(0, -o), min(n, n - o)
            acc[lo:hi] = _fma(v, x[lo + o:hi + o], acc[lo:hi])
        return acc

    vals = np.broadcast_to(np.array(val), keep.shape)[keep].copy()
    return ptr, col[keep].astype(np.uint32), vals, product


NARROW = ((-1, 0, 1), (-1.1, 2.35, -0.9))
WIDE = ((-7, -2, -1, 0, 1, 2, 7), (-0.7, -0.3, -1.1, 4.6, -0.9, -0.4, -0.6))


@pytest.mark.gpu
@pytest.mark.parametrize("band", [NARROW, WIDE], ids=["narrow", "wide"])
# one set; a few; around 3 and 6 sets of 256 rows and 1, 2, 3 and 4 of 512 per SM of 152
@pytest.mark.parametrize("n", [200, 700, 40001, 77825, 116800, 130000, 154625, 233500, 300001, 311300, 400000])
def test_one_iteration_bit_for_bit(cuda, pkg, band, n):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    by_rows = min(-(-n // NT), 6 * sms)
    by_vec = min(-(-n // (2 * NT)), 4 * sms)
    ptr, col, val, product = _band(n, *band)
    rng = np.random.default_rng(n)
    b = np.where(rng.random(n) < 0.5, -1.0, 1.0) * 2.0 ** -rng.integers(0, 4, n)  # (b, b) is exact in any order
    sg = 0.0371
    A = pkg.Matrix(pkg.Context(), ptr, col, val)
    assert A.format == "sell"
    S = pkg.Solver(A, 1, max_iter=4, shift_mode="incremental", refine=False)
    t = lambda v: torch.from_numpy(np.atleast_1d(v)).cuda()  # noqa: E731
    x = torch.empty(1, n, dtype=torch.float64, device="cuda")
    bd, sd = t(b), t(sg)
    torch.cuda.synchronize()
    h = S.run(bd, sd, seed=0, x=x).extra["hist"]

    bb = np.sum(b * b)
    s = _fma(sg, b, product(b))
    alpha = bb / _dot(b, s, by_rows)
    assert h["alpha"][1] == alpha
    q = _fma(-alpha, s, b)
    y = _fma(sg, q, product(q))
    omega = _dot(q, q, by_rows) / _dot(q, y, by_rows)
    assert h["omega"][1] == omega
    r = _fma(-omega, y, q)
    assert h["rr"][1] == _dot(r, r, by_vec)
    assert h["beta"][1] == (alpha / omega) * (_dot(b, r, by_vec) / bb)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3000, 3100, 4000, 5000, 22222])
def test_sums_of_many_blocks(cuda, pkg, n):
    """TILE products of few rows with many entries leave more sums than K2 has threads for its rows: alpha of the first
    iteration in the order that NT threads add them."""
    rng = np.random.default_rng(n)
    lens = np.full(n, 3)
    lens[::7] = 300  # a row of over 256 entries is a block of its own, as is every run of rows between
    ptr = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(lens, out=ptr[1:])
    row = np.repeat(np.arange(n), lens)
    col = ((row + np.arange(len(row)) - ptr[:-1].astype(np.int64)[row]) % n).astype(np.uint32)
    val = np.where(rng.random(len(row)) < 0.5, -0.125, 0.125)  # every product and sum of a row is exact
    b = np.where(rng.random(n) < 0.5, -1.0, 1.0) * (1.0 + rng.integers(0, 2**10, n) * 2.0**-10)  # (b, b) too
    A = pkg.Matrix(pkg.Context(), ptr, col, val)
    A.set_format("tile")
    sg = 0.00371  # (the sum cancels: another order shows)
    h = pkg.Solver(A, 1, max_iter=2, shift_mode="incremental", refine=False).run(b, np.array([sg])).extra["hist"]
    y = np.zeros(n)
    np.add.at(y, row, val * b[col])
    s = _fma(sg, b, y)
    # blocks of rows: 6 consecutive rows of 3 entries, one long row, in turn from row 0 (long)
    bounds = np.unique(np.concatenate([np.arange(0, n, 7), np.arange(1, n, 7), [n]]))
    blocks = len(bounds) - 1
    sets = min(blocks, 6 * cuda.cuda.get_device_properties(0).multi_processor_count)
    acc = np.zeros((sets, NT))
    for k, (lo, hi) in enumerate(zip(bounds[:-1], bounds[1:])):
        acc[k % sets, :hi - lo] = _fma(b[lo:hi], s[lo:hi], acc[k % sets, :hi - lo])
    part = np.array([_tree(a) for a in acc])
    thread = np.zeros(NT)
    for i in range(0, sets, NT):
        p = part[i:i + NT]
        thread[:len(p)] = thread[:len(p)] + p
    assert h["alpha"][1] == np.sum(b * b) / _tree(thread)
