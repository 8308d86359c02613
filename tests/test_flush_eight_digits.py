"""The basis flush's eight 8-bit digits (csrc/flush_tc.cu), restated with Python integers: the split, the bounds of the
diagonal sums, their conversion from FP32 and the dropped diagonals on the CPU, and the kernel's results bit for bit."""
import ctypes as C
import math
import random
from fractions import Fraction

import numpy as np
import pytest

K, ND = 64, 8
TWO23 = 1 << 23


def _fixed(v, scale, bits):
    """trunc(v 2^(bits - scale))"""
    q = Fraction(v) * Fraction(2) ** (bits - scale)
    return int(q)


def _digits(q):
    out = []
    for s in range(ND - 1, 0, -1):
        d = ((q + 128) & 255) - 128
        out.append(d)
        q = (q - d) >> 8
    return [q] + out[::-1]


def _f32(x):
    return float(np.float32(x))


def _result(D):
    """diag_sum: T / 2^13 from the eight sums, with the kernel's FP32 steps"""
    M2 = 1.5 * 2 ** 24
    f4 = _f32(D[4] + M2)
    d5 = _f32((D[4] - (f4 - M2)) * 256 + D[5])
    f5 = _f32(d5 + M2)
    d6 = _f32((d5 - (f5 - M2)) * 256 + D[6])
    half = [int(f4 - M2) // 2, int(f5 - M2) // 2, int(_f32(d6 + M2) - M2) // 2, int(_f32(D[7] + M2) - M2) // 2]
    h0, h1, h2, h3 = D[0] * 256 + D[1], D[2] * 256 + D[3], half[0] * 256 + half[1], half[2] * 256 + half[3]
    assert all(-(1 << 31) <= h < 1 << 31 for h in (h0, h1, h2, h3))
    return (h0 << 35) + (h1 << 19) + (h2 << 4) + ((h3 + 2048) >> 12)


def _join(T, k):
    a = abs(T)
    if a == 0:
        return 0.0
    e = a.bit_length()
    m = (a >> (e - 53)) + ((a >> (e - 54)) & 1) if e > 53 else a << (53 - e)
    return math.copysign(math.ldexp(m, e - 53 + k), T)


def _sums(A, B):
    """diagonal sums of digit rows A[l], B[l]"""
    D = [0] * (2 * ND - 1)
    for a, b in zip(A, B):
        for s in range(ND):
            for t in range(ND):
                D[s + t] += a[s] * b[t]
    return D


def test_digits_are_exact_and_balanced():
    rng = random.Random(1)
    for bits in (62, 63):  # basis, coefficients
        top = (1 << bits) - 1
        for q in [0, 1, -1, top, -top, 0x3F7F7F7F7F7F7F7F, -0x3F80808080808080] + [rng.randint(-top, top) for _ in range(5000)]:
            d = _digits(q)
            assert sum(x << (8 * (7 - s)) for s, x in enumerate(d)) == q
            assert all(-128 <= x <= 127 for x in d[1:]) and abs(d[0]) <= (64 if bits == 62 else 128)


def test_sums_fit_and_convert():
    """|D_d| <= (d + 1/2) 2^20: below 2^22 up to d = 3, below 2^23 beyond; T / 2^13 to within 0.54 units."""
    assert 3.5 * 2 ** 20 < 2 ** 22 and 7.5 * 2 ** 20 + 256 < TWO23
    rng = random.Random(2)
    bound = [int((d + 0.5) * 2 ** 20) for d in range(ND)]
    cases = [bound, [-b for b in bound], [0] * ND] + [[rng.choice((-1, 1)) for _ in range(ND)] for _ in range(200)]
    cases += [[rng.randint(-b, b) for b in bound] for _ in range(5000)]
    for D in cases:
        T = sum(x << (8 * (7 - d)) for d, x in enumerate(D))
        assert abs(Fraction(T, 1 << 13) - _result(D)) <= Fraction(54, 100)


def test_dropped_diagonals_are_below_two_to_minus_54():
    dropped = sum((2 * ND - 1 - d) * K * 128 * 128 * Fraction(2) ** (112 - 8 * d) for d in range(ND, 2 * ND - 1))
    assert dropped / Fraction(2) ** 125 < Fraction(2) ** -54


def _bits_exp(v):
    return math.frexp(v)[1] if v else -1074


def _model(V, c, se, F, i):
    """output of coefficient row c for element i (own terms 0)"""
    L = V.shape[0]
    a = [math.ldexp(c[l], se[l]) for l in range(L)]
    E = max(_bits_exp(x) for x in a)
    A = [_digits(_fixed(x, E, 63)) for x in a]
    B = [_digits(_fixed(V[l, i], F + se[l], 62)) for l in range(L)]
    return _join(_result(_sums(A, B)[:ND]), E + F - 56)


@pytest.mark.gpu
@pytest.mark.parametrize("L,n,kind", [(64, 60, "extreme"), (64, 49, "negative"), (59, 97, "random"), (1, 7, "random")])
def test_kernel_bit_for_bit(cuda, pkg, L, n, kind):
    """Column 0 holds 1 in every slot, so that the other columns' values can be small against their slot's maximum:
    with slot 0 large there, the rest have digits in every place ("extreme": all 127, D_7 close to 2^23)."""
    torch = cuda
    rng = np.random.default_rng(L + n)
    m, ld = 3, (n + 31) // 32 * 32
    V, c = np.zeros((L, ld)), rng.standard_normal((m, L))
    V[:, :n] = rng.standard_normal((L, n)) * 2.0 ** rng.integers(-12, 1, (L, n))
    if kind != "random":
        M = float(0x1F7F7F7F7F7F7F)
        V[:, :n] = M * 2.0 ** -62
        V[0, :n] = 1.0 - 2.0 ** -40
        c[:] = (M if kind == "extreme" else -M) * 2.0 ** -63
        c[:, 0] = 1.0 - 2.0 ** -41
        c[1, 5:] *= -1.0
    V[:, 0] = 1.0
    se = [_bits_exp(float(np.max(np.abs(V[l, :n])))) for l in range(L)]
    own, ws = torch.zeros(2 * m, dtype=torch.float64, device="cuda"), None
    lib = pkg.lib()
    fn = lib.hbk_flush_tc_run
    fn.restype = C.c_int
    fn.argtypes = [C.c_void_p, C.c_size_t, C.c_uint, C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_int,
                   C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    lib.hbk_flush_tc_workspace_bytes.restype = C.c_size_t
    lib.hbk_flush_tc_workspace_bytes.argtypes = [C.c_int]
    ws = torch.zeros(int(lib.hbk_flush_tc_workspace_bytes(m)) // 8 + 1, dtype=torch.float64, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    panels = -(-n // 48)
    X, P = (torch.zeros(m * 48 * panels, dtype=torch.float64, device="cuda") for _ in range(2))
    tV, tc = torch.tensor(V, device="cuda"), torch.tensor(c, device="cuda")
    tp = torch.tensor(-c, device="cuda")
    rc = fn(tV.data_ptr(), ld, n, L, tc.data_ptr(), tp.data_ptr(), L, own.data_ptr(), m, X.data_ptr(), P.data_ptr(), 1,
            ws.data_ptr(), err.data_ptr(), None)
    torch.cuda.synchronize()
    assert rc == 0 and int(err.item()) == 0
    x, p = (t.cpu().numpy().reshape(panels, m, 48).transpose(1, 0, 2).reshape(m, -1)[:, :n] for t in (X, P))
    for i in list(range(min(n, 9))) + list(range(max(9, n - 4), n)):
        F = max(_bits_exp(V[l, i]) - se[l] for l in range(L))
        for j in range(m):
            assert x[j, i] == _model(V, c[j], se, F, i), (j, i)
            assert p[j, i] == _model(V, -c[j], se, F, i), (j, i)
