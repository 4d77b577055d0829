"""The device's branch-free division against IEEE division, bit for bit, on
finite normal operands whose quotient is normal: 4e7 random ones; quotients as
close to a midpoint between two numbers as a quotient can be, where any error
of the reciprocal or of the residual shows; and divisors at the ends of a
binade, where the reciprocal's own rounding is at its worst. The division of
the units that keep IEEE rounding (the differentiated step's); the plain
step's, which promises half a unit and next to nothing more, on random
operands."""
import ctypes

import numpy as np
import pytest

from test_math_gpu import DIV

pytestmark = pytest.mark.gpu


def scaled(rng, m, bits=100):
    """Integers below 2^53 as doubles of random sign and exponent."""
    return rng.choice([-1.0, 1.0], m.size) * np.ldexp(m.astype(np.float64), rng.integers(-bits, bits, m.size))


def mantissas(rng, n):
    return rng.integers(1 << 52, 1 << 53, n, dtype=np.uint64)


def next_to_midpoints(B, c, below_one):
    """A with A 2^s = B M + c for an odd M of 54 bits and small odd c: A / B is
    c / (B 2^s) away from the midpoint M / 2^s. B odd, below 2^53; s = 54 for
    quotients below one, 53 for those above. Returns (A, B) where A < 2^53."""
    s = 54 if below_one else 53
    inv = B.copy()  # Newton's iteration for 1 / B mod 2^64: 3, 6, ... 96 bits
    for _ in range(5):
        inv = inv * (np.uint64(2) - B * inv)
    M = (np.uint64(0) - np.uint64(c % (1 << 64)) * inv) & np.uint64((1 << s) - 1)
    if not below_one:
        M |= np.uint64(1 << 53)
    keep = M >= np.uint64(1 << 53)
    B, M = B[keep], M[keep]
    h, low = np.uint64(27), np.uint64((1 << 27) - 1)
    b1, b0, m1, m0 = B >> h, B & low, M >> h, M & low
    mid = b1 * m0 + b0 * m1
    rest = ((mid & low) << h) + b0 * m0 + np.uint64(c % (1 << 64))
    A = b1 * m1 + (mid >> h) + (rest >> np.uint64(54))
    A = A if below_one else A * np.uint64(2) + ((rest >> np.uint64(53)) & np.uint64(1))
    keep = (A < np.uint64(1 << 53)) & (A > 0)
    return A[keep], B[keep]


def quotient(name, x, y):
    import torch

    from pyshield_b200.build import PROBE_LIB

    fn = getattr(ctypes.CDLL(PROBE_LIB), name)
    fn.argtypes = [ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 4
    a, b = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    out = torch.empty_like(a)
    assert fn(DIV, a.numel(), a.data_ptr(), b.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    return out.cpu().numpy()


def check(x, y, name="shield_probe_math_ieee"):
    got, want = quotient(name, x, y), x / y
    bad = np.flatnonzero(got != want)
    assert bad.size == 0, f"{bad.size} of {x.size}, first {x[bad[0]].hex()} / {y[bad[0]].hex()}"


@pytest.mark.parametrize("seed", range(10))
def test_random(seed):
    rng = np.random.default_rng(seed)
    n = 4_000_000
    x, y = scaled(rng, mantissas(rng, n)), scaled(rng, mantissas(rng, n))
    check(x, y)
    check(x, y, "shield_probe_math")


@pytest.mark.parametrize("below_one", [True, False])
@pytest.mark.parametrize("c", [-5, -3, -1, 1, 3, 5])
def test_quotients_next_to_midpoints(c, below_one):
    rng = np.random.default_rng(7)
    B = mantissas(rng, 1_000_000) | np.uint64(1)
    B[:20_000] = np.uint64(1 << 53) - np.uint64(1) - np.uint64(2) * np.arange(20_000, dtype=np.uint64)
    # the upper end of a binade, where a reciprocal just short of its rounding would show
    B[40_000:400_000] |= np.uint64(((1 << 8) - 1) << 44)
    B[20_000:40_000] = np.uint64(1 << 52) + np.uint64(1) + np.uint64(2) * np.arange(20_000, dtype=np.uint64)
    A, B = next_to_midpoints(B, c, below_one)
    assert A.size > 100_000
    for a, b in zip(A[:50].tolist(), B[:50].tolist()):  # the construction itself, in whole numbers
        s = 54 if below_one else 53
        M, r = divmod(a << s, b)
        assert (M if r == c else M + 1) % 2 == 1 and (r == c or r - b == c)
    check(scaled(rng, A), scaled(rng, B))


@pytest.mark.parametrize("end", ["ones", "one"])
def test_divisors_at_the_ends_of_a_binade(end):
    rng = np.random.default_rng(8)
    d = np.repeat(np.arange(1000, dtype=np.uint64), 500)
    B = np.uint64(1 << 53) - np.uint64(1) - d if end == "ones" else np.uint64(1 << 52) + d
    A = mantissas(rng, B.size)
    A[::5] = np.uint64(1 << 52)
    A[1::5] = np.uint64(1 << 53) - np.uint64(1) - rng.integers(0, 8, A[1::5].size, dtype=np.uint64)
    A[2::5] = np.uint64(1 << 52) + rng.integers(0, 8, A[2::5].size, dtype=np.uint64)
    check(scaled(rng, A), scaled(rng, B))
