"""The division step of tests/test_division_exact.py for uint16 patterns: ray sums to 253 x 65535 < 2^24 over
counts to 253 (the largest image the strip kernels take).  The sums nearest a rounding boundary of the
quotient are the ones that could round wrongly; they are the integers beside c times a midpoint of two
float32 values, so those are tested, with random sums beside them, every step emulated exactly in
float64 and the last rounding done in integers."""
import numpy as np


def quotient(s, c):
    """(the corrected value before its rounding as float64, its float32 rounding) of the kernels' steps."""
    r = np.float32(1.0 / c)
    q0 = (s * np.float64(r)).astype(np.float32)                 # a product of two float32 values: exact in float64
    rem_exact = s - q0.astype(np.float64) * c                   # multiples of q0's last place below 2^53
    rem = rem_exact.astype(np.float32)
    assert np.array_equal(rem.astype(np.float64), rem_exact)
    return q0.astype(np.float64) + rem.astype(np.float64) * np.float64(r)


def test_quotients_of_wide_sums_are_correctly_rounded():
    g = np.random.default_rng(0)
    for c in range(1, 254):
        top = c * 65535
        q = g.random(4000) * 65535.0
        f = q.astype(np.float32)
        mid = f.astype(np.float64) + np.spacing(f).astype(np.float64) / 2
        near = np.floor(mid * c)                                # 25 + 8 bits: exact
        s = np.concatenate([near, near + 1, near - 1, g.integers(0, top + 1, 4000).astype(np.float64), [0.0, 1.0, top]])
        s = np.unique(s[(s >= 0) & (s <= top)])
        t = quotient(s, c)
        got = t.astype(np.float32)
        ulp = np.spacing(got).astype(np.float64)
        for edge in (got - ulp / 2, got + ulp / 2):             # the emulation's own rounding cannot matter
            assert np.all(np.abs(t - edge) > np.abs(t) * 2.0 ** -50)
        # s / c lies strictly between the midpoints around `got`: 2^k-scaled integers, exact
        k = 25 - np.frexp(np.maximum(ulp, 2.0 ** -149))[1]
        k = np.maximum(k, 0)
        sc = np.ldexp(1.0, k)
        lo, hi = (got.astype(np.float64) - ulp / 2) * sc, (got.astype(np.float64) + ulp / 2) * sc
        for e in (lo, hi):
            assert np.array_equal(e, np.floor(e)) or np.all(s[e != np.floor(e)] == 0)
        num = [int(a) << int(b) for a, b in zip(s, k)]
        assert all(int(a) * c <= n <= int(b) * c for a, n, b, z in zip(lo, num, hi, s) if z > 0), c
