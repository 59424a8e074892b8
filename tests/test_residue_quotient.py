"""The residue pass's arithmetic, with exact rationals on the CPU (no GPU).

For t = a 2^(P - E) with |t| <= 2^P, P <= 53, and M = 1.5 2^52:

  H = RN(t 2^-32 + M) - M,  s = t - H 2^32,  sm = RN(s + M)
  a' = H 2^32 + (sm - M)                       (the integer nearest to t, ties to even)
  q = RN(a' RN(1/p) + M) - M,  r = a' - q p

r fits a signed byte and is congruent to a' for every odd modulus; it is the
centred representative for P <= 51.  The device forms r modulo 2^32 from the
low words of sm and of the FMA that gives q."""
from fractions import Fraction

import numpy as np
import pytest

ODD = [255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193, 191, 181]
MAGIC = 6755399441055744.0          # 1.5 2^52


def low_word(v):
    return int(np.array([v], dtype=np.float64).view(np.uint64)[0]) & 0xFFFFFFFF


def integer_of(t):
    """a' and its low word from the double t, as the kernel forms them."""
    H = Fraction(float(Fraction(t) / 2 ** 32 + Fraction(MAGIC))) - Fraction(MAGIC)
    s = Fraction(t) - H * 2 ** 32
    assert Fraction(float(s)) == s and abs(s) <= 2 ** 31            # the FMA is exact
    sm = float(s + Fraction(MAGIC))
    a = H * 2 ** 32 + (Fraction(sm) - Fraction(MAGIC))
    assert Fraction(float(a)) == a and a.denominator == 1
    return int(a), low_word(sm)


@pytest.mark.parametrize("P", [45, 51, 52, 53])
def test_integer_and_low_word(P):
    rng = np.random.default_rng(P)
    ts = [0.0, 0.5, 1.5, 2.5, -0.5, -2.5, 2.0 ** P, -2.0 ** P, 2.0 ** 31 + 0.5, -2.0 ** 31 - 0.5,
          2.0 ** 32 - 0.5, 3 * 2.0 ** 31 + 0.5]
    ts += [float(np.ldexp(rng.uniform(-1, 1), int(e))) for e in rng.integers(-3, P + 1, 3000)]
    ts += [float(int(x) + 0.5) for x in rng.integers(-2 ** 50, 2 ** 50, 500)]
    for t in ts:
        a, lo = integer_of(t)
        assert a == round(Fraction(t)), t                           # half to even
        assert lo == a % 2 ** 32, t


@pytest.mark.parametrize("P", [51, 52, 53])
@pytest.mark.parametrize("p", ODD)
def test_residue_fits_its_byte(p, P):
    rng = np.random.default_rng(100 * p + P)
    inv = float(Fraction(1, p))
    top = 2 ** P
    vals = [0, 1, -1, top, -top, top - 1]
    # the quotients nearest to half-integers at both ends of the range, and others
    for j in [top // p - i for i in range(40)] + [int(x) for x in rng.integers(0, top // p, 200)]:
        for d in (-1, 0, 1, 2):
            v = j * p + (p - 1) // 2 + d
            vals += [v, -v]
    for v in vals:
        if abs(v) > top:
            continue
        qm = float(Fraction(v) * Fraction(inv) + Fraction(MAGIC))
        q = int(Fraction(qm) - Fraction(MAGIC))
        r = v - q * p
        assert -128 <= r <= 127, (p, v, r)
        if P <= 51 or p == 255:
            assert abs(r) <= (p - 1) // 2, (p, v, r)
        byte = ((v % 2 ** 32) - low_word(qm) * p) & 0xFF
        assert (byte - 256 if byte >= 128 else byte) == r
