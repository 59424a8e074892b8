"""The arithmetic of the modular scheme's epilogue and reconstruction, restated
with Python integers on the CPU (no GPU).

Epilogue: an INT32 sum v becomes v i_t mod p_t with i_t = (M / p_t)^-1 mod p_t,
in 32-bit unsigned arithmetic.  Reconstruction: Y_g = sum of the group's u_t
(M_g / p_t) in 32 bits, S = sum_g Y_g (M / M_g) in 64-bit limb sums, the
quotient rint(S / M) from an FP64 estimate, C' = S - q M."""
from fractions import Fraction

import numpy as np
import pytest

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193, 191, 181]


def product(l):
    r = 1
    for x in l:
        r *= x
    return r


def centred(v, p):
    return v - p if v > (p - 1) // 2 else v


@pytest.mark.parametrize("N", range(8, 19))
def test_epilogue_reduction(N):
    rng = np.random.default_rng(N)
    M = product(MODULI[:N])
    for p in MODULI[:N]:
        # sums of k <= 131072 products of bytes: |r| <= 128 for p = 256 (whose sums may
        # wrap modulo 2^32), else at most 127
        lim = 131072 * (128 * 128 if p == 256 else 127 * 127)
        v = np.concatenate([rng.integers(-lim, lim + 1, 100000),
                            [0, 1, -1, lim, -lim, 32767, 32768, -32768, -32769, 65535, 65536,
                             lim - 32768, 32768 - lim]]).astype(np.int64)
        x = (v + 0x8000) & 0xFFFFFFFF                    # the accumulator
        x = (x ^ 0x8000).astype(np.uint32)
        h = (x >> np.uint32(16)).astype(np.uint16).view(np.int16).astype(np.int64)
        l = (x & np.uint32(0xFFFF)).astype(np.uint16).view(np.int16).astype(np.int64)
        inv = pow(M // p, -1, p)
        lo, hi = centred(inv, p), centred(65536 * inv % p, p)
        assert -128 <= lo <= 127 and -128 <= hi <= 127
        most = 32768 * (256 if p == 256 else 254)
        y = h * hi + l * lo + (most + p - 1) // p * p
        assert np.all(y >= 0) and np.all(y < (1 << 24 if p != 256 else 1 << 25))
        mrec = ((1 << 32) + p - 1) // p
        q = (y.astype(np.uint64) * np.uint64(mrec) >> np.uint64(32)).astype(np.int64)
        r = y - q * p
        assert np.all((r >= 0) & (r < p)) and np.all((r - v * inv) % p == 0)


def reconstruct(N, u):
    """As the kernel: sums, carries, estimate; returns C' and checks the ranges."""
    M = product(MODULI[:N])
    G = (N + 2) // 3
    sizes = [N // G + (g < N % G) for g in range(G)]
    groups, at = [], 0
    for z in sizes:
        assert z in (2, 3)
        groups.append(list(range(at, at + z)))
        at += z
    limbs = max(2, max(-(-(M // product(MODULI[t] for t in g)).bit_length() // 32) for g in groups))
    assert limbs <= 4
    a = [0] * limbs
    for g in groups:
        mg = product(MODULI[t] for t in g)
        assert mg < 2 ** 24 and all(mg // MODULI[t] < 2 ** 16 for t in g)
        Y = sum(u[t] * (mg // MODULI[t]) for t in g)
        assert Y < 2 ** 26
        for q in range(limbs):
            a[q] += Y * ((M // mg >> 32 * q) & 0xFFFFFFFF)
    assert all(x < 2 ** 63 for x in a)
    s = []
    for q in range(limbs - 1):
        s.append(a[q] & 0xFFFFFFFF)
        a[q + 1] += a[q] >> 32
    top = a[-1]
    assert top < 2 ** 64
    unit = 2 ** (32 * (limbs - 1))
    # the estimate: S 2^-shift cut to an integer below 2^52
    shift = M.bit_length() + 5 - 52
    assert shift >= 32 * (limbs - 2)
    est = (top * unit + sum(x << 32 * i for i, x in enumerate(s))) >> shift
    assert est < 2 ** 52
    q = round(Fraction(est) * Fraction(float(Fraction(2 ** shift, M))))
    S = top * unit + sum(x << 32 * i for i, x in enumerate(s))
    assert abs(est * 2 ** shift - S) < Fraction(M, 2 ** 45)
    # the kernel's words of S + q (2^128 - M)
    c = 0
    carry = 0
    low = s + [top & 0xFFFFFFFF, top >> 32, 0, 0]
    for i in range(4):
        v = q * ((2 ** 128 - M) >> 32 * i & 0xFFFFFFFF) + low[i] + carry
        c |= (v & 0xFFFFFFFF) << 32 * i
        carry = v >> 32
    assert c == (S - q * M) % 2 ** 128
    return c - 2 ** 128 if c >> 127 else c


@pytest.mark.parametrize("N", range(8, 19))
def test_reconstruction(N):
    import ca3dmm_b200 as cb
    rng = np.random.default_rng(100 + N)
    M = product(MODULI[:N])
    for k in (1, 100, 8000, 131072):
        P = cb.lib().ca3dmm_crt_bits(N, k)
        if P < 2:
            continue
        top = k * 2 ** (2 * P)                      # |C'| <= top
        vals = [0, 1, -1, top, -top, top - 1, 1 - top]
        for _ in range(400):
            b = int(rng.integers(0, top.bit_length()))
            x = int.from_bytes(rng.bytes(20), "little") % 2 ** (b + 1)
            vals += [min(x, top), -min(x, top)]
        for c in vals:
            u = [c * pow(M // p, -1, p) % p for p in MODULI[:N]]
            assert reconstruct(N, u) == c, (N, k, c)


def test_rounding_of_the_128_bit_integer():
    """hi 2^64 + lo with m = lo 2^-12 rounded to odd: for 2^32 <= |hi| < 2^51 one
    rounding of (hi - 1) 2^52 + (2^52 + m) is the rounding of the exact integer."""
    rng = np.random.default_rng(7)
    for _ in range(20000):
        bits = int(rng.integers(32, 51))
        hi = int(rng.integers(2 ** bits, 2 ** (bits + 1))) * (1 if rng.integers(2) else -1)
        # lo near a tie of the result, or anywhere
        ulp = 2 ** max(0, abs(hi).bit_length() + 64 - 53)
        lo = int.from_bytes(rng.bytes(8), "little")
        if rng.integers(2):
            lo = (lo // ulp * ulp + ulp // 2 + int(rng.integers(-2, 3))) % 2 ** 64
        m = lo >> 12 | (1 if lo & 0xFFF else 0)
        assert float(2 ** 52 + m) == 2 ** 52 + m and float(hi - 1) == hi - 1
        assert float(Fraction((hi - 1) * 2 ** 52 + (2 ** 52 + m))) * 4096.0 == \
            float(Fraction(hi * 2 ** 64 + lo)), (hi, lo)
