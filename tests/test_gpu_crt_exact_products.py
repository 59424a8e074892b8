"""The modular mode on products that are known exactly: k equal terms x y, so that C'
is the integer k x' y', of any length from a few bits to the widest that the modulus
count admits -- around the limits between the conversion's branches (2^96, 2^115),
one bit from a tie, both signs.  The reference is Python's integer arithmetic and its
round-to-nearest-even conversion; every modulus count's tables meet it in the kernels."""
import random

import numpy as np
import pytest

import ca3dmm_b200 as cb
from oracle import oracle as orc
from tests._util import dev_zeros, from_dev, to_dev

pytestmark = pytest.mark.gpu


def _integers(rng, bits, count):
    """Signed integers below 2^bits of all lengths, ends of binades among them."""
    out = [1, (1 << bits) - 1, (1 << (bits - 1)) + 1, (1 << (bits // 2)) - 1]
    while len(out) < count:
        b = rng.randint(max(1, bits - 30), bits) if len(out) % 2 else rng.randint(1, bits)
        out.append(rng.choice([(1 << b) - rng.randint(1, min(3, 1 << (b - 1))),
                               (1 << (b - 1)) + rng.randint(0, 2) if b > 2 else 1,
                               rng.getrandbits(b) | 1]))
    return [rng.choice([-1, 1]) * min(v, (1 << bits) - 1) for v in out]


@pytest.mark.parametrize("terms", [1, 3, 4096, 65536])
@pytest.mark.parametrize("nmod", range(8, 19))
def test_exact_products(cuda, nmod, terms):
    k, m, n = terms + 2, 100, 72
    P = orc.crt_bits(nmod, k)
    bits = min(P - 1, 52)
    rng = random.Random(100 * nmod + terms)
    x, y = _integers(rng, bits, m), _integers(rng, bits, n)
    # the leading 1 fixes the scale of a row of A (a column of B); its partner is 0
    A, B = np.empty((m, k), order="F"), np.empty((k, n), order="F")
    A[:, 0], A[:, 1] = 1.0, 0.0
    B[0, :], B[1, :] = 0.0, 1.0
    A[:, 2:] = np.ldexp(np.array(x, dtype=np.float64), -bits)[:, None]
    B[2:, :] = np.ldexp(np.array(y, dtype=np.float64), -bits)[None, :]
    dA, lda = to_dev(A)
    dB, ldb = to_dev(B)
    dC = dev_zeros(m * n)
    e = cb.Ca3dmmEngine(m, n, k, 0, 0, p=1)
    assert e.ok and e.set_gemm_mode(cb.GEMM_CRT, nmod) == 0
    assert e.exec(dA, lda, dB, ldb, dC, m) == 0
    got = from_dev(dC, m, n)
    e.free()
    want = np.array([[float(terms * a * b) for b in y] for a in x])
    assert np.array_equal(got, np.ldexp(want, -2 * bits))
