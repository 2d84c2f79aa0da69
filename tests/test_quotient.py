"""The mean over a node's neighbours divides by way of the reciprocal
(`quotient` in gtd_gnn.cu): q = x inv, then q + (x - q d) inv with the residue
in one fused multiply-add and the sum in another. Restated here in integers,
rounding where the device rounds, and compared with the correctly rounded
quotient (Markstein's theorem says that they agree when inv is 1 / d correctly
rounded)."""
import numpy as np
import pytest

B = 24  # bits of a float's significand


def _normal(n):
    """(significand, shift) of n > 0 rounded to 24 bits, ties to even: the value
    significand * 2^shift with the significand in [2^23, 2^24)."""
    bits = np.frexp(n.astype(np.float64))[1].astype(np.int64)  # n may round up to a power of two here
    bits -= (n < (np.int64(1) << np.minimum(bits - 1, 62))).astype(np.int64)
    shift = np.maximum(bits - B, 0)
    q, rest = n >> shift, n & ((np.int64(1) << shift) - 1)
    half = np.where(shift > 0, np.int64(1) << np.maximum(shift - 1, 0), np.int64(1))
    q = q + ((rest > half) | ((rest == half) & (q & 1 == 1)))
    up = q == 1 << B
    q, shift = np.where(up, q >> 1, q), np.where(up, shift + 1, shift)
    left = np.where(q < 1 << (B - 1), B - np.frexp(q.astype(np.float64))[1].astype(np.int64), 0)
    return q << left, shift - left


def _mismatches(x, d):
    """Significands x (in [2^23, 2^24)) whose quotient by d comes out otherwise."""
    k = (d - 1).bit_length()
    e = B - 1 + k                     # inv = I 2^-e, I in [2^23, 2^24]
    I, r = divmod(1 << e, d)
    I += 2 * r > d or (2 * r == d and I & 1)
    q, sh = _normal(x * np.int64(I))  # q 2^(sh - e)
    residue = (x << (e - sh)) - q * d
    assert np.all(np.abs(residue) < 1 << B)  # the first fused multiply-add is exact
    got, gs = _normal((q << e) + residue * np.int64(I))  # in units of 2^(sh - 2 e)
    # x / d, correctly rounded: 27 quotient bits or more, the remainder as a sticky bit
    num = x << (k + 4)
    true, ts = _normal(((num // d) << 1) | (num % d != 0))
    return np.flatnonzero((got != true) | (gs + sh - 2 * e != ts - (k + 5)))


@pytest.mark.parametrize("d", [3, 25, 127])
def test_every_significand(d):
    x = np.arange(1 << (B - 1), 1 << B, dtype=np.int64)
    assert _mismatches(x, d).size == 0


def test_random_significands_over_degrees_up_to_4096():
    rng = np.random.default_rng(1)
    edge = np.array([1 << 23, (1 << 23) + 1, (1 << 24) - 1, (1 << 24) - 2], dtype=np.int64)
    for d in range(1, 4097):
        x = np.concatenate([edge, rng.integers(1 << 23, 1 << 24, 500)])
        assert _mismatches(x, d).size == 0, d


def test_a_plain_product_with_the_reciprocal_is_not_enough():
    """What the second step is for."""
    x = np.arange(1 << (B - 1), (1 << (B - 1)) + 4096, dtype=np.float64).astype(np.float32)
    assert np.any(x * (np.float32(1) / np.float32(7)) != x / np.float32(7))
