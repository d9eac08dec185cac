"""The residue products' arithmetic on the CPU, in exact integers: moduli pairwise coprime, the bound of the
scaled integers against their product, residues from a 32-bit word and a high part, division of an int32 sum by a
38-bit reciprocal, and the fraction sum, for sums at the extremes of their range."""
from math import gcd

import numpy as np

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223]
P = int(np.prod([int(m) for m in MODULI], dtype=object))


def _signed(v, p):
    r = v % p
    return r - p if 2 * r >= p else r


def test_moduli_and_bound():
    assert all(gcd(a, b) == 1 for i, a in enumerate(MODULI) for b in MODULI[:i])
    k = 65536
    assert (2 ** 43 + k ** 0.5 / 2) ** 2 < P / 2


def test_products_recombine_exactly():
    rng = np.random.default_rng(0)
    for k in (1, 31, 400):
        a = [int(x) for x in rng.integers(-(2 ** 43), 2 ** 43 + 1, k) // max(1, int(k ** 0.5))]
        b = [int(x) for x in rng.integers(-(2 ** 43), 2 ** 43 + 1, k) // max(1, int(k ** 0.5))]
        if k == 1:
            a, b = [2 ** 43], [-(2 ** 43)]
        y = 0
        for p in MODULI:
            f = pow(P // p % p, -1, p)
            ra, rb = [], []
            for vs, g, out in ((a, 1, ra), (b, f, rb)):
                for v in vs:
                    lo, hi = v & 0xFFFFFFFF, v >> 32
                    t = hi * _signed(2 ** 32 * g, p) + sum(((lo >> 8 * i) & 255) * _signed(256 ** i * g, p) for i in range(4))
                    assert abs(t) < 2 ** 19
                    m = np.float32(12582912.0) + np.float32(t)
                    q = np.float32(np.float64(np.float32(t)) * np.float64(np.float32(1.0) / np.float32(p)) + 12582912.0)
                    r = int(m) - 12582912 - p * (int(q) - 12582912)
                    assert -128 <= r <= 128
                    out.append(((r + 128) % 256) - 128)
            c = sum(x * z for x, z in zip(ra, rb))
            r = c - ((c * -(-(2 ** 38) // p)) >> 38) * p
            assert 0 <= r <= p and r < 256
            y += r * (2 ** 64 // p)
        y %= 2 ** 64
        y -= 2 ** 64 if y >= 2 ** 63 else 0
        exact = sum(x * z for x, z in zip(a, b))
        assert abs(y * P / 2 ** 64 - exact) <= P * 2.0 ** -52


def test_int32_sum_division_at_its_extremes():
    for p in MODULI:
        inv = -(-(2 ** 38) // p)
        assert inv < 2 ** 31
        for c in [s * (2 ** 30 - d) for s in (1, -1) for d in range(3 * p)] + list(range(-3 * p, 3 * p)):
            r = c - ((c * inv) >> 38) * p
            assert 0 <= r <= p and r < 256 and (r - c) % p == 0
