"""The division steps of fp_inv.cuh, modelled in Python as the device runs them (thirty
steps on the low words, then the matrix on the whole values): the low limbs vanish,
the word-sized matrices and |d|, |e| < 37 p hold, and the result is the inverse."""
import random

import bls_ref as B

P, BITS, ROUNDS = B.P, 30, 37
MASK, M32 = (1 << BITS) - 1, (1 << 32) - 1
NINV = (-pow(P, -1, 1 << 32)) & M32


def low(x):
    return ((x & MASK) | (((x >> BITS) & MASK) << BITS)) & M32


def inverse(x):
    f, g, d, e, delta = P, x, 0, 1, 1
    for _ in range(ROUNDS):
        if g == 0:
            break
        u, v, q, r, f0, g0 = 1, 0, 0, 1, low(f), low(g)
        for _ in range(BITS):
            odd = g0 & 1
            swap = odd and delta > 0
            s = -1 if swap else 1
            af, au, av = (s * f0, s * u, s * v) if odd else (0, 0, 0)
            delta = 2 + s * delta
            f0, u, v = (g0, 2 * q, 2 * r) if swap else (f0, 2 * u, 2 * v)
            g0, q, r = ((g0 + af) & M32) >> 1, q + au, r + av
        assert abs(u) + abs(v) <= 1 << BITS and abs(q) + abs(r) <= 1 << BITS
        nf, ng, nd, ne = u * f + v * g, q * f + r * g, u * d + v * e, q * d + r * e
        assert nf & MASK == ng & MASK == 0
        nd += (((nd & M32) * NINV) & MASK) * P
        ne += (((ne & M32) * NINV) & MASK) * P
        assert nd & MASK == ne & MASK == 0
        f, g, d, e = nf >> BITS, ng >> BITS, nd >> BITS, ne >> BITS
        assert max(abs(f), abs(g)) < 2 * P and max(abs(d), abs(e)) < 37 * P
    assert g == 0 and abs(f) in (1, P)
    return (d if f > 0 else -d) % P


def test_inverse_of_extremes_and_random_values():
    rng = random.Random(3)
    edges = [1, 2, 3, P - 1, P - 2, (P + 1) // 2, (P - 1) // 2, 1 << 380, (1 << 381) % P, (1 << 384) % P]
    for x in edges + [rng.randrange(1, P) for _ in range(300)] + [rng.randrange(1, 1 << rng.randrange(1, 380)) for _ in range(200)]:
        assert inverse(x) * x % P == 1
    assert inverse(0) == 0
