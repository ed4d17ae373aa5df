"""Field products on paired columns (fp.cuh, fp2ops.cuh).

On the CPU: a word-by-word model of the rows, with every word that the device code
lets go asserted to be zero, at the ends of each routine's operand range.  On the
GPU: points and line tables made of extreme limbs (the verify path's arithmetic does
not ask whether a point is on the curve), against the oracle, for every kernel."""
import itertools

import numpy as np
import pytest

import bls_ref as B
import cpu as C
import workload_py as W

M32 = (1 << 32) - 1
P = B.P
NINV = (-pow(P, -1, 1 << 32)) % (1 << 32)
R = 1 << 384


def limbs(v, n=12):
    return [(v >> (32 * i)) & M32 for i in range(n)]


def value(w):
    return sum(x << (32 * i) for i, x in enumerate(w))


def chain(t, at, xs, b, carry=0):
    """t[at..] += sum xs[k] b 2^(64 k) + carry in place; the carry out"""
    n = 2 * len(xs)
    v = value(t[at:at + n]) + sum((x * b) << (64 * k) for k, x in enumerate(xs)) + carry
    t[at:at + n] = limbs(v & ((1 << (32 * n)) - 1), n)
    return v >> (32 * n)


def row(E, O, prev, xs, b):
    s = E[0] + prev
    E[0] = s & M32
    assert chain(O, 0, xs[1::2], b, s >> 32) == 0       # nothing leaves O
    O[11] += chain(E, 0, xs[0::2], b)
    assert O[11] <= M32


def mont(a, b=None, t=None):
    """fp_mul_redundant(a, b), or mont_reduce12(t)"""
    E, O, prev = limbs(t or 0), [0] * 12, 0
    for i in range(12):
        if t is None:
            row(E, O, prev, limbs(a), limbs(b)[i])
            prev = 0
        m = ((E[0] + prev) * NINV) & M32
        row(E, O, prev, limbs(P), m)
        assert E[0] == 0
        prev, E, O = E[1], O, E[2:] + [0, 0]
    v = value(E) + prev + (value(O) << 32)
    assert v < R and O[10] == O[11] == 0
    return v


def sqr_columns(a):
    """the 24-word square of fp_sqr"""
    w, d = limbs(a), limbs(2 * a)
    A, O = [0] * 24, [0] * 24
    for i in range(12):
        x = [w[i]] + d[i + 2::2]
        y = ([(w[i + 1] << 1) & M32] if i < 11 else []) + d[i + 3::2]
        na, nb = len(x), len(y)
        assert na == 1 + (11 - i) // 2 and nb == (12 - i) // 2
        ca, cb = chain(A, 2 * i, x, w[i]), chain(O, 2 * i, y, w[i]) if nb else 0
        if i & 1:
            assert ca == 0
            if nb:
                assert O[2 * i + 2 * nb] == 0
                O[2 * i + 2 * nb] = cb
        else:
            assert cb == 0
            if i:
                assert A[2 * i + 2 * na] == 0
                A[2 * i + 2 * na] = ca
            else:
                assert ca == 0
    return value(A) + (value(O) << 32)


EDGES = [0, 1, M32, (1 << 192) - 1, (1 << 381) - 1, P - 1, P, P + 1, 2 * P - 1, (0x1a0111e9 << 352) | ((1 << 352) - 1),
         int("ffffffff00000000" * 6, 16) % P, int("00000000ffffffff" * 6, 16) % P, (-R) % P, R % P]


def test_rows_at_the_ends_of_their_ranges():
    redundant = [v for v in EDGES] + [8 * P - 1, 7 * P + M32]
    for a, b in itertools.product(redundant, repeat=2):
        v = mont(a, b)
        assert (v * R - a * b) % P == 0 and v < 7.5 * P
    for t in EDGES + [R - 1, R - 2, (R - 1) // M32]:
        v = mont(0, t=t)
        assert (v * R - t) % P == 0 and v <= P
    for a in [v for v in EDGES if v < 2 * P] + [3 * P, 3 * P - 1]:
        assert sqr_columns(a) == a * a and a * a // R + P < 2 * P


@pytest.mark.gpu
@pytest.mark.parametrize("lanes,tpb", [(6, 384), (6, 64), (8, 0), (1, 0)])
def test_extreme_limbs(golden, lanes, tpb):
    import bls_gpu as G
    rng = np.random.default_rng(7)
    pick = [np.array([v % P >> (64 * i) & (2 ** 64 - 1) for i in range(6)], dtype=np.uint64) for v in EDGES]
    n = 67                                      # two full blocks of 32 and a remainder
    draw = lambda k: np.stack([pick[j] for j in rng.integers(0, len(pick), k)])     # noqa: E731
    sigs, nhms = draw(2 * n).reshape(n, 12), draw(2 * n).reshape(n, 12)
    tabs = draw(3 * 68 * 6).reshape(3, 2448)
    tabs[0] = W.plain_config(n=1, seed=3)["pk_tabs"][0]       # a key's table, all rows with an inverse
    index = (np.arange(n) % 3).astype(np.int32)
    want, wml, wgt = C.verify_batch(sigs, nhms, golden["g2_gen_coeffs"], tabs, pk_index=index, want_values=True, nthreads=4)
    keep = ~(wml == 0).all(axis=1)              # a vanished Miller value has no inverse
    assert keep.sum() > n // 4
    for k in (1, 3):                            # the first table alone: normalised lines; all: raw tables
        with G.Context(lanes=lanes, threads_per_block=tpb) as ctx:
            ids = np.array([ctx.register_pk_coeffs(t) for t in tabs[:k]], dtype=np.int32)
            use = keep & (index < k)
            res, ml, gt = ctx.verify(sigs[use], nhms[use], ids[index[use]], want_values=True)
            assert (res == want[use]).all() and (ml == wml[use]).all() and (gt == wgt[use]).all()
