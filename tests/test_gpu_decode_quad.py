"""The G1 decoder's small-batch form (k_g1_decompress_quad) against the oracle:
block edges and remainders, the batch size where the dispatch changes, every reject
reason, and points of small order, whose scalar multiplication meets the addition's
exceptional cases."""
import random
import re
import os

import numpy as np
import pytest

import bls_ref as B
import bls_gpu as G
import cpu as C

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def _limit():
    text = open(os.path.join(HERE, "..", "icp-gpu_b200", "csrc", "kernels.cu")).read()
    return int(re.search(r"kQuadMaxPoints = (\d+);", text).group(1))


def _random_point(rng):
    while True:
        x = rng.randrange(B.P)
        y = B.fp_sqrt((x * x * x + 4) % B.P)
        if y is not None:
            return (x, y if rng.random() < 0.5 else B.P - y)


@pytest.fixture(scope="module")
def pool():
    rng = random.Random(11)
    n_e = B.R_ORDER * ((B.X_ABS + 1) ** 2 // 3) if hasattr(B, "X_ABS") else None
    r = 0x73eda753299d7d483339d80809a1d80553bda402fffe5bfeffffffff00000001
    h = (0xd201000000010000 + 1) ** 2 // 3
    pts = []
    for _ in range(12):
        pts.append(B.g1_compress(B.g1_mul(_random_point(rng), h)))             # in G1
        pts.append(B.g1_compress(_random_point(rng)))                          # outside
    for q in (3, 11, 10177):                                                  # small orders
        for _ in range(3):
            p = B.g1_mul(_random_point(rng), r * h // (q * q if (h % (q * q)) == 0 else q))
            if p is not None:
                pts.append(B.g1_compress(p))
                pts.append(B.g1_compress(B.g1_neg(p)))
    pts += [B.g1_compress((0, 2)), B.g1_compress((0, B.P - 2))]               # x = 0, order 3
    pts.append(bytes([0xC0]) + bytes(47))                                    # identity
    pts.append(bytes([0xE0]) + bytes(47))                                    # infinity with the sort flag
    pts.append(bytes([0x40]) + bytes(47))
    pts.append(bytes([pts[0][0] & 0x7F]) + pts[0][1:])                        # compression bit clear
    for v in (B.P, B.P + 1, (1 << 381) - 1):                                  # x >= p
        b = bytearray(v.to_bytes(48, "big"))
        b[0] |= 0x80
        pts.append(bytes(b))
    x = 1
    while B.fp_is_square((x ** 3 + 4) % B.P):
        x += 1
    b = bytearray(x.to_bytes(48, "big"))
    b[0] |= 0x80
    pts.append(bytes(b))                                                     # off the curve
    assert n_e is None or n_e % r == 0
    return np.stack([np.frombuffer(p, dtype=np.uint8) for p in pts])


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 63, 193, "limit", "limit + 1"])
def test_points_and_statuses(pool, n):
    n = {"limit": _limit(), "limit + 1": _limit() + 1}.get(n, n)
    rng = np.random.default_rng(n)
    pick = np.concatenate([rng.permutation(len(pool)), rng.integers(0, len(pool), n)])[:n] if n > 1 else np.array([0])
    want_st, want = C.g1_decompress(pool, nthreads=4)
    assert {int(s) for s in want_st} == {0, 1, 2, 3, 4}
    with G.Context() as ctx:
        st, xy = ctx.g1_decompress(pool[pick].tobytes())
    assert (st == want_st[pick]).all()
    assert (xy == want[pick]).all()
