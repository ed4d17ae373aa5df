"""The key kernels' small-set forms (eight lanes a key) against the oracle: warp
remainders, the set size where the dispatch changes, every reject reason, keys of
small order on the twist, the identity, and the whole line tables."""
import os
import random
import re

import numpy as np
import pytest

import bls_ref as B
import bls_gpu as G
import workload_py as W

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
LIMIT = int(re.search(r"kOctMaxKeys = (\d+);",
                      open(os.path.join(HERE, "..", "icp-gpu_b200", "csrc", "kernels.cu")).read()).group(1))


@pytest.fixture(scope="module")
def pool():
    rng = random.Random(9)
    keys = [B.g2_compress(B.g2_mul(B.G2_GEN, rng.randrange(1, 1 << 250))) for _ in range(6)]
    pts, bad = [], list(keys)
    while len(pts) < 4:
        x = (rng.randrange(B.P), rng.randrange(B.P))
        y = B.f2_sqrt(B.f2_add(B.f2_mul(B.f2_sqr(x), x), (4, 4)))
        if y is not None:
            pts.append((x, y))
        else:
            b = bytearray(x[1].to_bytes(48, "big") + x[0].to_bytes(48, "big"))
            b[0] |= 0x80
            bad.append(bytes(b))                                           # off the curve
    bad += [B.g2_compress(p) for p in pts]                                # outside the subgroup
    z = -0xd201000000010000
    h2 = (z ** 8 - 4 * z ** 7 + 5 * z ** 6 - 4 * z ** 4 + 6 * z ** 3 - 4 * z ** 2 - 4 * z + 13) // 9
    r = 0x73eda753299d7d483339d80809a1d80553bda402fffe5bfeffffffff00000001
    for q in (13, 23):                                                   # small orders
        assert h2 % q == 0
        n = r * h2
        while n % q == 0:
            n //= q
        for p in pts:
            s = B.g2_mul(p, n)
            while s is not None and B.g2_mul(s, q) is not None:
                s = B.g2_mul(s, q)
            if s is not None:
                bad.append(B.g2_compress(s))
    bad.append(bytes([0xC0]) + bytes(95))
    bad.append(bytes([0xE0]) + bytes(95))
    bad.append(bytes([0xC0]) + bytes(94) + b"\1")
    bad.append(bytes([keys[0][0] & 0x7F]) + keys[0][1:])
    b = bytearray(keys[1])
    b[48:] = B.P.to_bytes(48, "big")
    bad.append(bytes(b))
    return keys, bad


@pytest.mark.parametrize("n", [1, 3, 4, 5, 33, LIMIT, LIMIT + 1])
def test_statuses_and_points(pool, n):
    _, bad = pool
    dec = [B.g2_decompress(e) for e in bad]
    want = np.array([st for st, _ in dec], dtype=np.int32)
    assert set(want.tolist()) == {0, 1, 2, 3, 4}
    q = np.zeros((len(bad), 24), dtype=np.uint64)
    for i, (_, pt) in enumerate(dec):
        if pt is not None:
            q[i] = W.g2_affine_u64(pt)
    pick = np.concatenate([np.random.default_rng(n).permutation(len(bad)), np.arange(n)])[:n] % len(bad)
    with G.Context() as ctx:
        st, got = ctx.g2_decompress(b"".join(bad[i] for i in pick))
    assert (st == want[pick]).all()
    assert (got == q[pick]).all()


@pytest.mark.parametrize("n", [1, 2, 4, 5, 41, LIMIT, LIMIT + 1])
def test_line_tables(n):
    keys = W.WL._keys(W.WL.SplitMix64(n), min(n, 24))
    pick = np.arange(n) % min(n, 24)
    with G.Context(max_pks=n) as ctx:
        ids = ctx.register_pk_affine_batch(keys["pk_affine"][pick])
        for j in sorted({0, 1, 2, 3, 4, 5, n // 2, n - 2, n - 1} & set(range(n))):
            assert (ctx.pk_table(int(ids[j])) == keys["pk_tables"][pick[j]]).all(), j
