"""The hash to G1's small-batch form (k_neg_hash_to_g1_quad): warp remainders, the
batch size where the dispatch changes, and the stream's edges around SHA-256's block
and padding boundaries, against the workload's C++ hash and the oracle."""
import os
import re

import numpy as np
import pytest

import bls_ref as B
import bls_gpu as G
import workload_py as W

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
LIMIT = int(re.search(r"kHashQuadMax = (\d+);",
                      open(os.path.join(HERE, "..", "icp-gpu_b200", "csrc", "hash.cu")).read()).group(1))


@pytest.fixture(scope="module")
def ctx():
    with G.Context() as c:
        yield c


@pytest.mark.parametrize("n", [1, 3, 4, 5, 33, LIMIT, LIMIT + 1])
def test_batch_sizes(ctx, n):
    rng = W.SplitMix64(n)
    msgs = [rng.msg() for _ in range(min(n, 64))]
    want = W.WL.g1_neg(W.WL.hash_to_g1(msgs))
    pick = np.arange(n) * 7 % len(msgs) if n > 1 else np.array([0])
    got = ctx.neg_hash_to_g1([msgs[i] for i in pick], W.DST)
    assert (got == want[pick]).all()


@pytest.mark.parametrize("dst_len", [1, 21, 22, 23, 30, 255])
def test_padding_boundaries(ctx, dst_len):
    """lengths that end the stream at 55, 56, 63, 64 and 65 bytes into a block"""
    dst = bytes(range(1, dst_len + 1)) if dst_len < 255 else bytes(range(255))
    lens = sorted({(e - 4 - dst_len) % 64 for e in (54, 55, 56, 57, 62, 63, 64, 65)})
    msgs = [bytes((5 * i + n) & 0xff for i in range(n)) for n in lens]
    got = ctx.neg_hash_to_g1(msgs, dst)
    for row, m in zip(got, msgs):
        assert (row == np.array(B.g1_to_mont_u64(B.g1_neg(B.hash_to_g1(m, dst))), dtype=np.uint64)).all(), len(m)
