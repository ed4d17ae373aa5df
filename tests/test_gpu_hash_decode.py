"""Verify from message bytes with compressed signatures: hashes and decoded points of a
batch come from one launch (k_neg_hash_decode, k_neg_hash_decode_wide).  Remainders of
their blocks, the batch sizes where the dispatch changes, every reject reason, against
the workload's known results."""
import os
import re

import numpy as np
import pytest

import bls_gpu as G
import workload_py as W

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
TEXT = open(os.path.join(HERE, "..", "icp-gpu_b200", "csrc", "hash.cu")).read()
QUAD, TWO = (int(re.search(name + r" = (\d+);", TEXT).group(1)) for name in ("kHashDecodeQuadMax", "kHashDecodeTwoMax"))


@pytest.fixture(scope="module")
def wl():
    return W.WL.config_compressed(96, 8, seed=21, invalid_frac=0.25)


@pytest.mark.parametrize("lanes", [6, 1])
@pytest.mark.parametrize("n", [1, 4, 5, 11, 12, 13, 16, 17, 33, QUAD, QUAD + 1, TWO, TWO + 1, TWO + 17])
def test_batch_sizes(wl, n, lanes):
    pick = np.arange(n) * 5 % 96
    with G.Context(lanes=lanes) as c:
        ids = np.asarray(c.register_pk_affine_batch(wl["pk_affine"]), dtype=np.int32)
        for _ in range(2):
            res = c.verify_messages(wl["sigs_compressed"][pick].tobytes(), [wl["msgs"][i] for i in pick],
                                    ids[wl["pk_index"][pick]], W.DST, compressed=True)
            assert (res == wl["expect"][pick]).all()
    if n > 96:
        assert set(wl["expect"].tolist()) >= {1, 0, -1, -2, -3, -4}
