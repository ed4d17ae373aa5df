"""A call that fails after it has queued copies from page-locked caller memory returns
only when they are done; offsets that decrease are refused before anything is queued."""
import numpy as np
import pytest
import torch

import bls_gpu as G
import workload_py as W

pytestmark = pytest.mark.gpu

ITEMS = 1 << 20


@pytest.fixture(scope="module")
def big():
    """page-locked items (their copy takes milliseconds) and a context that has room for
    them, but not for their messages"""
    wl = W.WL.config_compressed(n=8, nkeys=2, seed=3, invalid_frac=0.0)
    sigs = torch.zeros((ITEMS, 12), dtype=torch.int64).pin_memory()
    ids = torch.zeros(ITEMS, dtype=torch.int32).pin_memory()
    with G.Context(max_pks=4, mem_cap_bytes=ITEMS * 300) as ctx:
        ctx.register_pk_affine_batch(wl["pk_affine"])
        yield ctx, sigs, ids


def call(ctx, sigs, ids, offsets):
    msgs = np.zeros(int(offsets.max()) or 1, dtype=np.uint8)      # not touched: never paged in
    res = np.zeros(ITEMS, dtype=np.int32)
    dst = np.frombuffer(W.DST, dtype=np.uint8).copy()
    return ctx.lib.bls_verify_messages(ctx.h, G.SIG_AFFINE, sigs.data_ptr(), G._ptr(msgs), G._ptr(offsets), ids.data_ptr(),
                                       ITEMS, G._ptr(dst), dst.size, G._ptr(res))


def test_no_copy_is_left_behind_by_an_error(big):
    ctx, sigs, ids = big
    stream = torch.cuda.ExternalStream(ctx.stream())
    offsets = (np.arange(ITEMS + 1, dtype=np.uint64) * 1000).astype(np.uint32)
    for _ in range(3):
        assert call(ctx, sigs, ids, offsets) == -4            # BLS_ERR_NOMEM: the messages' buffer
        assert stream.query()


def test_decreasing_offsets_queue_nothing(big):
    ctx, sigs, ids = big
    stream = torch.cuda.ExternalStream(ctx.stream())
    offsets = np.arange(ITEMS + 1, dtype=np.uint32)
    offsets[ITEMS // 2] = 0
    for _ in range(3):
        assert call(ctx, sigs, ids, offsets) == G.BLS_ERR_INVALID
        assert stream.query()
