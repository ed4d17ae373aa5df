"""The 32-item kernel with several lanes to an item (small batches and the last, nearly
empty wave of large ones): accept bits, Miller and Gt values at the batch sizes where
the dispatch changes, over normalised and raw line tables, with and without a key
index, affine and compressed, and in a persistent launch, against the oracle."""
import numpy as np
import pytest
import torch

import bls_gpu as G
import cpu as C
import workload_py as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.fixture(scope="module")
def wl(golden):
    w = W.WL.config_compressed(n=96, nkeys=5, seed=41, invalid_frac=0.1)
    w["want"], w["ml"], w["gt"] = C.verify_batch(w["sigs"], w["nhms"], golden["g2_gen_coeffs"], w["pk_tables"],
                                                 pk_index=w["pk_index"], want_values=True, nthreads=8)
    return w


# (waves of 32 a SM, eighths of one, items more)
SIZES = [(0, 0, 1), (0, 0, 9), (0, 2, -1), (0, 2, 0), (0, 2, 1), (0, 4, 0), (0, 4, 1), (1, 0, 0), (1, 0, 1), (1, 2, 1),
         (2, 4, 0), (1, 4, 1)]


@pytest.mark.parametrize("raw", [False, True], ids=["normalised", "raw"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%d-%d/8%+d" % s)
def test_values_at_dispatch_edges(wl, sms, size, raw):
    waves, eighths, more = size
    n = 32 * sms * waves + 4 * sms * eighths + more
    pick = np.concatenate([np.random.default_rng(n).permutation(96), np.arange(n)])[:n] % 96
    with G.Context() as ctx:
        ids = ctx.register_pk_affine_batch(wl["pk_affine"])
        if raw:                                  # a table with a zero c2 turns normalised lines off
            bad = wl["pk_tables"][0].copy()
            bad[24:36] = 0
            ctx.register_pk_coeffs(bad)
        values = n <= 16 * sms
        got = ctx.verify(wl["sigs"][pick], wl["nhms"][pick], ids[wl["pk_index"][pick]], want_values=values)
        if values:
            assert (got[1] == wl["ml"][pick]).all() and (got[2] == wl["gt"][pick]).all()
        assert ((got[0] if values else got) == wl["want"][pick]).all()
        if not raw:
            res = ctx.verify(wl["sigs_compressed"][pick], wl["nhms"][pick], ids[wl["pk_index"][pick]], compressed=True)
            assert (res == wl["expect"][pick]).all()
            cut = n // 3
            reqs = [(wl["sigs"][p], wl["nhms"][p], ids[wl["pk_index"][p]]) for p in (pick[:cut], pick[cut:])]
            assert (np.concatenate(ctx.verify_requests(reqs)) == wl["want"][pick]).all()


def test_a_table_per_item_over_the_last_wave(wl, sms, golden):
    """the reference entry point with mostly distinct tables: no key index"""
    n = 32 * sms + 13
    rng = np.random.default_rng(5)
    tabs = np.broadcast_to(wl["pk_tables"][0], (n, 2448)).copy()
    tabs[:, :5] = rng.integers(0, 2 ** 60, (n, 5), dtype=np.uint64)      # a c0 of its own
    pick = np.arange(n) % 96
    tabs[-40:] = wl["pk_tables"][wl["pk_index"][pick[-40:]]]             # the tail's own keys
    got = np.array(G.batch_bls_verify(wl["sigs"][pick], wl["nhms"][pick], golden["g2_gen_coeffs"], tabs), dtype=np.int32)
    assert (got[-40:] == wl["want"][pick[-40:]]).all() and got[-40:].any()
    assert not got[:-40].any()
