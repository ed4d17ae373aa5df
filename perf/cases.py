"""Performance cases: the calls that a user of this library makes, by kind and size.

A kind is one public entry point (icp-gpu_b200/bls_gpu.py over the C ABI in
include/bls_gpu.h) together with what its caller holds before the call:

  verify      Context.verify: signatures, -H(m) and key ids in host memory, affine or
              48-byte compressed; optionally with the Miller and Gt values
  device      Context.verify_device: the same arrays and outputs resident on the GPU
  requests    Context.verify_requests: many uneven requests in one persistent launch
  serve       Server in slots mode: requests submitted one by one, then awaited
  messages    Context.verify_messages: RFC 9380 hash on the GPU, then the verify
  hash        Context.neg_hash_to_g1 alone
  decompress  Context.g1_decompress: points of a catch-up package
  keys        a fresh key set: a new Context, 96-byte keys decoded and prepared, the
              first signatures verified with their values
  rlc         Context.verify_rlc: one combined check over a batch of valid signatures, with
              the caller's random scalars, and the aggregates it checked
  reference   batch_bls_verify: the reference's entry point, a line table per item

Inputs follow the seeded workloads of icp-gpu_b200/workload.py (40 keys unless stated,
one item in eight corrupted, message flips and wrong keys).  Signing is the
CPU's work and slow, so a state signs at most POOL items and repeats them in random
order; the library does not look for equal items.

Every output is a whole number (accept bits, statuses, limbs of exact field elements),
so there are no values to compute in floating point.
"""
import importlib
import math

import numpy as np
import torch

G = importlib.import_module("icp-gpu_b200.bls_gpu")
WL = importlib.import_module("icp-gpu_b200.workload")

POOL = 1024
FP_MUL_IMAD = 588          # 32-bit multiply-adds of one 381-bit Montgomery product
VERIFY_FP_MULS = 16941     # two-pair Miller loop and final exponentiation
G1_DECODE_FP_MULS = 1550   # square root, 127 doublings and 16 additions of the subgroup test
HASH_FP_MULS = 2000        # two maps (a square root and the isogeny each), 63 doublings
KEY_FP_MULS = 5000         # Fp2 square root, the subgroup test, 68 lines
RLC_FP_MULS = 3100         # two 64-bit scalings and two subgroup tests
TABLE_BYTES = 2448 * 8


def listed():
    return [
        # one signature as it arrives, with its pairing values: latency alone
        {"name": "verify_1", "kind": "verify", "n": 1, "keys": 1, "compressed": False, "values": True},
        # a subnet's shares of one round, as they travel, an odd number of them
        {"name": "verify_compressed_333", "kind": "verify", "n": 333, "keys": 13, "compressed": True,
         "values": False},
        # the headline batch: inputs resident, 40 keys
        {"name": "device_4096", "kind": "device", "n": 4096, "keys": 40, "compressed": False, "values": False},
        # raw bytes of a long catch-up, 2% of them invalid encodings
        {"name": "verify_compressed_65536", "kind": "verify", "n": 65536, "keys": 40, "compressed": True,
         "values": False},
        # the batching workload: 256 requests of log-uniform size, over 50,000 items
        {"name": "requests_256", "kind": "requests", "n": 256, "max_size": 2048, "keys": 40, "compressed": False},
        # continuous batching: 48 requests in flight
        {"name": "serve_48", "kind": "serve", "n": 48, "max_size": 512, "keys": 40, "compressed": False},
        # a block's worth of signed messages, hashed on the GPU
        {"name": "messages_3000", "kind": "messages", "n": 3000, "keys": 40, "compressed": True, "max_len": 128},
        {"name": "hash_1000", "kind": "hash", "n": 1000, "max_len": 300},
        # the points of one catch-up package (the reference quotes its decoder at 448)
        {"name": "decompress_448", "kind": "decompress", "n": 448},
        # a new epoch's key set and its first signatures
        {"name": "keys_500", "kind": "keys", "n": 500},
        # a batch expected to be valid, combined
        {"name": "rlc_16384", "kind": "rlc", "n": 16384, "keys": 40, "compressed": False},
        # unchanged callers of the reference's ABI
        {"name": "reference_1024", "kind": "reference", "n": 1024, "keys": 40},
    ]


# kind -> smallest and largest n drawn (requests for the two request kinds).  The kinds that
# return accept bits alone begin where the bits of two seeds differ; the kinds with values at one.
RANGE = {"verify": (1, 32768), "device": (1, 32768), "requests": (12, 256), "serve": (12, 48),
         "messages": (32, 16384), "hash": (1, 16384), "decompress": (1, 32768), "keys": (1, 2048),
         "rlc": (1, 32768), "reference": (32, 2048)}


def draw(rng):
    kind = rng.choice(sorted(RANGE))
    n = int(round(math.exp(rng.uniform(*map(math.log, RANGE[kind])))))
    case = {"kind": kind, "n": n}
    if kind in ("verify", "device", "requests", "serve", "messages", "rlc", "reference"):
        case["keys"] = int(round(math.exp(rng.uniform(0.0, math.log(64)))))
    if kind in ("verify", "device", "requests", "serve", "messages", "rlc"):
        case["compressed"] = rng.random() < 0.5
    if kind in ("verify", "device"):
        case["values"] = n < 32 or rng.random() < 0.3
    if kind in ("requests", "serve"):
        case["max_size"] = int(round(math.exp(rng.uniform(math.log(8), math.log(512)))))
    if kind in ("messages", "hash"):
        case["max_len"] = int(round(math.exp(rng.uniform(0.0, math.log(600)))))
    return case


class _Context(G.Context):
    """A context that is released with its state."""

    def __del__(self):
        if getattr(self, "h", None):
            self.close()


class _Server(G.Server):
    def __init__(self, ctx, **kw):
        self.ctx = ctx          # outlives the server
        super().__init__(ctx, **kw)

    def __del__(self):
        if getattr(self, "h", None):
            self.close()


def _sizes(case):
    """log-uniform request sizes on [1, max_size], the same for every seed of a case"""
    u = np.random.default_rng(case["n"] + 1000 * case["max_size"]).random(case["n"])
    return np.clip(np.exp(u * math.log(case["max_size"] + 1)).astype(np.int64), 1, case["max_size"])


def _total(case):
    return int(_sizes(case).sum()) if case["kind"] in ("requests", "serve") else case["n"]


def _corruption(rng, n, nkeys):
    """one item in eight corrupted, at random: message flips (1) and, with several keys, wrong keys (2)"""
    return np.where(rng.random(n) < 0.125, rng.integers(1, 3 if nkeys > 1 else 2, n), 0).tolist()


def _invalidate(comp, frac, seed, rng):
    """invalid encodings of every kind in a fraction of the items"""
    n = comp.shape[0]
    bad = rng.permutation(n)[:int(round(frac * n))]
    off_curve = WL.special_points(seed + 1, 32, 0)
    outside = WL.special_points(seed + 2, 32, 1)
    for j, i in enumerate(bad):
        if j % 4 == 0:
            comp[i, 0] &= 0x7F                    # compression bit clear
        elif j % 4 == 1:
            comp[i, 0] |= 0x1F                    # x >= p
        elif j % 4 == 2:
            comp[i] = off_curve[(j // 4) % 32]
        else:
            comp[i] = outside[(j // 4) % 32]
    return comp


def _items(case, seed, rng, n, valid=False):
    """keys and n items: signed ones from a pool, repeated in random order"""
    nkeys = case["keys"]
    m = min(n, POOL)
    sm = WL.SplitMix64(seed)
    keys = WL._keys(sm, nkeys, with_tables=case["kind"] == "reference")
    corrupt = [0] * m if valid else _corruption(rng, m, nkeys)
    pool = WL._items(sm, keys, [i % nkeys for i in range(m)], corrupt)
    pick = np.concatenate([rng.permutation(m), rng.integers(0, m, n - m)])
    sigs = pool["sigs"][pick]
    if case.get("compressed"):
        sigs = WL.g1_compress(sigs)
        if not valid:
            sigs = _invalidate(sigs, 0.02, seed, rng)
    return keys, sigs, pool["nhms"][pick], pool["pk_index"][pick].astype(np.int32), [pool["msgs"][i] for i in pick]


def _messages(case, rng, n):
    return [rng.bytes(int(k)) for k in rng.integers(1, case["max_len"] + 1, n)]


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    rng = np.random.default_rng(seed)
    s = {"kind": kind, "n": n, "compressed": case.get("compressed", False)}
    if kind == "keys":
        sm = WL.SplitMix64(seed)
        keys = WL._keys(sm, n, with_tables=False)
        m = min(n, 512)
        it = WL._items(sm, keys, list(range(m)), _corruption(rng, m, n))
        s.update(pks=keys["pk_compressed"].tobytes(), sigs=it["sigs"], nhms=it["nhms"], index=it["pk_index"])
        return s
    if kind == "reference":
        keys, sigs, nhms, index, _ = _items(case, seed, rng, n)
        G.init()
        s.update(sigs=sigs, nhms=nhms, g2=_generator_table(), tables=np.ascontiguousarray(keys["pk_tables"][index]))
        return s
    ctx = s["ctx"] = _Context(max_pks=64)
    if kind == "decompress":
        sm = WL.SplitMix64(seed)
        m = min(n, POOL)
        points = WL.g1_mul(WL.hash_to_g1([sm.msg() for _ in range(m)]),
                           np.array([WL.scalar_limbs(sm.scalar()) for _ in range(m)], dtype=np.uint64))
        comp = WL.g1_compress(points)[np.concatenate([rng.permutation(m), rng.integers(0, m, n - m)])]
        s["points"] = _invalidate(comp, 0.02, seed, rng).tobytes()
        return s
    if kind == "hash":
        s["msgs"] = _messages(case, rng, n)
        return s
    sizes = _sizes(case) if kind in ("requests", "serve") else None
    total = n if sizes is None else int(sizes.sum())
    if kind == "messages":
        # messages of uneven length; each is hashed and signed here, on the CPU, up to POOL of them
        sm = WL.SplitMix64(seed)
        keys = WL._keys(sm, case["keys"], with_tables=False)
        m = min(n, POOL)
        lens = rng.integers(1, case["max_len"] + 1, 8)      # eight lengths: the CPU hash takes equal ones
        signer = np.arange(m) % case["keys"]
        msgs, sigs = [None] * m, np.zeros((m, 12), dtype=np.uint64)
        for c, length in enumerate(lens):
            ix = np.arange(c, m, 8)
            if ix.size:
                part = [rng.bytes(int(length)) for _ in ix]
                sigs[ix] = WL.g1_mul(WL.hash_to_g1(part, int(length)), keys["sk"][signer[ix]])
                for i, p in zip(ix, part):
                    msgs[i] = p
        pick = np.concatenate([rng.permutation(m), rng.integers(0, m, n - m)])
        index = signer[pick].astype(np.int32)
        wrong = rng.random(n) < 0.125
        sigs = sigs[pick]
        sigs[wrong] = np.roll(sigs, 1, axis=0)[wrong]      # another message's signature
        if case["compressed"]:
            sigs = _invalidate(WL.g1_compress(sigs), 0.02, seed, rng)
        s.update(sigs=sigs, msgs=[msgs[i] for i in pick])
    else:
        keys, sigs, nhms, index, _ = _items(case, seed, rng, total, valid=kind == "rlc")
        s.update(sigs=sigs, nhms=nhms)
    ids = ctx.register_pk_affine_batch(keys["pk_affine"])
    s["ids"] = np.ascontiguousarray(ids[index], dtype=np.int32)
    s["values"] = case.get("values", False)
    if kind == "rlc":
        s["scalars"] = rng.integers(1, 2 ** 63, total, dtype=np.uint64)
    if kind == "device":
        s["d_sigs"] = torch.from_numpy(sigs.view(np.uint8).reshape(-1).copy()).cuda()
        s["d_nhms"] = torch.from_numpy(nhms.view(np.int64)).cuda()
        s["d_ids"] = torch.from_numpy(s["ids"]).cuda()
        s["d_res"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        if s["values"]:
            s["d_ml"] = torch.zeros((n, 72), dtype=torch.int64, device="cuda")
            s["d_gt"] = torch.zeros((n, 72), dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()       # the library's stream does not wait for torch's
    if sizes is not None:
        at = np.concatenate([[0], np.cumsum(sizes)])
        s["requests"] = [(np.ascontiguousarray(s["sigs"][a:b]), np.ascontiguousarray(s["nhms"][a:b]),
                          np.ascontiguousarray(s["ids"][a:b])) for a, b in zip(at[:-1], at[1:])]
    if kind == "serve":
        s["server"] = _Server(ctx, compressed=case["compressed"], max_batch_items=8192)
    return s


_g2_table = []


def _generator_table():
    """the generator's line table, as a caller of the reference's ABI holds it"""
    if not _g2_table:
        with G.Context(max_pks=1) as ctx:
            _g2_table.append(ctx.pk_table(-1))
    return _g2_table[0]


def run(s):
    kind = s["kind"]
    if kind == "verify":
        return s["ctx"].verify(s["sigs"], s["nhms"], s["ids"], compressed=s["compressed"], want_values=s["values"])
    if kind == "device":
        out = {"ml_ptr": s["d_ml"].data_ptr(), "gt_ptr": s["d_gt"].data_ptr()} if s["values"] else {}
        s["ctx"].verify_device(s["n"], s["d_sigs"].data_ptr(), s["d_nhms"].data_ptr(), s["d_ids"].data_ptr(),
                               s["d_res"].data_ptr(), compressed=s["compressed"], **out)
        return (s["d_res"], s["d_ml"], s["d_gt"]) if s["values"] else s["d_res"]
    if kind == "requests":
        return np.concatenate(s["ctx"].verify_requests(s["requests"], compressed=s["compressed"]))
    if kind == "serve":
        tickets = [s["server"].submit(*r) for r in s["requests"]]
        for t, _, _ in tickets:
            s["server"].wait(t)
        return np.concatenate([res for _, _, res in tickets])
    if kind == "messages":
        return s["ctx"].verify_messages(s["sigs"], s["msgs"], s["ids"], WL.DST, compressed=s["compressed"])
    if kind == "hash":
        return s["ctx"].neg_hash_to_g1(s["msgs"], WL.DST)
    if kind == "decompress":
        return s["ctx"].g1_decompress(s["points"])
    if kind == "keys":
        with G.Context(max_pks=s["n"]) as ctx:
            ids, status = ctx.register_pk_compressed(s["pks"])
            return (ids, status, ctx.pk_table(int(ids[-1]))) + ctx.verify(s["sigs"], s["nhms"], ids[s["index"]],
                                                                          want_values=True)
    if kind == "rlc":
        return s["ctx"].verify_rlc(s["sigs"], s["nhms"], s["ids"], compressed=s["compressed"], scalars=s["scalars"],
                                   want_agg=True)
    if kind == "reference":
        return np.array(G.batch_bls_verify(s["sigs"], s["nhms"], s["g2"], s["tables"]), dtype=np.int32)
    raise ValueError(kind)


def work(case):
    """Inputs read once and outputs written once; 32-bit multiply-adds of the field products,
    two operations each."""
    kind, n = case["kind"], _total(case)
    comp = case.get("compressed", False)
    sig_bytes = 48 if comp else 96
    muls, nbytes = 0, 0
    if kind in ("verify", "device", "requests", "serve", "messages", "rlc"):
        muls += n * (G1_DECODE_FP_MULS if comp else 0)
        nbytes += n * (sig_bytes + 4 + 4) + case["keys"] * TABLE_BYTES
    if kind in ("verify", "device", "requests", "serve"):
        muls += n * VERIFY_FP_MULS
        nbytes += n * 96 + (n * 1152 if case.get("values") else 0)
    elif kind == "messages":
        muls += n * (VERIFY_FP_MULS + HASH_FP_MULS)
        nbytes += n * case["max_len"] // 2
    elif kind == "hash":
        muls += n * HASH_FP_MULS
        nbytes += n * (case["max_len"] // 2 + 96)
    elif kind == "decompress":
        muls += n * G1_DECODE_FP_MULS
        nbytes += n * (48 + 96 + 4)
    elif kind == "keys":
        m = min(n, 512)
        muls += n * KEY_FP_MULS + m * VERIFY_FP_MULS
        nbytes += n * (96 + TABLE_BYTES) + m * (196 + 1152)
    elif kind == "rlc":
        muls += n * RLC_FP_MULS + case["keys"] * VERIFY_FP_MULS
        nbytes += n * 96
    elif kind == "reference":
        muls += n * VERIFY_FP_MULS
        nbytes += n * (96 + 96 + 4) + case["keys"] * TABLE_BYTES
    return {"bytes": float(nbytes), "flops": 2.0 * FP_MUL_IMAD * muls}
