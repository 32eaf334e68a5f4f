"""Workloads of the batched trie update path, as its users call it.

A case is one kind of work (``op``) at one size.  Batches have the layout of
the reference's callers (hex-nibble keys with inclusive index pairs, raw value
bytes with inclusive index pairs) and are made on the GPU from the seed:

  load      bulk load of an empty trie, root hash (a snapshot import)
  step      bulk load of YCSB-shaped keys + root, then as many zipf(0.99)
            updates of them + root: the benchmark's step
  vocab     bulk load of variable-length word keys with values of 128 B - 4 KB
  update    zipf updates of a trie that is already there + root
  request   one drained window of a request loop over the tenants of a forest:
            the library picks the schedule, then hash + the tenants' roots
  gets      lookups in a standing trie, nine in ten present
  mixed     read/write batch on a standing trie (reads answered in index
            order) + root
  delete    keys deleted + root, then put back + root
  block     Ethereum-shaped block: storage tries, their roots written into
            account values, the state trie, all roots, in one launch
  small     a handful of keys from host arrays: put, root, look up
  pipeline  host batches (pinned) with copy / compute overlap: load + updates
  keccak    Keccak-256 of host rows (account addresses, storage slots)
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT / "gpu-merkle-patricia-trie_b200"))

import gmpt  # noqa: E402

DEV = "cuda:0"


def listed():
    return [
        # one transaction's worth of state changes through the host API
        {"name": "small_31", "op": "small", "n": 31, "base": 200003},
        # a request of the serving loop's lower end, four tenants, schedule chosen by the library
        {"name": "request_1000", "op": "request", "n": 1000, "base": 262144, "tries": 4, "key_bytes": 41},
        # YCSB update window on a 1M-key store
        {"name": "update_16k", "op": "update", "n": 16384, "base": 1 << 20, "two_phase": False},
        # an Ethereum block (275 accounts and their storage) on a 1M-account state
        {"name": "block_275", "op": "block", "accounts": 275, "base": 1 << 20},
        # pruning: an odd number of accounts removed and restored (PhaseNU insert into a live trie)
        {"name": "delete_65521", "op": "delete", "n": 65521, "base": 1 << 20, "two_phase": True},
        # read-mostly store window, 95 % reads
        {"name": "mixed_256k", "op": "mixed", "n": 262144, "base": 1 << 20, "write_pct": 5, "two_phase": False},
        # snapshot import of raw (not yet hex) 20-byte keys, LockNU, ragged count
        {"name": "load_raw_300007", "op": "load", "n": 300007, "key_bytes": 20, "value_bytes": 33, "raw": True,
         "two_phase": False},
        # 2^20 random 32-byte keys, 64-byte values, PhaseNU: the reference's bulk-load experiment
        {"name": "load_1m", "op": "load", "n": 1 << 20, "key_bytes": 32, "value_bytes": 64, "raw": False,
         "two_phase": True},
        # article titles: word keys of 8 - 96 B, long values
        {"name": "vocab_512k", "op": "vocab", "n": 1 << 19, "two_phase": True},
        # point lookups
        {"name": "gets_2m", "op": "gets", "n": 2000003, "base": 1 << 22},
        # end to end from pinned host memory
        {"name": "pipeline_1m", "op": "pipeline", "n": 1 << 20},
        # the benchmark's step: 16M inserts + 16M zipf updates
        {"name": "step_16m", "op": "step", "n": 1 << 24},
    ]


def draw(rng):
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["load", "step", "vocab", "update", "request", "gets", "mixed", "delete", "block", "small",
                     "pipeline", "keccak"])
    if op == "small":
        return {"op": op, "n": span(1, 256), "base": span(1000, 1 << 20)}
    if op == "request":
        tries, kb = rng.randint(1, 16), rng.randint(20, 96)
        return {"op": op, "n": span(1000, 1 << 20), "base": span(4096, min(1 << 20, (1 << 30) // (tries * (2 * kb + 1)))),
                "tries": tries, "key_bytes": kb}
    if op == "update":
        return {"op": op, "n": span(256, 1 << 18), "base": span(1 << 14, 1 << 22), "two_phase": rng.random() < 0.3}
    if op == "block":
        return {"op": op, "accounts": span(20, 400), "base": span(1 << 14, 1 << 21)}
    if op == "delete":
        return {"op": op, "n": span(100, 1 << 17), "base": 1 << rng.randint(18, 21), "two_phase": rng.random() < 0.5}
    if op == "mixed":
        return {"op": op, "n": span(1000, 1 << 20), "base": span(1 << 16, 1 << 22),
                "write_pct": rng.choice([5, 20, 50]), "two_phase": rng.random() < 0.3}
    if op == "load":
        return {"op": op, "n": span(1000, 1 << 23), "key_bytes": rng.choice([20, 32]),
                "value_bytes": rng.randint(1, 120), "raw": rng.random() < 0.3, "two_phase": rng.random() < 0.6}
    if op == "vocab":
        return {"op": op, "n": span(1000, 1 << 20), "two_phase": rng.random() < 0.7}
    if op == "gets":
        return {"op": op, "n": span(1000, 1 << 23), "base": span(1 << 16, 1 << 22)}
    if op == "pipeline":
        return {"op": op, "n": span(1 << 12, 1 << 21)}
    if op == "keccak":
        return {"op": op, "n": span(1000, 1 << 20), "width": rng.choice([20, 32, 64, 100, 140, 300])}
    return {"op": "step", "n": span(1000, 1 << 23)}


# --------------------------------------------------------------------------
# inputs


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _bytes(g, *shape):
    return torch.randint(0, 256, shape, dtype=torch.uint8, device=DEV, generator=g)


def _pairs(n, size, dtype):
    """Inclusive index pairs of n items of one size, back to back."""
    s = torch.arange(n, device=DEV, dtype=torch.int64) * size
    return torch.stack([s, s + (size - 1)], 1).reshape(-1).to(dtype)


def _hex(kb):
    """Rows of key bytes -> rows of nibbles + terminator."""
    n, m = kb.shape
    out = torch.empty((n, 2 * m + 1), dtype=torch.uint8, device=DEV)
    out[:, 0:2 * m:2] = kb >> 4
    out[:, 1:2 * m:2] = kb & 15
    out[:, 2 * m] = 16
    return out


def _ycsb_rows(g, n):
    """'user' + 19 decimal digits of a hashed id, as nibble rows."""
    out = torch.empty((n, 47), dtype=torch.uint8, device=DEV)
    for i, c in enumerate(b"user"):
        out[:, 2 * i] = c >> 4
        out[:, 2 * i + 1] = c & 15
    out[:, 8:46:2] = 3
    out[:, 9:46:2] = torch.randint(0, 10, (n, 19), dtype=torch.uint8, device=DEV, generator=g)
    out[:, 46] = 16
    return out


def _zipf(g, items, n, theta=0.99):
    """n zipfian draws over `items` ids, scrambled over the id space."""
    u = torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
    zetan = float(torch.arange(1, items + 1, dtype=torch.float64, device=DEV).pow(-theta).sum())
    zeta2 = 1.0 + 0.5 ** theta
    eta = (1.0 - (2.0 / items) ** (1.0 - theta)) / (1.0 - zeta2 / zetan)
    r = (items * (eta * u - eta + 1.0).clamp_min(0.0).pow(1.0 / (1.0 - theta))).to(torch.int64)
    uz = u * zetan
    r = torch.where(uz < zeta2, torch.ones_like(r), r)
    r = torch.where(uz < 1.0, torch.zeros_like(r), r)
    return torch.randperm(items, device=DEV, generator=g)[r.clamp(0, items - 1)]


class Dev:
    """A device-resident batch: key rows, values and their index pairs."""

    def __init__(self, rows, vals, vidx):
        self.n = rows.shape[0]
        self.keys = rows.reshape(-1)
        self.kidx = _pairs(self.n, rows.shape[1], torch.int32)
        self.vals = vals
        self.vidx = vidx

    @classmethod
    def fixed(cls, rows, g, value_bytes):
        n = rows.shape[0]
        return cls(rows, _bytes(g, n * value_bytes), _pairs(n, value_bytes, torch.int64))

    @classmethod
    def sized(cls, rows, g, sizes):
        vals, vidx = _sized_values(g, sizes)
        return cls(rows, vals, vidx)

    def args(self):
        return (self.keys.data_ptr(), self.kidx.data_ptr(), self.vals.data_ptr(), self.vidx.data_ptr(), self.n,
                self.keys.numel(), self.vals.numel())


def _sized_values(g, sizes):
    end = torch.cumsum(sizes, 0)
    return _bytes(g, int(end[-1])), torch.stack([end - sizes, end - 1], 1).reshape(-1)


def _word_keys(g, n):
    """Keys of 8 - 96 B made of zipf-drawn words of a 10k vocabulary, hex
    nibbles back to back, with their index pairs."""
    v, most = 10000, 49
    wl = torch.randint(2, 11, (v,), device=DEV, generator=g)
    woff = torch.cumsum(wl, 0) - wl
    letters = torch.randint(97, 123, (int(wl.sum()),), dtype=torch.uint8, device=DEV, generator=g)
    klen = (3.0 + 0.5 * torch.randn(n, device=DEV, generator=g)).exp().round().clamp(8, 96).to(torch.int64)
    words = _zipf(g, v, n * most, 0.8).reshape(n, most)
    cum = torch.cumsum(wl[words], 1)
    piece = torch.minimum(wl[words], (klen[:, None] - (cum - wl[words])).clamp_min(0)).reshape(-1)
    used = torch.nonzero(piece).reshape(-1)
    piece, start = piece[used], woff[words.reshape(-1)[used]]
    pend = torch.cumsum(piece, 0)
    src = torch.repeat_interleave(start - (pend - piece), piece) + torch.arange(int(pend[-1]), device=DEV)
    kb = letters[src]
    kid = torch.repeat_interleave(torch.arange(n, device=DEV), klen)
    pos = 2 * torch.arange(kb.numel(), device=DEV) + kid
    end = torch.cumsum(2 * klen + 1, 0)
    out = torch.full((int(end[-1]),), 16, dtype=torch.uint8, device=DEV)
    out[pos] = kb >> 4
    out[pos + 1] = kb & 15
    return out, torch.stack([end - (2 * klen + 1), end - 1], 1).reshape(-1).to(torch.int32)


# --------------------------------------------------------------------------


def _root(t):
    return np.frombuffer(t.get_root_hash(), np.uint8)


def _base(t, rows, g, value_bytes=100, hps=0):
    """A standing trie: `rows` loaded and hashed."""
    b = Dev.fixed(rows, g, value_bytes)
    torch.cuda.synchronize()
    t.puts_device(True, *b.args(), hps)
    t.hash_onepass_v2()


def _room(t, n, key_bytes, value_bytes, new=0.0, most=4 << 30):
    """Pool room for many more batches of n keys (a server's reservation)."""
    per = max(1, n * (key_bytes + value_bytes + 24) + int(new * n * 300))
    k = max(2, min(20000, most // per))
    t.reserve_nodes(int(2 * n + new * n * k), int(4 * n + 2 * new * n * k), int(n + new * n * k), n * k + 1,
                    n * k * key_bytes + 64 * k, n * k * value_bytes + 64 * k)


class State:
    pass


def prepare(case, seed):
    g = _gen(seed)
    s = State()
    s.op, s.case = case["op"], case
    n = case.get("n", 0)
    if s.op in ("load", "vocab", "step"):
        s.t = t = gmpt.MPT()
        if s.op == "load":
            kb = _bytes(g, n, case["key_bytes"])
            s.b = Dev.fixed(kb if case["raw"] else _hex(kb), g, case["value_bytes"])
        elif s.op == "vocab":
            keys, kidx = _word_keys(g, n)
            sizes = (6.0 + 0.8 * torch.randn(n, device=DEV, generator=g)).exp().round().clamp(128, 4096)
            s.b = Dev.sized(keys[:n].reshape(n, 1), g, sizes.to(torch.int64))
            s.b.keys, s.b.kidx = keys, kidx
        else:
            rows = _ycsb_rows(g, n)
            s.b = Dev.fixed(rows, g, 100)
            s.u = Dev.fixed(rows[_zipf(g, n, n)], g, 100)
        k = 2 if s.op == "step" else 1
        hexs = s.b.keys.numel() * (2 if case.get("raw") else 1) + n
        t.reserve_nodes(2 * n + (n // 2 if k == 2 else 0), 4 * n + (2 * n if k == 2 else 0), k * n, k * n, k * hexs,
                        k * s.b.vals.numel())
    elif s.op == "update":
        s.t = t = gmpt.MPT()
        rows = _ycsb_rows(g, case["base"])
        _base(t, rows, g)
        s.b = Dev.fixed(rows[_zipf(g, case["base"], n)], g, 100)
        _room(t, n, 47, 100)
    elif s.op == "request":
        tries, per, kb = case["tries"], case["base"], case["key_bytes"]
        s.t = t = gmpt.MPT(max_tries=tries + 1)
        rows = _hex(_bytes(g, tries * per, kb))
        tid = torch.arange(tries * per, device=DEV, dtype=torch.int64) // per
        b = Dev.fixed(rows, g, 32)
        torch.cuda.synchronize()
        base_tid = tid.to(torch.int32)
        a = b.args()
        t.puts_forest_device(True, *a[:4], base_tid.data_ptr(), *a[4:])
        t.hash_onepass_v2()
        # zipf updates of each tenant's keys; the window's requests are put back to back
        old = _zipf(g, per, n) + torch.sort(torch.randint(0, tries, (n,), device=DEV, generator=g))[0] * per
        s.tid = tid[old].to(torch.int32)
        s.b = Dev.fixed(rows[old], g, 32)
        s.touched = torch.unique(s.tid).cpu().numpy().astype(np.int32)
        s.trie_keys = per * len(s.touched)
        _room(t, n, 2 * kb + 1, 32)
        t.reserve_block(n, n * (2 * kb + 1), n * 32, tries)
        s.sel = gmpt.CSelector()
    elif s.op == "gets":
        s.t = t = gmpt.MPT()
        rows = _hex(_bytes(g, case["base"], 32))
        hps = torch.arange(1, case["base"] + 1, device=DEV, dtype=torch.int64)
        _base(t, rows, g, 64, hps.data_ptr())
        pick = rows[torch.randint(0, case["base"], (n,), device=DEV, generator=g)]
        absent = torch.rand(n, device=DEV, generator=g) < 0.1
        pick[absent, 12:60] = torch.randint(0, 16, (int(absent.sum()), 48), dtype=torch.uint8, device=DEV, generator=g)
        s.b = Dev.fixed(pick, g, 1)
        s.hp = torch.zeros(n, dtype=torch.int64, device=DEV)
        s.len = torch.zeros(n, dtype=torch.int32, device=DEV)
    elif s.op == "mixed":
        s.t = t = gmpt.MPT()
        rows = _ycsb_rows(g, case["base"])
        hps = torch.arange(1, case["base"] + 1, device=DEV, dtype=torch.int64)
        _base(t, rows, g, 100, hps.data_ptr())
        # a fixed number of writes at random places; a read carries no value
        s.rw = torch.zeros(n, dtype=torch.uint8, device=DEV)
        s.rw[torch.randperm(n, device=DEV, generator=g)[:max(1, n * case["write_pct"] // 100)]] = 1
        s.b = Dev.sized(rows[_zipf(g, case["base"], n)], g, 100 * s.rw.to(torch.int64))
        s.hp = torch.zeros(n, dtype=torch.int64, device=DEV)
        s.len = torch.zeros(n, dtype=torch.int32, device=DEV)
        _room(t, n, 47, case["write_pct"])
    elif s.op == "delete":
        s.t = t = gmpt.MPT()
        rows = _hex(_bytes(g, case["base"], 32))
        _base(t, rows, g, 64)
        s.b = Dev.fixed(rows[torch.randperm(case["base"], device=DEV, generator=g)[:n]], g, 64)
        _room(t, n, 65, 64, 1.0)
    elif s.op == "block":
        acc, base = case["accounts"], case["base"]
        s.t = t = gmpt.MPT(mode=gmpt.MODE_GETH, max_tries=acc + 1)
        rows = _hex(_bytes(g, base, 32))

        def account_sizes(k):
            return (70 + torch.randint(0, 9, (k,), device=DEV, generator=g)
                    + torch.randint(1, 33, (k,), device=DEV, generator=g))

        b = Dev.sized(rows, g, account_sizes(base))
        torch.cuda.synchronize()
        t.puts_device(True, *b.args())
        t.hash_onepass_v2()
        # entries per storage trie: density ~ s^-1.5 on [1, 5000]
        u = torch.rand(acc, dtype=torch.float64, device=DEV, generator=g)
        sizes = (u * (5000.0 ** -0.5 - 1.0) + 1.0).pow(-2.0).floor().clamp(1, 5000).to(torch.int64)
        n0 = int(sizes.sum())
        sid = torch.arange(1, acc + 1, device=DEV, dtype=torch.int32)
        srows = _hex(_bytes(g, n0, 32))
        arows = rows[torch.randperm(base, device=DEV, generator=g)[:acc]]
        av = account_sizes(acc)
        sv = torch.randint(1, 33, (n0,), device=DEV, generator=g)
        s.b = Dev.sized(torch.cat([srows, arows]), g, torch.cat([sv, av]))
        s.tid = torch.cat([torch.repeat_interleave(sid, sizes), torch.zeros(acc, dtype=torch.int32, device=DEV)])
        s.ptrie = torch.cat([torch.full((n0,), -1, dtype=torch.int32, device=DEV), sid])
        s.poff = torch.cat([torch.zeros(n0, dtype=torch.int32, device=DEV), (av - 65).to(torch.int32)])
        s.n0 = n0
        s.out_ids = np.arange(acc + 1, dtype=np.int32)
        _room(t, s.b.n, 65, 32)
        t.reserve_block(s.b.n, s.b.keys.numel(), s.b.vals.numel(), acc + 1)
    elif s.op == "small":
        s.t = t = gmpt.MPT(mode=gmpt.MODE_GETH)
        rows = _hex(_bytes(g, case["base"], 32))
        _base(t, rows, g, 64)
        b = Dev.fixed(rows[torch.randperm(case["base"], device=DEV, generator=g)[:n]], g, 64)
        s.host = [x.cpu().numpy() for x in (b.keys, b.kidx, b.vals, b.vidx)]
        s.hps = np.arange(1, n + 1, dtype=np.uint64)
        _room(t, n, 65, 64, most=256 << 20)
    elif s.op == "pipeline":
        s.t = t = gmpt.MPT()
        rows = _ycsb_rows(g, n)
        load, upd = Dev.fixed(rows, g, 100), Dev.fixed(rows[_zipf(g, n, n)], g, 100)
        s.pinned = [[x.cpu().pin_memory() for x in (b.keys, b.kidx, b.vals, b.vidx)] for b in (load, upd)]
        s.raw = [tuple(x.data_ptr() for x in p) + (n,) for p in s.pinned]
        t.reserve_nodes(2 * n + n // 2, 6 * n, 2 * n, 2 * n, 2 * n * 47, 2 * n * 100)
    else:
        s.msgs = _bytes(g, n, case["width"]).cpu().numpy()
    torch.cuda.synchronize()
    return s


def run(s):
    op, c = s.op, s.case
    t = getattr(s, "t", None)
    if op in ("load", "vocab"):
        t.reset()
        (t.puts_raw_device if c.get("raw") else t.puts_device)(c["two_phase"], *s.b.args())
        t.hash_onepass_v2()
        return _root(t)
    if op == "step":
        t.reset()
        out = []
        for b, two_phase in ((s.b, True), (s.u, False)):
            t.puts_device(two_phase, *b.args())
            t.hash_onepass_v2()
            out.append(_root(t))
        return out
    if op == "update":
        t.puts_device(c["two_phase"], *s.b.args())
        t.hash_onepass_v2()
        return _root(t)
    if op == "request":
        a = s.b.args()
        t.puts_auto_device(*a, d_tids=s.tid.data_ptr(), tries_touched=len(s.touched), trie_keys=s.trie_keys,
                           selector=s.sel)
        t.hash_onepass_v2()
        return [np.frombuffer(r, np.uint8) for r in t.get_roots(s.touched)]
    if op == "gets":
        t.gets_device(s.b.keys.data_ptr(), s.b.kidx.data_ptr(), s.b.n, s.b.keys.numel(), s.hp.data_ptr(),
                      s.len.data_ptr())
        return s.hp, s.len
    if op == "mixed":
        a = s.b.args()
        reads = t.puts_with_read_device(c["two_phase"], *a[:2], s.rw.data_ptr(), *a[2:], s.hp.data_ptr(),
                                        s.len.data_ptr())
        t.hash_onepass_v2()
        return s.hp[:reads], s.len[:reads], _root(t)
    if op == "delete":
        a = s.b.args()
        t.deletes_device(a[0], a[1], a[4], a[5])
        t.hash_onepass_v2()
        gone = _root(t)
        t.puts_device(c["two_phase"], *a)
        t.hash_onepass_v2()
        return gone, _root(t)
    if op == "block":
        a = s.b.args()
        out = np.zeros(32 * len(s.out_ids), np.uint8)
        sizes = np.zeros(len(s.out_ids), np.int32)
        t.block_update_device(*a[:4], s.tid.data_ptr(), s.ptrie.data_ptr(), s.poff.data_ptr(), s.b.n, s.n0, a[5], a[6],
                              s.out_ids, out, sizes)
        return out, sizes
    if op == "small":
        t.puts_latching_with_valuehp_v2(*s.host, s.hps)
        t.hash_onepass_v2()
        root = _root(t)
        hps, sizes = t.gets_parallel(s.host[0], s.host[1])
        return root, hps.view(np.int64), sizes
    if op == "pipeline":
        t.reset()
        return [np.frombuffer(r, np.uint8) for r in t.puts_pipeline(None, [True, False], raw=s.raw)]
    return gmpt.keccak256_rows(s.msgs)


def work(case):
    """Bytes in and out of one pass: the batch read once, its nibbles, values
    and records kept, 32 bytes of hash per key; lookups read the key and write
    12 bytes."""
    op, n = case["op"], case.get("n", 0)

    def put(k, v, stored):
        return n * (k + v + 24 + (k + v + 24 + 32 if stored else 8))

    if op == "load":
        k = case["key_bytes"]
        return {"bytes": n * ((k if case["raw"] else 2 * k + 1) + case["value_bytes"] + 24
                              + 2 * k + 1 + case["value_bytes"] + 56), "flops": 0}
    if op == "step":
        return {"bytes": 2 * put(47, 100, True), "flops": 0}
    if op == "vocab":
        return {"bytes": put(47, 555, True), "flops": 0}
    if op in ("update", "request", "small"):
        k = {"update": 47, "small": 65}.get(op) or 2 * case["key_bytes"] + 1
        return {"bytes": put(k, {"update": 100, "small": 64}.get(op, 32), True), "flops": 0}
    if op == "gets":
        return {"bytes": n * (65 + 8 + 12), "flops": 0}
    if op == "mixed":
        w = case["write_pct"] / 100.0
        return {"bytes": n * (47 + 9 + 12 * (1 - w) + w * (100 + 16 + 47 + 100 + 56)), "flops": 0}
    if op == "delete":
        return {"bytes": n * (65 + 8) + put(65, 64, True), "flops": 0}
    if op == "block":
        n = case["accounts"] * 71
        return {"bytes": put(65, 17, True), "flops": 0}
    if op == "pipeline":
        return {"bytes": 2 * put(47, 100, True), "flops": 0}
    return {"bytes": n * (case["width"] + 32), "flops": 0}
