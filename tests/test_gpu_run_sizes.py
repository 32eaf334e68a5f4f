"""PhaseNU's CTA- and warp-local sort and build at the sizes where they change
hands (32, 512 and 2048 positions), with repeated keys, keys of different
lengths and keys that part only in their last nibble; scans of one element to
several tiles."""
import numpy as np
import pytest

import oracle as O
from conftest import make_batch, nib
from gmpt import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [O.MODE_REF, O.MODE_GETH])
@pytest.mark.parametrize("sizes", [(1, 2, 3), (31, 32, 33), (511, 512, 513, 30), (2047, 2048, 5), (2049, 33, 513)])
def test_runs_that_share_a_prefix(gpu_lib, mode, sizes):
    rng = W.Xoshiro256ss(sum(sizes), lanes=256)
    keys, vals = [], []
    for g, size in enumerate(sizes):
        head = bytes([7, g]) + b"prefix"  # runs tie on two chunks, then part
        for i in range(size):
            tail = rng.bytes(1 + i % 7).tobytes() if i % 5 else bytes([i % 3]) * 6
            keys.append(head + tail)
            if i % 11 == 0:  # a repeat, and a key that differs in its last nibble only
                keys.append(keys[-1][:-1] + bytes([keys[-1][-1] ^ 1]))
                keys.append(keys[-2])
    order = np.argsort(rng.words(len(keys)), kind="stable")
    keys = [keys[i] for i in order]
    vals = [rng.bytes(3 + i % 40).tobytes() for i in range(len(keys))]
    b = make_batch([nib(k) for k in keys], vals)
    o = O.OracleTrie(mode)
    o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    o.hash()
    for split in (False, True):  # into an empty trie, and onto its first half
        t = gpu_lib.MPT(mode=mode)
        parts = [b] if not split else [b.subset(np.arange(0, b.n // 2)), b.subset(np.arange(b.n // 2, b.n))]
        for p in parts:
            t.puts_2phase_with_valuehp(p.keys_hexs, p.keys_indexs, p.values, p.values_indexs)
        t.hash_onepass_v2()
        assert t.get_root_hash() == o.root(), (sizes, split)
        assert t.get_values(b.keys_hexs, b.keys_indexs) == o.gets(b.keys_hexs, b.keys_indexs)
        t.close()


@pytest.mark.parametrize("n", [1, 2, 4095, 4096, 4097, 65535, 70000])
def test_scan_tiles(gpu_lib, n):
    """Raw keys of different lengths: their offsets are one scan over n."""
    rng = W.Xoshiro256ss(n, lanes=1024)
    lens = 1 + (rng.words(n) % np.uint64(12)).astype(np.int64)
    offs = np.concatenate([[0], np.cumsum(lens)])
    raw = rng.bytes(int(offs[-1]))
    ki = np.stack([offs[:-1], offs[1:] - 1], 1).reshape(-1).astype(np.int32)
    vb, vi = W.fixed_values(rng, n, 9)
    kh, hi = W.keys_to_hexs(raw, lens)
    o = O.OracleTrie()
    o.puts(kh, hi, vb, vi)
    o.hash()
    for two_phase in (False, True):
        t = gpu_lib.MPT()
        t.puts_raw(two_phase, raw, ki, vb, vi)
        t.hash_onepass_v2()
        assert t.get_root_hash() == o.root()
        t.close()


@pytest.mark.parametrize("mode", [O.MODE_REF, O.MODE_GETH])
@pytest.mark.parametrize("width", [1, 2, 40])
def test_split_groups_in_pieces(gpu_lib, mode, width):
    """PhaseNU onto extensions that split while keys anchored below their
    branch sort between the splitting ones (and extensions that split on one
    side only, or next to each other)."""
    rng = W.Xoshiro256ss(width, lanes=64)
    first, second = [], []
    for g in range(width):
        p = [g >> 4, g & 15]
        first += [p + [5, 5, 5, c, 7, 7, 16] for c in range(4)]  # extension 5 5 5 above a branch of 4
        second += [p + [5, 5, 1, 0, 0, 0, 16], p + [5, 5, 5, 9, 0, 0, 16], p + [5, 5, 5, 1, 3, 0, 16],
                   p + [5, 5, 9, 0, 0, 0, 16], p + [5, 6, 0, 0, 0, 0, 16]][: 5 - g % 4]
        second += [p + [5, 5, 5, c, 7, 7, 16] for c in range(0, 4, 2)]  # updates in between
    batches = []
    for keys in (first, second):
        keys = [keys[i] for i in np.argsort(rng.words(len(keys)), kind="stable")]
        batches.append(make_batch(keys, [rng.bytes(1 + i % 50).tobytes() for i in range(len(keys))]))
    o = O.OracleTrie(mode)
    t = gpu_lib.MPT(mode=mode)
    for b in batches:
        o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
        o.hash()
        t.puts_2phase_with_valuehp(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
        t.hash_onepass_v2()
        assert t.get_root_hash() == o.root()
    t.close()
