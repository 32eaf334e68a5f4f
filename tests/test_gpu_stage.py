"""Staging of a batch in one pass: device streams at any byte offset, pairs
that do not tile the stream, host batches on both sides of the packed copy,
and malformed batches, which must leave the trie as it was."""
import numpy as np
import pytest

import oracle as O
from conftest import make_batch, nib
from gmpt import workloads as W

pytestmark = pytest.mark.gpu


def oracle_root(*batches):
    o = O.OracleTrie()
    for b in batches:
        o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    o.hash()
    return o.root()


def at_offset(a, off):
    """A device copy of array a starting `off` bytes into an allocation."""
    import torch

    raw = np.ascontiguousarray(a).view(np.uint8)
    t = torch.zeros(len(raw) + 64, dtype=torch.uint8, device="cuda:0")
    t[off: off + len(raw)] = torch.from_numpy(raw.copy()).cuda()
    return t, t.data_ptr() + off


@pytest.mark.parametrize("two_phase", [False, True])
@pytest.mark.parametrize("off", [0, 1, 4, 8, 15])
def test_device_streams_at_any_offset(gpu_lib, two_phase, off):
    import torch

    for n, vb in ((1, 1), (3, 7), (1000, 33), (20001, 5)):
        b = W.random_keys(n, 11, vb, seed=0x5EED0B00 + n)
        keep = [at_offset(a, off) for a in (b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)]
        torch.cuda.synchronize()
        t = gpu_lib.MPT()
        for _ in range(2):  # the second batch starts at another arena offset
            t.puts_device(two_phase, *[p for _, p in keep], n, len(b.keys_hexs), len(b.values))
        t.hash_onepass_v2()
        assert t.get_root_hash() == oracle_root(b), (n, vb)
        t.close()


@pytest.mark.parametrize("two_phase", [False, True])
@pytest.mark.parametrize("n", [1, 900, 1100, 40000])  # 256 KiB of host arrays lie in between
def test_host_batches_and_lookups(gpu_lib, two_phase, n):
    b = W.random_keys(n, 32, 100, seed=0x5EED0B10 + n)
    hps = np.arange(1, n + 1, dtype=np.uint64)
    t = gpu_lib.MPT()
    put = t.puts_2phase_with_valuehp if two_phase else t.puts_latching_with_valuehp_v2
    put(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs, hps)
    t.hash_onepass_v2()
    assert t.get_root_hash() == oracle_root(b)
    hp, size = t.gets_parallel(b.keys_hexs, b.keys_indexs)
    assert np.array_equal(hp, hps) and np.all(size == 100)
    t.close()


@pytest.mark.parametrize("two_phase", [False, True])
@pytest.mark.parametrize("tiled", [True, False])
@pytest.mark.parametrize("bad", [17, 200, 16])
def test_malformed_batches_are_not_applied(gpu_lib, two_phase, tiled, bad):
    first = W.random_keys(500, 8, 20, seed=0x5EED0B20)
    b = W.random_keys(3000, 8, 20, seed=0x5EED0B21)
    kh, ki = b.keys_hexs.copy(), b.keys_indexs.copy()
    if not tiled:  # a hole in front of every key
        kh = np.concatenate([np.zeros((b.n, 1), np.uint8), kh.reshape(b.n, -1)], axis=1).reshape(-1)
        ki = ki + np.repeat(np.arange(1, b.n + 1, dtype=np.int32), 2)
    t = gpu_lib.MPT()
    put = t.puts_2phase_with_valuehp if two_phase else t.puts_latching_with_valuehp_v2
    put(first.keys_hexs, first.keys_indexs, first.values, first.values_indexs)
    t.hash_onepass_v2()
    good = kh.copy()
    kh[ki[2 * 1234] + 3] = bad  # an interior nibble
    with pytest.raises(gpu_lib.GmptError) as ei:
        put(kh, ki, b.values, b.values_indexs)
    assert ei.value.code == 2
    t.hash_onepass_v2()
    assert t.get_root_hash() == oracle_root(first)
    put(good, ki, b.values, b.values_indexs)
    t.hash_onepass_v2()
    assert t.get_root_hash() == oracle_root(first, b)
    t.close()


@pytest.mark.parametrize("off", [0, 1, 7])
def test_lookups_of_every_key_length(gpu_lib, off):
    """Stored keys, and keys that differ in the first, a middle or the last
    nibble, of 1 to 70 bytes (leaf keys of 1 to 140 nibbles), read from device
    memory at any byte offset, the last key ending its allocation's view."""
    import torch

    rng = W.Xoshiro256ss(5 + off, lanes=256)
    keys, vals = [], []
    for size in range(1, 71):
        for c in (1, 2):
            keys.append(nib(bytes([size, c]) + rng.bytes(size).tobytes()))
            vals.append(bytes(size))
    b = make_batch(keys, vals)
    hps = np.arange(1, len(keys) + 1, dtype=np.uint64)
    t = gpu_lib.MPT()
    t.puts_2phase_with_valuehp(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs, hps)
    asked, want = [], []
    for i, k in enumerate(keys):
        asked.append(k)
        want.append(i + 1)
        for at in (4, 4 + (len(k) - 5) // 2, len(k) - 2):  # behind the two bytes every key has its own
            asked.append(k[:at] + [k[at] ^ 5] + k[at + 1:])
            want.append(0)
    q = make_batch(asked, [b"x"] * len(asked))
    n = len(asked)
    dk = at_offset(q.keys_hexs, off)
    di = torch.from_numpy(q.keys_indexs.copy()).cuda()
    hp = torch.zeros(n, dtype=torch.int64, device="cuda:0")
    ln = torch.zeros(n, dtype=torch.int32, device="cuda:0")
    torch.cuda.synchronize()
    t.gets_device(dk[1], di.data_ptr(), n, len(q.keys_hexs), hp.data_ptr(), ln.data_ptr())
    assert hp.cpu().tolist() == want
    assert ln.cpu().tolist() == [len(vals[w - 1]) if w else 0 for w in want]
    host_hp, _ = t.gets_parallel(q.keys_hexs, q.keys_indexs)
    assert host_hp.tolist() == want
    t.close()


@pytest.mark.parametrize("off", [0, 1, 4, 8])
def test_block_arrays_at_any_offset(gpu_lib, off):
    """A block update from device arrays read where they lie (or copied, where
    their alignment asks for it) equals the same block from host arrays."""
    import torch

    rng = W.Xoshiro256ss(31 + off, lanes=64)
    n0, n = 700, 741
    b = W.random_keys(n, 16, 48, seed=0x5EED0B30)
    tid = np.concatenate([1 + (rng.words(n0) % np.uint64(40)).astype(np.int32), np.zeros(n - n0, np.int32)])
    pt = np.concatenate([np.full(n0, -1, np.int32), np.arange(n - n0, dtype=np.int32)])
    po = np.full(n, 5, np.int32)
    out_ids = np.arange(41, dtype=np.int32)
    host = gpu_lib.MPT(max_tries=41)
    keep = [at_offset(a, off) for a in (b.keys_hexs, b.keys_indexs, b.values, b.values_indexs, tid, pt, po)]
    torch.cuda.synchronize()
    t = gpu_lib.MPT(max_tries=41)
    for _ in range(2):  # the second one replays the captured launch (and patches another root of trie 0 in)
        want = host.block_update(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs, tid, n0, out_ids, pt, po)
        got = t.block_update_device(*[p for _, p in keep], n, n0, len(b.keys_hexs), len(b.values), out_ids)
        assert got == want
    assert t.get_roots(out_ids) == want
    host.close()
    t.close()
