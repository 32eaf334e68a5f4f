"""Deletes make room for the keys their collapses append, not for the longest
key of the trie each: with one key of 1000 nibbles the arena grows by what is
needed, and the trie is the oracle's, for every shape of collapse."""
import numpy as np
import pytest

import oracle as O
from conftest import make_batch, nib
from gmpt import workloads as W

pytestmark = pytest.mark.gpu

LONG = bytes(range(1, 251)) * 2  # 500 bytes


def root_of(mode, items):
    if not items:
        return b""
    ks = sorted(items)
    o = O.OracleTrie(mode)
    b = make_batch([nib(k) for k in ks], [items[k] for k in ks])
    o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    o.hash()
    return o.root()


def test_one_long_key_does_not_size_the_arena(gpu_lib):
    b = W.random_keys(200000, 20, 8, seed=0x5EED1001)
    one = make_batch([nib(LONG)], [b"long"])
    t = gpu_lib.MPT()
    for x in (b, one):
        t.puts_latching_with_valuehp_v2(x.keys_hexs, x.keys_indexs, x.values, x.values_indexs)
    t.hash_onepass_v2()
    before = t.stats()
    gone, kept = b.subset(np.flatnonzero(np.arange(b.n) % 4 != 0)), b.subset(np.arange(0, b.n, 4))
    t.deletes(gone.keys_hexs, gone.keys_indexs)
    after = t.stats()
    # some 50K branches collapse into keys of about 40 nibbles (2 MB); 1008 bytes each would be 50 MB
    assert after["key_bytes"] - before["key_bytes"] < 4 << 20
    assert after["device_bytes"] - before["device_bytes"] < 20 << 20
    t.hash_onepass_v2()
    o = O.OracleTrie()
    for x in (kept, one):
        o.puts(x.keys_hexs, x.keys_indexs, x.values, x.values_indexs)
    o.hash()
    assert t.get_root_hash() == o.root()
    t.close()


@pytest.mark.parametrize("mode", [O.MODE_REF, O.MODE_GETH])
@pytest.mark.parametrize("alpha,max_len", [(2, 9), (3, 12), (256, 4)])
def test_collapses_of_every_shape(gpu_lib, mode, alpha, max_len):
    """Chains of collapses, branches that vanish, values at branches,
    extensions above and below, in a trie whose long key makes the bound too
    large for the arena."""
    rng = W.Xoshiro256ss(0xDE20 + alpha + mode, lanes=256)
    keys = set()
    while len(keys) < 700:
        w = rng.words(max_len + 1)
        keys.add(bytes(int(x) % alpha for x in w[1: 2 + int(w[0] % np.uint64(max_len))]))
    items = {k: rng.bytes(1 + int(rng.words(1)[0] % np.uint64(50))).tobytes() for k in sorted(keys)}
    items[LONG] = b"long"
    t = gpu_lib.MPT(mode=mode)

    def put(part):
        ks = list(part)
        b = make_batch([nib(k) for k in ks], [part[k] for k in ks])
        t.puts_2phase_with_valuehp(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)

    put(items)
    t.hash_onepass_v2()
    for share in (200, 700, 950, 1000):
        sel = [k for k in sorted(items) if int(rng.words(1)[0] % np.uint64(1000)) < share and k != LONG]
        if not sel:
            continue
        b = make_batch([nib(k) for k in sel], [b"x"] * len(sel))
        t.deletes(b.keys_hexs, b.keys_indexs)
        t.hash_onepass_v2()
        dropped = {k: items.pop(k) for k in sel}
        assert t.get_root_hash() == root_of(mode, items), share
        back = {k: v for i, (k, v) in enumerate(dropped.items()) if i % 3 == 0 and share < 1000}
        if back:  # dirty nodes of a put that was not hashed yet are in the next delete's list
            put(back)
            items.update(back)
    t.close()
