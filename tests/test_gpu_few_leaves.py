"""Hash passes of more than 2^17 dirty nodes with few leaves in the
list: keys that end at branches of a binary trie are updated, and a few of the
leaves below, on both sides of the number that is hashed a warp each."""
import numpy as np
import pytest

import oracle as O
from gmpt import workloads as W

pytestmark = pytest.mark.gpu

BASE = 17  # letters of the longest words: 2^17 leaves, a key at every branch


def words(ln):
    i = np.arange(1 << ln)
    return np.stack([97 + ((i >> (ln - 1 - k)) & 1) for k in range(ln)], 1).astype(np.uint8)


def batch(parts, value_bytes, seed):
    lens = np.concatenate([np.full(len(p), p.shape[1]) for p in parts]).astype(np.int64)
    kh, ki = W.keys_to_hexs(np.concatenate([p.reshape(-1) for p in parts]), lens)
    vb, vi = W.fixed_values(W.Xoshiro256ss(seed, lanes=1024), len(lens), value_bytes)
    return W.Batch(kh, ki, vb, vi)


@pytest.mark.parametrize("value_bytes", [40, 200])
@pytest.mark.parametrize("mode", [O.MODE_REF, O.MODE_GETH])
def test_few_leaves_in_a_large_list(gpu_lib, mode, value_bytes):
    full, pre = words(BASE), [words(ln) for ln in range(1, BASE)]
    load = batch([full] + pre, 20, 0x5EED1201)
    o = O.OracleTrie(mode)
    t = gpu_lib.MPT(mode=mode)
    o.puts(load.keys_hexs, load.keys_indexs, load.values, load.values_indexs)
    t.puts_2phase_with_valuehp(load.keys_hexs, load.keys_indexs, load.values, load.values_indexs)
    t.hash_onepass_v2()
    o.hash()
    assert t.get_root_hash() == o.root()
    for k, leaves in enumerate((0, 1, 2048, 2049)):
        sel = np.sort(np.random.default_rng(k).choice(len(full), leaves, replace=False))
        b = batch(pre + ([full[sel]] if leaves else []), value_bytes, 0x5EED1202 + k)
        o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
        o.hash()
        t.puts_latching_with_valuehp_v2(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
        t.hash_onepass_v2()
        assert t.get_root_hash() == o.root(), leaves
        s = t.stats()
        # the leaves' launch, and one over the branches of the deep trie
        assert s["last_dirty"] > 1 << 17 and s["last_hash_levels"] == (2 if leaves else 1)
    t.close()
