"""PhaseNU's local sort when long keys keep the batch sort going past the last
chunk of shorter ones: a key and the same key followed by zero bytes tie on
every 8-nibble chunk and part by length alone."""
import numpy as np
import pytest

import oracle as O
from conftest import make_batch, nib
from gmpt import workloads as W

pytestmark = pytest.mark.gpu


# copies of each key of a pair: runs of 2, of 33 to 512 and of more than 512 positions
@pytest.mark.parametrize("copies", [1, 20, 300])
@pytest.mark.parametrize("prefix", [16, 24])
@pytest.mark.parametrize("longer_first", [False, True])
def test_keys_that_part_by_length_only(gpu_lib, prefix, copies, longer_first):
    rng = W.Xoshiro256ss(100 * prefix + copies, lanes=256)
    head = bytes(range(1, prefix + 1))
    keys = [head + rng.bytes(12).tobytes() for _ in range(3000)]  # more than one CTA's run, behind a shared prefix
    for short in (b"A", b"abc", b"abcdefg", b"zyxwvuts"):
        pair = [short, short + b"\0"] if copies > 1 else [short, short + b"\0", short + b"\0\0"]
        keys += (pair[::-1] if longer_first else pair) * copies
    vals = [rng.bytes(1 + i % 40).tobytes() for i in range(len(keys))]
    b = make_batch([nib(k) for k in keys], vals)
    o = O.OracleTrie()
    o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    o.hash()
    for split in (False, True):  # into an empty trie, and onto the long keys
        t = gpu_lib.MPT()
        parts = [b.subset(np.arange(3000)), b] if split else [b]
        for p in parts:
            t.puts_2phase_with_valuehp(p.keys_hexs, p.keys_indexs, p.values, p.values_indexs)
        t.hash_onepass_v2()
        assert t.get_root_hash() == o.root(), split
        assert t.get_values(b.keys_hexs, b.keys_indexs) == o.gets(b.keys_hexs, b.keys_indexs), split
        t.close()
