"""Branches hashed a pair of lanes each (every wave: warp_full_max 0) under
extensions whose own encoding takes more than one Keccak block, alone in their
warp, side by side, and next to branches with a short extension or none."""
import pytest

import oracle as O
from conftest import make_batch, nib
from gmpt import workloads as W

pytestmark = pytest.mark.gpu


# 97 packed key bytes fill one block ([header 2][key header 2][98 bytes with the flag][33]); 98 and more take two
@pytest.mark.parametrize("head", [96, 97, 98, 99, 150, 400])
@pytest.mark.parametrize("groups", [1, 2, 40, 700])
@pytest.mark.parametrize("mode", [O.MODE_REF, O.MODE_GETH])
def test_long_extensions(gpu_lib, mode, groups, head):
    rng = W.Xoshiro256ss(1000 * head + groups, lanes=64)
    for mixed in (False, True):
        keys = []
        for g in range(groups):
            size = head if not mixed or g % 3 else 1 + g % 4
            pre = bytes([g >> 4, (g & 15) * 16]) + rng.bytes(size).tobytes()
            keys += [pre + bytes([16 * c]) + rng.bytes(1).tobytes() for c in range(2 + g % 4)]
        vals = [rng.bytes(1 + i % 40).tobytes() for i in range(len(keys))]
        b = make_batch([nib(k) for k in keys], vals)
        o = O.OracleTrie(mode)
        o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
        o.hash()
        t = gpu_lib.MPT(mode=mode)
        t.set_option("warp_full_max", 0)
        t.puts_2phase_with_valuehp(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
        t.hash_onepass_v2()
        assert t.get_root_hash() == o.root(), mixed
        t.close()
