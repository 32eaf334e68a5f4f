"""The warp-cooperative node hashing (a warp builds one node's message in
8-block windows) vs the oracle, at the edges of blocks and windows: number of
children, values of 0 bytes to several windows in a branch, several long
values in one branch (keys without a terminator), long extension keys."""
import pytest

import oracle as O
from conftest import make_batch, nib
from gmpt import workloads as W

pytestmark = pytest.mark.gpu

MODES = [O.MODE_REF, O.MODE_GETH]


def check(gpu_lib, keys, vals, mode, warp_max):
    b = make_batch(keys, vals)
    o = O.OracleTrie(mode)
    o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    o.hash()
    t = gpu_lib.MPT(mode=mode)
    t.set_option("warp_full_max", warp_max)
    t.puts_2phase_with_valuehp(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    t.hash_onepass_v2()
    assert t.get_root_hash() == o.root()
    t.close()


@pytest.mark.parametrize("warp_max", [0, 4096])
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("vlen", [0, 1, 2, 31, 32, 33, 55, 56, 99, 100, 101, 135, 136, 255, 256, 483, 484, 1020, 1088,
                                  1089, 2175, 2176, 4096])
def test_branch_value_lengths(gpu_lib, mode, vlen, warp_max):
    """A key that ends at a branch of 1 to 16 children."""
    rng = W.Xoshiro256ss(1000 + vlen, lanes=64)
    for kids in (1, 2, 15, 16):
        keys = [nib(b"ab")] + [nib(b"ab" + bytes([16 * c, 7])) for c in range(kids)]
        vals = [rng.bytes(vlen).tobytes()] + [rng.bytes(1 + 9 * c).tobytes() for c in range(kids)]
        check(gpu_lib, keys, vals, mode, warp_max)


@pytest.mark.parametrize("mode", MODES)
def test_branch_of_many_long_values(gpu_lib, mode):
    """Keys without a terminator put their values straight into the slots."""
    rng = W.Xoshiro256ss(77, lanes=64)
    for size in (30, 33, 200, 1100):
        keys = [[5, c] for c in range(16)]
        vals = [rng.bytes(size + 13 * c).tobytes() for c in range(16)]
        check(gpu_lib, keys, vals, mode, 4096)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("klen", [1, 2, 3, 55, 56, 100, 101, 102, 103, 255, 400, 500])
def test_extension_and_leaf_key_lengths(gpu_lib, mode, klen):
    """klen bytes above a branch and klen bytes below it."""
    rng = W.Xoshiro256ss(klen, lanes=64)
    head = rng.bytes(klen // 2 + 1).tobytes()
    for tail in (0, 1, klen // 2):
        keys = [nib(head + bytes([c]) + rng.bytes(tail).tobytes()) for c in range(5)]
        vals = [rng.bytes(1 + 40 * c).tobytes() for c in range(5)]
        check(gpu_lib, keys, vals, mode, 4096)


@pytest.mark.parametrize("warp_max", [0, 1, 4096])
@pytest.mark.parametrize("mode", MODES)
def test_pass_sizes(gpu_lib, mode, warp_max):
    """Hash passes of one node to beyond one cooperative launch: new keys,
    updates and splits above untouched subtrees, deletes, both strategies."""
    t = gpu_lib.MPT(mode=mode)
    t.set_option("warp_full_max", warp_max)
    o = O.OracleTrie(mode)
    load = W.ycsb_load(60000, value_bytes=24, seed=0x5EED0A01)
    rand = W.random_keys(70000, 23, 24, seed=0x5EED0A02)  # same key length, other prefixes
    import numpy as np

    pos = 0
    for k, n in enumerate((1, 1, 2, 40, 700, 5000, 30000)):
        for b in (load.subset(np.arange(pos, pos + n)), load.subset(np.arange(max(0, pos - n // 2), pos + 1)),
                  rand.subset(np.arange(pos, pos + n))):
            put = t.puts_2phase_with_valuehp if k % 2 else t.puts_latching_with_valuehp_v2
            put(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
            o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
        t.hash_onepass_v2()
        o.hash()
        assert t.get_root_hash() == o.root(), (k, n)
        gone = rand.subset(np.arange(pos, pos + n))
        t.deletes(gone.keys_hexs, gone.keys_indexs)
        t.hash_onepass_v2()
        t.puts_2phase_with_valuehp(gone.keys_hexs, gone.keys_indexs, gone.values, gone.values_indexs)
        t.hash_onepass_v2()
        assert t.get_root_hash() == o.root(), (k, n)
        pos += n
    t.hash_onepass_v2()  # nothing dirty
    assert t.get_root_hash() == o.root()
    t.close()
