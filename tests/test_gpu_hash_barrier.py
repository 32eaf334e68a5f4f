"""Hash passes whose cooperative launch gives up at a grid barrier (the wait
set to 1 ns) are hashed again level by level: the call succeeds with the
oracle's root, and the trie goes on as before.  A value of many megabytes, one
serial chain, is not waited for at a barrier at all."""
import numpy as np
import pytest

import oracle as O
from conftest import make_batch, nib
from gmpt import workloads as W

pytestmark = pytest.mark.gpu

DEFAULT_NS = 2_000_000_000


def words(n, seed):
    """Keys over two letters, 12 to 20 of them: branches at some forty nibble depths."""
    rng = W.Xoshiro256ss(seed, lanes=1024)
    w = rng.words(2 * n)
    lens = 12 + (w[:n] % np.uint64(9)).astype(int)
    keys = [bytes(97 + ((int(x) >> k) & 1) for k in range(ln)) for x, ln in zip(w[n:], lens)]
    return make_batch([nib(k) for k in keys], [rng.bytes(1 + i % 60).tobytes() for i in range(n)])


def batches(kind):
    if kind == "deep":  # more dirty nodes than one launch takes, its branches at many depths
        return [words(120000, 0x5EED0C01), words(110000, 0x5EED0C02)]
    out = []
    for n, seed in ((20000, 0x5EED0C03), (3000, 0x5EED0C04), (300, 0x5EED0C05)):
        rng = W.Xoshiro256ss(seed, lanes=256)
        keys = [rng.bytes(20).tobytes() for _ in range(n)]
        vals = [rng.bytes(40).tobytes() for _ in keys[1:]] + [rng.bytes(100000).tobytes()]  # 736 blocks: the others wait
        out.append(make_batch([nib(k) for k in keys], vals))
    return out


@pytest.mark.parametrize("kind", ["whole", "deep"])
@pytest.mark.parametrize("two_phase", [False, True])
def test_a_pass_that_gives_up_is_hashed_by_levels(gpu_lib, kind, two_phase):
    o = O.OracleTrie()
    t, ref = gpu_lib.MPT(), gpu_lib.MPT()
    for x in (t, ref):
        x.set_timing(True)
        x.set_option("track_dirty", 1)
    for k, b in enumerate(batches(kind)):
        o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
        o.hash()
        for x in (t, ref):
            put = x.puts_2phase_with_valuehp if two_phase else x.puts_latching_with_valuehp_v2
            put(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
        t.set_option("block_barrier_ns", 1)
        t.hash_onepass_v2()
        ref.hash_onepass_v2()
        assert t.get_root_hash() == ref.get_root_hash() == o.root(), k
        a, z = t.stats(), ref.stats()
        assert a["last_hash_levels"] > z["last_hash_levels"], k  # the wait did run out
        assert [a[f] for f in ("last_hashed", "last_enc_bytes", "last_keccak_blocks")] == [
            z[f] for f in ("last_hashed", "last_enc_bytes", "last_keccak_blocks")], k
        t.hash_onepass_v2()  # nothing is left over
        assert t.get_root_hash() == o.root(), k
        t.set_option("block_barrier_ns", DEFAULT_NS)
    assert sorted(t.flush_dirty()) == sorted(ref.flush_dirty())
    # and cooperative passes again
    b = W.random_keys(3000, 20, 40, seed=0x5EED0C06)
    t.puts_latching_with_valuehp_v2(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    t.hash_onepass_v2()
    o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    o.hash()
    assert t.get_root_hash() == o.root() and t.stats()["last_hash_levels"] == 1
    t.close()
    ref.close()


@pytest.mark.parametrize("size", [(16 << 20) - 1, (16 << 20) + 1])
def test_values_of_many_megabytes(gpu_lib, size):
    rng = W.Xoshiro256ss(size, lanes=4096)
    keys = [bytes([c, 7, 9]) for c in range(200)]
    vals = [rng.bytes(30).tobytes() for _ in keys[1:]] + [rng.bytes(size).tobytes()]
    b = make_batch([nib(k) for k in keys], vals)
    o = O.OracleTrie()
    o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    o.hash()
    t = gpu_lib.MPT()
    t.puts_latching_with_valuehp_v2(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    t.hash_onepass_v2()
    assert t.get_root_hash() == o.root()
    assert (t.stats()["last_hash_levels"] > 1) == (size > 16 << 20)
    t.close()
