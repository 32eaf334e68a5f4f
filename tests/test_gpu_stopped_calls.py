"""Calls after one that stopped half way (an allocation that cannot succeed,
made after the batch was begun): its error is reported once, and the trie --
whose counts the host then reads anew -- takes deletes, puts, blocks and
hashes as before."""
import numpy as np
import pytest
import torch

import oracle as O
from gmpt import workloads as W

pytestmark = pytest.mark.gpu


def oracle_root(*batches):
    o = O.OracleTrie()
    for b in batches:
        o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    o.hash()
    return o.root()


@pytest.mark.parametrize("two_phase", [False, True])
@pytest.mark.parametrize("then", ["delete", "put", "block", "hash"])
def test_after_a_put_that_ran_out_of_memory(gpu_lib, two_phase, then):
    a = W.random_keys(5000, 20, 40, seed=0x5EED0D01)
    b = W.random_keys(4000, 20, 40, seed=0x5EED0D02)
    t = gpu_lib.MPT()
    put = t.puts_2phase_with_valuehp if two_phase else t.puts_latching_with_valuehp_v2
    put(a.keys_hexs, a.keys_indexs, a.values, a.values_indexs)
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda()
           for x in (b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)]
    torch.cuda.synchronize()
    with pytest.raises(gpu_lib.GmptError) as ei:  # an arena of 16 TiB is refused on the host
        t.puts_device(two_phase, *[d.data_ptr() for d in dev], b.n, len(b.keys_hexs), 1 << 44)
    assert ei.value.code == 1 and "memory" in str(ei.value)
    left = [a]
    if then == "delete":
        gone = a.subset(np.arange(0, a.n, 3))
        t.deletes(gone.keys_hexs, gone.keys_indexs)
        left = [a.subset(np.array([i for i in range(a.n) if i % 3]))]
    elif then == "put":
        put(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
        left = [a, b]
    elif then == "block":
        roots = t.block_update(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs, np.zeros(b.n, np.int32), b.n, [0])
        left = [a, b]
        assert roots == [oracle_root(a, b)]
    t.hash_onepass_v2()
    assert t.get_root_hash() == oracle_root(*left)
    t.close()
