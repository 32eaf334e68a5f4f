"""Growth of large node pools: past 8 GiB a pool has an allocation per array
and grows array by array, so a branch pool of 84 GB can still grow to 120 on a
device that could not hold both; tries keep their nodes through every form of
a pool."""
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


def test_nodes_survive_every_form_of_the_pools(gpu_lib):
    bs = [W.random_keys(4000, 20, 30, seed=0x5EED1100 + k) for k in range(4)]
    t = gpu_lib.MPT()
    # branch pool: 120 bytes a node, short pool 64, records 24: one block, then arrays, then larger arrays
    for b, nodes in zip(bs, (0, 4 << 20, 80 << 20, 140 << 20)):
        if nodes:
            t.reserve_nodes(nodes, nodes, nodes, nodes, 1 << 20, 1 << 20)
        t.puts_latching_with_valuehp_v2(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
        if nodes != 80 << 20:  # one growth with dirty nodes pending
            t.hash_onepass_v2()
    assert t.get_root_hash() == oracle_root(*bs)
    for b in bs:
        want = [b.values.reshape(-1, 30)[i].tobytes() for i in range(b.n)]
        assert t.get_values(b.keys_hexs, b.keys_indexs) == want
    t.close()


def test_a_pool_beyond_half_of_the_device_grows(gpu_lib):
    free, _ = torch.cuda.mem_get_info()
    if free < 160 << 30:
        pytest.skip("needs 160 GiB of free device memory")
    b = W.random_keys(4000, 20, 30, seed=0x5EED1110)
    t = gpu_lib.MPT()
    t.reserve_nodes(700_000_000, 8000, 8000, 8000, 1 << 20, 1 << 20)  # 84 GB of branches
    t.puts_latching_with_valuehp_v2(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    t.reserve_nodes(1_000_000_000, 8000, 8000, 8000, 1 << 20, 1 << 20)  # 120 GB
    t.hash_onepass_v2()
    assert t.get_root_hash() == oracle_root(b)
    t.close()
