"""Persistent block updates of device streams of every length modulo 8, each
followed by bytes that do not belong to it (terminators and bytes above 16,
which the block's checks would count)."""
import numpy as np
import pytest
import torch

import oracle as O
from conftest import make_batch
from gmpt import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail", range(8))
@pytest.mark.parametrize("junk", [16, 17, 255])
def test_streams_of_every_length(gpu_lib, tail, junk):
    rng = W.Xoshiro256ss(8 * junk + tail, lanes=64)
    n = 40
    nibs = [[int(x) & 15 for x in rng.words(6)] + [c >> 4, c & 15, 16] for c in range(n)]
    nibs[-1] = [1] * (1 + (tail - sum(map(len, nibs[:-1])) - 2) % 8) + [16]  # the key stream ends at tail mod 8
    vals = [rng.bytes(5).tobytes() for _ in range(n - 1)]
    vals.append(rng.bytes(1 + (tail - 5 * (n - 1) - 1) % 8).tobytes())
    b = make_batch(nibs, vals)
    assert len(b.keys_hexs) % 8 == tail and len(b.values) % 8 == tail
    o = O.OracleTrie()
    o.puts(b.keys_hexs, b.keys_indexs, b.values, b.values_indexs)
    o.hash()
    dev = []
    for a in (b.keys_hexs, b.values):
        dev.append(torch.from_numpy(np.concatenate([a, np.full(16, junk, np.uint8)])).cuda())
    idx = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (b.keys_indexs, b.values_indexs, np.zeros(n, np.int32))]
    torch.cuda.synchronize()
    t = gpu_lib.MPT()
    for _ in range(2):
        got = t.block_update_device(dev[0].data_ptr(), idx[0].data_ptr(), dev[1].data_ptr(), idx[1].data_ptr(),
                                    idx[2].data_ptr(), 0, 0, n, n, len(b.keys_hexs), len(b.values), [0])
        assert got == [o.root()]
    assert t.get_values(b.keys_hexs, b.keys_indexs) == vals
    t.close()
