"""Device entry points with the caller's arrays wherever they may lie: index
pairs and trie ids off their alignment, arrays in pinned host memory, arrays
that end with their allocation."""
import numpy as np
import pytest
import torch

import oracle as O
from gmpt import workloads as W

pytestmark = pytest.mark.gpu

TRIES = 5


def at_offset(a, off):
    raw = np.ascontiguousarray(a).view(np.uint8)
    t = torch.zeros(len(raw) + 64, dtype=torch.uint8, device="cuda:0")
    t[off: off + len(raw)] = torch.from_numpy(raw.copy()).cuda()
    return t, t.data_ptr() + off


def place(a, where):
    """(owner, address) of a copy of array a."""
    if isinstance(where, int):
        return at_offset(a, where)
    raw = torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).copy())
    t = raw.pin_memory() if where == "pinned" else raw.cuda()
    return t, t.data_ptr()


@pytest.fixture(scope="module")
def batch():
    b = W.random_keys(3000, 20, 40, seed=0x5EED0E01)
    tids = (np.arange(b.n) * 7 % TRIES).astype(np.int32)
    roots = []
    for tr in range(TRIES):
        s = b.subset(np.flatnonzero(tids == tr))
        o = O.OracleTrie()
        o.puts(s.keys_hexs, s.keys_indexs, s.values, s.values_indexs)
        o.hash()
        roots.append(o.root())
    return b, tids, roots


@pytest.mark.parametrize("where", [0, 1, 2, 3, "pinned", "exact"])
def test_lookups_and_deletes(gpu_lib, batch, where):
    b, tids, roots = batch
    hps = np.arange(1, b.n + 1, dtype=np.uint64)
    t = gpu_lib.MPT(max_tries=TRIES)
    t.puts_forest(False, b.keys_hexs, b.keys_indexs, b.values, b.values_indexs, tids, hps)
    t.hash_onepass_v2()
    assert t.get_roots(n=TRIES) == roots
    keep = [place(a, where) for a in (b.keys_hexs, b.keys_indexs, tids)]
    dk, di, dt = (p for _, p in keep)
    hp = torch.zeros(b.n, dtype=torch.int64, device="cuda:0")
    ln = torch.zeros(b.n, dtype=torch.int32, device="cuda:0")
    torch.cuda.synchronize()
    t.gets_device(dk, di, b.n, len(b.keys_hexs), hp.data_ptr(), ln.data_ptr(), d_tids=dt)
    assert hp.cpu().tolist() == hps.tolist() and set(ln.cpu().tolist()) == {40}
    got, size = t.gets_forest_device(dk, di, dt, b.n, len(b.keys_hexs))
    assert got.tolist() == hps.tolist() and set(size.tolist()) == {40}
    t.deletes_device(dk, di, b.n, len(b.keys_hexs), d_tids=dt)
    t.hash_onepass_v2()
    assert t.get_roots(n=TRIES) == [b""] * TRIES
    t.close()


@pytest.mark.parametrize("two_phase", [False, True])
@pytest.mark.parametrize("where", [0, 3, "pinned", "exact"])
def test_puts_and_blocks(gpu_lib, batch, two_phase, where):
    b, tids, roots = batch
    keep = [place(a, where) for a in (b.keys_hexs, b.keys_indexs, b.values, b.values_indexs, tids)]
    dk, di, dv, dx, dt = (p for _, p in keep)
    torch.cuda.synchronize()
    t = gpu_lib.MPT(max_tries=TRIES)
    t.puts_forest_device(two_phase, dk, di, dv, dx, dt, b.n, len(b.keys_hexs), len(b.values))
    t.hash_onepass_v2()
    assert t.get_roots(n=TRIES) == roots
    t.reset()
    ids = np.arange(TRIES, dtype=np.int32)
    assert t.block_update_device(dk, di, dv, dx, dt, 0, 0, b.n, b.n, len(b.keys_hexs), len(b.values), ids) == roots
    t.close()
