"""The cuckoo insert where its kernel changes: tables of 2^24 slots and more,
empty ones and ones that hold keys, calls that are captured.  New keys, keys
that are there, both in one call (those that are there first), keys that the
map refuses, values given or not, and chains that run out."""
import numpy as np
import pytest
import torch

import voxel_b200 as vx

pytestmark = pytest.mark.gpu
LINE = 1 << 24


def keys_of(n, device, seed):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    k = torch.unique(torch.randint(-2**63, 2**63 - 2, (n,), dtype=torch.int64, device=device,
                                   generator=g))
    return k[torch.randperm(k.numel(), device=device, generator=g)].contiguous()


@pytest.mark.parametrize("slots", [1 << 16, 1 << 20, (1 << 22) - 1, LINE, LINE + 2])
@pytest.mark.parametrize("load", [0.02, 0.8])
def test_insert_and_replace(cuda, slots, load):
    m = vx.CuckooMap(slots, 2000)
    keys = keys_of(int(slots * load), cuda, slots)
    n = keys.numel()
    half = n // 2
    st = torch.full((n,), -1, dtype=torch.int32, device=cuda)
    m.insert(keys[:half], None, st[:half])
    assert (st[:half] == vx.HASH_INSERTED).all()
    assert torch.equal(m.find(keys[:half]), torch.arange(half, dtype=torch.int32, device=cuda))
    values = torch.arange(n, dtype=torch.int32, device=cuda) * 3 + 1
    m.insert(keys, values, st)  # half there, half new
    assert (st[:half] == vx.HASH_REPLACED).all()
    assert (st[half:] == vx.HASH_INSERTED).all()
    assert torch.equal(m.find(keys), values)
    m.insert(keys, None, st)
    assert (st == vx.HASH_REPLACED).all()
    assert torch.equal(m.find(keys), torch.arange(n, dtype=torch.int32, device=cuda))
    assert m.dropped() == 0


@pytest.mark.parametrize("slots", [LINE, LINE + 2])
def test_refused_keys_and_a_full_table(cuda, slots):
    m = vx.CuckooMap(slots, 4)
    keys = keys_of(slots + slots // 8, cuda, 7)
    keys[5], keys[77] = -1, -2  # the two words that mark free and erased slots
    st = torch.full((keys.numel(),), -1, dtype=torch.int32, device=cuda)
    m.insert(keys, None, st)
    s = st.cpu().numpy()
    bad = [i for i in (5, 77) if s[i] == vx.HASH_INVALID_KEY]
    assert bad == [5, 77]
    lost = int((s == vx.HASH_OVERFLOW).sum())
    assert lost == m.dropped() > slots // 8 - 2
    assert (s == vx.HASH_INSERTED).sum() == keys.numel() - 2 - lost
    got = m.find(keys)
    held = got != np.uint32(vx.HASH_NOT_FOUND_VALUE).view(np.int32).item()
    # every key but the dropped ones is there, under its own index
    assert int(held.sum()) == keys.numel() - 2 - lost
    index = torch.arange(keys.numel(), dtype=torch.int32, device=cuda)
    assert torch.equal(got[held], index[held])


def test_a_captured_insert_leaves_no_table_known_empty(cuda):
    """A graph captured on an empty table fills it when it is replayed; the
    direct call after it replaces those keys and adds others."""
    slots = 1 << 20
    m = vx.CuckooMap(slots, 2000)
    keys = keys_of(int(slots * 0.8), cuda, 3)
    half = keys.numel() // 2
    there = keys[:half].contiguous()
    st = torch.full((keys.numel(),), -1, dtype=torch.int32, device=cuda)
    m.insert(there, None, st)
    m.clear()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        m.insert(there, None, st)
    m.clear()
    graph.replay()
    values = torch.arange(keys.numel(), dtype=torch.int32, device=cuda) + 5
    m.insert(keys, values, st)
    assert (st[:half] == vx.HASH_REPLACED).all()
    assert (st[half:] == vx.HASH_INSERTED).all()
    assert torch.equal(m.find(keys), values)
