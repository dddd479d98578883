"""The host-array calls on pinned memory, which the kernels use in place, on
pageable memory and on arrays that share memory, which are copied: the same
results, all equal to the oracle's map."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import unique_u32, unique_u64

pytestmark = pytest.mark.gpu


def _host(a, kind):
    import torch
    if kind == "pageable":
        return a
    raw = np.ascontiguousarray(a).view(np.uint8)
    pad = a.itemsize if kind == "pinned offset" else 0  # not on the allocation's first byte
    p = torch.zeros(raw.size + pad, dtype=torch.uint8).pin_memory().numpy()
    p[pad:] = raw
    return p[pad:].view(a.dtype)


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("n", [1, 33, 32768, 32769, 100001])
@pytest.mark.parametrize("kind", ["pageable", "pinned", "pinned offset", "in place"])
def test_host_arrays_match_oracle(kb, n, kind):
    import databases_gpu_gb300 as dg
    rng = np.random.default_rng(n + kb)
    kt = np.uint32 if kb == 4 else np.uint64
    pool = (unique_u32 if kb == 4 else unique_u64)(2 * n + 2, seed=n).astype(kt)
    t = dg.DyCuckoo(4 * n + 1024, key_bytes=kb, value_bytes=kb)
    m = O.Map()
    where = "pinned" if kind == "in place" else kind
    k = pool[rng.integers(0, n + 1, n)]  # repeats
    k[rng.random(n) < 0.01] = 0
    v = rng.integers(1, 1 << 31, n).astype(kt)
    t.insert_host(_host(k, where), _host(v, where))
    m.insert(k.astype(np.uint64), v.astype(np.uint64))
    q = pool[rng.integers(0, 2 * n + 2, n)]
    keys = _host(q, where)
    out = keys if kind == "in place" else _host(np.full(n, 7, kt), where)
    bits = _host(np.full((n + 31) // 32, 0xFFFFFFFF, np.uint32), where)
    t.find_host(keys, out, bits)
    ov, oh = m.find(q.astype(np.uint64))
    assert np.array_equal(out.astype(np.uint64), ov)
    hit = np.unpackbits(bits.view(np.uint8), bitorder="little")[:n].astype(bool)
    assert np.array_equal(hit, oh.astype(bool))
    eb = _host(np.full((n + 31) // 32, 0xFFFFFFFF, np.uint32), where)
    cnt = t.erase_host(_host(q, where), eb)
    _, eh = m.erase(q.astype(np.uint64))
    gone = np.unpackbits(eb.view(np.uint8), bitorder="little")[:n].astype(bool)
    assert cnt == int(eh.sum()) and np.array_equal(gone, eh.astype(bool))
    assert t.size == len(m)
    t.close()


@pytest.mark.parametrize("n", [3 << 22, (3 << 22) + 1])
def test_long_pinned_finds_match_device_finds(n):
    """The longest find in place and the shortest one by copies."""
    import torch
    import databases_gpu_gb300 as dg
    from tests.helpers import to_dev, to_host
    pool = unique_u32(1 << 21, seed=3)
    t = dg.DyCuckoo(pool.size)
    t.insert(to_dev(pool[: 1 << 20]), to_dev(pool[: 1 << 20] ^ np.uint32(0x77)))
    q = pool[np.random.default_rng(n).integers(0, pool.size, n)]
    out = _host(np.full(n, 7, np.uint32), "pinned")
    bits = _host(np.full((n + 31) // 32, 0xFFFFFFFF, np.uint32), "pinned")
    t.find_host(_host(q, "pinned"), out, bits)
    dv, db = t.find(to_dev(q))
    assert np.array_equal(out, to_host(dv, 4))
    assert np.array_equal(bits.view(np.int32), db.cpu().numpy())
    t.close()
