"""GPU parity of batches resolved by bins (dyc_bins.cuh) against the oracle's
map: sizes at the edges of the small-batch kernel (32768 ops, bins of 384) and
of the split kernels' tiles, batches of distinct keys, of few keys (bins that
go over their capacity and take the general path) and of both together, key 0,
and 8-byte keys with equal record tags. Whole numbers: everything is equal."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import assert_same_contents, to_dev, to_host, unique_u32, unique_u64

pytestmark = pytest.mark.gpu


def _keys(rng, kb, n, pattern):
    """n keys: all but a few distinct, drawn from 7 keys, or half and half; some are 0."""
    if kb == 4:
        pool = unique_u32(n + 8, seed=n + 1)
    else:
        pool = unique_u64(n + 8, seed=n + 1)
        # equal tags: low word = high word * 0x85EBCA6B
        hi = np.arange(1, min(n, 60) + 1, dtype=np.uint64)
        pool[: hi.size] = (hi << np.uint64(32)) | ((hi * np.uint64(0x85EBCA6B)) & np.uint64(0xFFFFFFFF))
    few = pool[rng.integers(0, 7, n)]
    if pattern == "distinct":
        k = pool[rng.permutation(n)]
        k[rng.integers(0, n, n // 50)] = k[0]
    elif pattern == "few":
        k = few
    else:
        k = np.where(rng.random(n) < 0.5, few, pool[rng.permutation(n)])
    k[rng.random(n) < 0.01] = 0
    return np.ascontiguousarray(k)


@pytest.mark.parametrize("kb,vb", [(4, 4), (8, 8), (8, 4)])
@pytest.mark.parametrize("pattern", ["distinct", "few", "both"])
@pytest.mark.parametrize("n", [1, 2, 385, 4096, 32768, 32769, 70001, 300007])
def test_batches_by_bins_match_oracle(kb, vb, pattern, n):
    import databases_gpu_gb300 as dg
    rng = np.random.default_rng(n * 10 + kb)
    vd = np.uint32 if vb == 4 else np.uint64
    t = dg.DyCuckoo(1024, key_bytes=kb, value_bytes=vb)  # grows on the way: counted passes too
    m = O.Map()
    for step in range(3):
        k = _keys(rng, kb, n, pattern)
        v = rng.integers(1, 1 << 31, n).astype(vd)
        ops = rng.choice(np.array([0, 1, 2], np.uint8), size=n)
        out, bits = t.apply(to_dev(ops), to_dev(k), to_dev(v))
        ov, oh = m.apply(ops, k.astype(np.uint64), v.astype(np.uint64))
        assert np.array_equal(dg.unpack_bits(bits, n), oh), step
        assert np.array_equal(to_host(out, vb).astype(np.uint64), ov), step
        assert_same_contents(t, m, "apply %d" % step)

        k = _keys(rng, kb, n, pattern)
        v = rng.integers(1, 1 << 31, n).astype(vd)
        st = t.insert(to_dev(k), to_dev(v))
        before = len(m)
        m.insert(k.astype(np.uint64), v.astype(np.uint64))
        distinct = np.unique(k[k != 0]).size
        assert st["rejected"] == int((k == 0).sum())
        assert st["inserted"] == len(m) - before
        assert st["updated"] == distinct - st["inserted"]
        assert st["superseded"] == int((k != 0).sum()) - distinct
        assert_same_contents(t, m, "insert %d" % step)

        k = _keys(rng, kb, n, pattern)
        import torch
        eb = torch.full(((n + 31) // 32,), -1, dtype=torch.int32, device="cuda")
        got = t.erase(to_dev(k), erased_bits=eb)
        _, eh = m.erase(k.astype(np.uint64))
        assert got == int(eh.sum())
        assert np.array_equal(dg.unpack_bits(eb, n), eh)
        assert_same_contents(t, m, "erase %d" % step)
    t.close()


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("pattern", ["distinct", "few", "both"])
@pytest.mark.parametrize("n", [1024, 32769, 100003])
def test_wide_batches_by_bins(kb, pattern, n):
    """Rows of 12 bytes: the last row of a key wins, an erase returns it once."""
    from databases_gpu_gb300.table import DyCuckooWide
    import databases_gpu_gb300 as dg
    rng = np.random.default_rng(n + kb)
    w = DyCuckooWide(2 * n, 12, key_bytes=kb)
    k = _keys(rng, kb, n, pattern)
    rows = rng.integers(1, 1 << 30, (n, 3)).astype(np.int32)
    st = w.insert(to_dev(k), to_dev(rows.view(np.uint32).reshape(-1)))
    uniq, last = np.unique(k[::-1], return_index=True)  # last occurrence of each key
    want = {int(a): rows[n - 1 - int(b)] for a, b in zip(uniq, last) if a}
    assert st["inserted"] == len(want) == w.size
    v, bits = w.find(to_dev(uniq))
    hit = dg.unpack_bits(bits, uniq.size)
    assert np.array_equal(hit, uniq != 0)
    got = v.cpu().numpy()
    for a, r in zip(uniq[hit], got[hit]):
        assert np.array_equal(want[int(a)], r)
    e = _keys(rng, kb, n, pattern)
    cnt, ev, eb = w.erase(to_dev(e))
    first = np.zeros(n, bool)
    first[np.unique(e, return_index=True)[1]] = True
    gone = first & np.isin(e, uniq[uniq != 0])
    assert cnt == int(gone.sum()) and np.array_equal(dg.unpack_bits(eb, n), gone)
    ev = ev.cpu().numpy()
    assert not ev[~gone].any()
    assert all(np.array_equal(want[int(a)], r) for a, r in zip(e[gone], ev[gone]))
    assert w.size == len(want) - cnt
    w.close()
