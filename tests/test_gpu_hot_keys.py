"""Batches with keys that repeat thousands of times (bins that go over their
capacity): inserts and erases against the oracle's map at the edges of the hot
pass's tiles of 4096 ops, and their time against distinct keys'."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import assert_same_contents, to_dev, unique_u32, unique_u64

pytestmark = pytest.mark.gpu


def _pool(kb, n, seed):
    return (unique_u32 if kb == 4 else unique_u64)(n, seed=seed).astype(np.uint32 if kb == 4 else np.uint64)


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("n", [36863, 36864, 36865, 131072])
@pytest.mark.parametrize("hot,share", [(1, 1.0), (2, 0.999), (40, 0.9), (3000, 1.0), (5, 0.3)])
def test_inserts_and_erases_of_hot_keys(kb, n, hot, share):
    """share of the ops on `hot` keys, the others distinct; some are key 0."""
    import torch
    import databases_gpu_gb300 as dg
    rng = np.random.default_rng(n + hot)
    pool = _pool(kb, n + hot, n)
    t = dg.DyCuckoo(4 * n, key_bytes=kb, value_bytes=kb)
    m = O.Map()
    for step in range(2):
        k = np.where(rng.random(n) < share, pool[rng.integers(0, hot, n)], pool[hot:][rng.permutation(n)])
        k[rng.random(n) < 0.001] = 0
        v = rng.integers(1, 1 << 31, n).astype(k.dtype)
        before = len(m)
        st = t.insert(to_dev(k), to_dev(v))
        m.insert(k.astype(np.uint64), v.astype(np.uint64))
        distinct = np.unique(k[k != 0]).size
        assert st["inserted"] == len(m) - before and st["updated"] == distinct - st["inserted"]
        assert st["superseded"] == int((k != 0).sum()) - distinct
        assert_same_contents(t, m, "insert %d" % step)
        e = np.where(rng.random(n) < share, pool[rng.integers(0, hot, n)], pool[hot:][rng.permutation(n)])
        eb = torch.full(((n + 31) // 32,), -1, dtype=torch.int32, device="cuda")
        got = t.erase(to_dev(e), erased_bits=eb)
        _, eh = m.erase(e.astype(np.uint64))
        assert got == int(eh.sum()) and np.array_equal(dg.unpack_bits(eb, n), eh)
        assert_same_contents(t, m, "erase %d" % step)
    t.close()


def _bin(keys, nbins):
    """The bin of each key among nbins (bin_of in dyc_bins.cuh)."""
    k = keys.astype(np.uint64)
    lo, hi = (k & np.uint64(0xFFFFFFFF)).astype(np.uint32), (k >> np.uint64(32)).astype(np.uint32)
    with np.errstate(over="ignore"):
        x = lo if keys.itemsize == 4 else (lo ^ hi ^ (np.uint32(0x9E3779B9) * hi)) ^ hi
        x = x ^ (x >> np.uint32(16))
        x = x * np.uint32(0x7FEB352D)
        x = x ^ (x >> np.uint32(15))
        x = x * np.uint32(0x846CA68B)
        x = x ^ (x >> np.uint32(16))
    return (x.astype(np.uint64) * np.uint64(nbins)) >> np.uint64(32)


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("bucket_bytes", [32, 64, 128])
@pytest.mark.parametrize("mix", ["one", "seven", "tenth", "hundred", "bin", "bin twice"])
@pytest.mark.parametrize("n", [1025, 2049, 8192, 24576])
def test_small_batches_with_a_bin_over_its_capacity(kb, bucket_bytes, mix, n):
    """Batches of one kernel in which a bin gets more than 1024 ops: a few keys,
    a tenth of the ops on one key, or distinct keys all of one bin (more than
    1024 of them: the bin is taken in parts), once and repeated."""
    import torch
    import databases_gpu_gb300 as dg
    rng = np.random.default_rng(n + kb)
    pool = _pool(kb, 1 << 20, n)
    nbins = (n + 383) // 384
    if mix.startswith("bin"):
        pool = np.concatenate([pool, _pool(kb, 3 << 20, n + 1)])
        pool = np.unique(pool[_bin(pool, nbins) == nbins // 2])
    draw = {"one": lambda: pool[np.zeros(n, np.int64)],
            "seven": lambda: pool[rng.integers(0, 7, n)],
            "hundred": lambda: pool[rng.integers(0, 100, n)],
            "tenth": lambda: np.where(rng.random(n) < 0.1, pool[0], pool[rng.integers(0, pool.size, n)]),
            "bin": lambda: pool[rng.permutation(pool.size)[np.arange(n) % pool.size]],
            "bin twice": lambda: pool[rng.integers(0, min(n // 2, pool.size), n)]}[mix]
    t = dg.DyCuckoo(2 * n, key_bytes=kb, value_bytes=kb, bucket_bytes=bucket_bytes)
    m = O.Map()
    for step in range(2):
        k = draw().copy()
        k[rng.random(n) < 0.001] = 0
        kt = k.dtype
        v = rng.integers(1, 1 << 31, n).astype(kt)
        before = len(m)
        st = t.insert(to_dev(k), to_dev(v))
        m.insert(k.astype(np.uint64), v.astype(np.uint64))
        distinct = np.unique(k[k != 0]).size
        assert st["inserted"] == len(m) - before and st["updated"] == distinct - st["inserted"]
        assert st["superseded"] == int((k != 0).sum()) - distinct and st["rejected"] == int((k == 0).sum())
        assert_same_contents(t, m, "insert %d" % step)
        k, v = draw(), rng.integers(1, 1 << 31, n).astype(kt)
        ops = rng.choice(np.array([0, 1, 2, 9], np.uint8), size=n, p=[0.4, 0.3, 0.2, 0.1])
        out, bits = t.apply(to_dev(ops), to_dev(k), to_dev(v))
        ov, oh = m.apply(ops, k.astype(np.uint64), v.astype(np.uint64))
        assert np.array_equal(dg.unpack_bits(bits, n), oh), step
        assert np.array_equal(out.cpu().numpy().view(kt).astype(np.uint64), ov), step
        assert_same_contents(t, m, "apply %d" % step)
        e = draw()
        eb = torch.full(((n + 31) // 32,), -1, dtype=torch.int32, device="cuda")
        got = t.erase(to_dev(e), erased_bits=eb)
        _, eh = m.erase(e.astype(np.uint64))
        assert got == int(eh.sum()) and np.array_equal(dg.unpack_bits(eb, n), eh)
        assert_same_contents(t, m, "erase %d" % step)
    t.close()


def _us(f, reps=9):
    import time

    import torch
    best = 1e9
    for _ in range(reps):
        torch.cuda.synchronize()
        a = time.perf_counter()
        f()
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - a)
    return best * 1e6


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("n", [8192, 32768, 100000, 1 << 20])
@pytest.mark.parametrize("hot", [1, 7, 100])
def test_hot_inserts_take_no_more_than_twice_the_time_of_distinct_ones(kb, n, hot):
    """The split and the grouping read as many ops either way and the probes are
    fewer, so one block must not be left with most of the batch."""
    import databases_gpu_gb300 as dg
    pool = _pool(kb, n, 5)
    t = dg.DyCuckoo(4 * n, key_bytes=kb, value_bytes=kb, auto_resize=False)
    v = to_dev(pool)
    d, h = to_dev(pool), to_dev(pool[np.random.default_rng(1).integers(0, hot, n)])
    plain = _us(lambda: t.insert(d, v))
    assert _us(lambda: t.insert(h, v)) < 2.0 * plain
    t.close()


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("bucket_bytes", [32, 64, 128])
def test_mixed_batches_of_long_segments(kb, bucket_bytes):
    """Keys with 256 to 20000 ops each (replayed by a block beyond 256, sorted
    in pieces beyond 4096), among keys with few, through a table and a set."""
    import databases_gpu_gb300 as dg
    rng = np.random.default_rng(kb + bucket_bytes)
    counts = [255, 256, 257, 511, 512, 513, 2000, 4095, 4096, 4097, 8193, 20000] + [1, 2, 9] * 50
    pool = _pool(kb, len(counts), 3)
    k = np.repeat(pool, counts)
    n = k.size
    kt = k.dtype
    t = dg.DyCuckoo(4096, key_bytes=kb, value_bytes=kb, bucket_bytes=bucket_bytes)
    S = dg.DyCuckooSet([2048, 2048], key_bytes=kb, bucket_bytes=bucket_bytes)
    m, ms = O.Map(), [O.Map(), O.Map()]
    off = np.array([0, n // 3, n], np.uint32)
    for step in range(3):
        k = k[rng.permutation(n)]
        v = rng.integers(1, 1 << 31, n).astype(kt)
        ops = rng.choice(np.array([0, 1, 2, 7], np.uint8), size=n, p=[0.5, 0.2, 0.2, 0.1])
        if step == 1:  # long runs without a mutation
            ops[rng.random(n) < 0.995] = 0
        out, bits = t.apply(to_dev(ops), to_dev(k), to_dev(v))
        ov, oh = m.apply(ops, k.astype(np.uint64), v.astype(np.uint64))
        assert np.array_equal(dg.unpack_bits(bits, n), oh), step
        assert np.array_equal(out.cpu().numpy().view(kt).astype(np.uint64), ov), step
        assert_same_contents(t, m, "step %d" % step)
        out, bits = S.apply(to_dev(off), to_dev(ops), to_dev(k), to_dev(v), h_offsets=off)
        hit, val = dg.unpack_bits(bits, n), out.cpu().numpy().view(kt).astype(np.uint64)
        for i in range(2):
            a, b = int(off[i]), int(off[i + 1])
            ov, oh = ms[i].apply(ops[a:b], k[a:b].astype(np.uint64), v[a:b].astype(np.uint64))
            assert np.array_equal(hit[a:b], oh) and np.array_equal(val[a:b], ov), (step, i)
            assert_same_contents(S.table(i), ms[i], "step %d table %d" % (step, i))
    t.close()
    S.close()


@pytest.mark.parametrize("kb", [4, 8])
def test_mixed_batch_of_long_segments_takes_no_more_than_three_times_distinct_keys(kb):
    """2^22 ops on 5000 keys: each op's index is sorted and its code and value
    read in three or four more passes than a distinct key's op; a block must not
    replay its segment with one warp."""
    import databases_gpu_gb300 as dg
    n = 1 << 22
    rng = np.random.default_rng(4)
    pool = _pool(kb, n, 6)
    t = dg.DyCuckoo(4 * n, key_bytes=kb, value_bytes=kb, auto_resize=False)
    ops, v = to_dev(rng.integers(0, 3, n).astype(np.uint8)), to_dev(pool)
    d, h = to_dev(pool), to_dev(pool[rng.integers(0, 5000, n)])
    plain = _us(lambda: t.apply(ops, d, v))
    assert _us(lambda: t.apply(ops, h, v)) < 3.0 * plain
    t.close()
