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
@pytest.mark.parametrize("n", [100000, 1 << 20])
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
