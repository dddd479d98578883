"""Table-set batches by bins (dyc_bins.cuh) where the set's scratch is new, small
for its tables or much larger than the batch. Whole numbers, each table against
its own oracle map: everything is equal."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import assert_same_contents, to_dev, to_host

pytestmark = pytest.mark.gpu


def _check(S, maps, off, ops, k, v, out, bits, label):
    import databases_gpu_gb300 as dg
    gv = to_host(out, S.value_bytes).astype(np.uint64)
    gh = dg.unpack_bits(bits, k.size)
    for t in range(S.ntables):
        a, b = int(off[t]), int(off[t + 1])
        if a == b:
            continue
        ov, oh = maps[t].apply(ops[a:b], k[a:b].astype(np.uint64), v[a:b].astype(np.uint64))
        assert np.array_equal(gh[a:b], oh), "%s: table %d hit bits" % (label, t)
        assert np.array_equal(gv[a:b], ov), "%s: table %d values" % (label, t)
    sizes, _ = S.sizes()
    assert np.array_equal(sizes, np.array([len(m) for m in maps])), label


@pytest.mark.parametrize("kb", [4, 8])
def test_first_set_call_on_a_side_stream_beside_a_busy_default_stream(kb):
    """The bins' counts are cleared in the order of the batch's own stream: the
    default stream is still at work when the set's first batch runs on another."""
    import torch
    import databases_gpu_gb300 as dg
    rng = np.random.default_rng(kb)
    kt = np.uint32 if kb == 4 else np.uint64
    S = dg.DyCuckooSet([4000] * 8, key_bytes=kb)
    maps = [O.Map() for _ in range(8)]
    off = np.arange(9, dtype=np.uint32) * 3000
    n = int(off[-1])
    side = torch.cuda.Stream()
    work = torch.zeros(1 << 29, dtype=torch.uint8, device="cuda")
    old = torch.full((1 << 26,), -1, dtype=torch.int32, device="cuda")  # memory the scratch may get
    del old
    torch.cuda.empty_cache()
    for r in range(2):
        ops = rng.choice(np.array([0, 1, 2], np.uint8), size=n)
        k = rng.integers(1, 2000, n).astype(kt)
        v = rng.integers(1, 1 << 31, n).astype(kt)
        args = [to_dev(a) for a in (off, ops, k, v)]
        torch.cuda.synchronize()
        for _ in range(200):
            work.add_(1)  # about 30 ms
        with torch.cuda.stream(side):
            out, bits = S.apply(*args, h_offsets=off)
        _check(S, maps, off, ops, k, v, out, bits, "round %d" % r)
    torch.cuda.synchronize()
    S.close()


@pytest.mark.parametrize("kb", [4, 8])
def test_device_offsets_out_of_order_beside_a_hot_key(kb):
    """Device offsets [0, 4096, 5000, 0, 9000]: the ops from 5000 on fall to
    table 3, whose bins start below those of table 1, and repeat one key, so
    the bin of that key goes over its capacity. The tile of ops 4096 to 8191
    looks for such bins among the ones from table 1's on. The call reports the
    offsets, and the records it did not write are not read."""
    import torch
    import databases_gpu_gb300 as dg
    from databases_gpu_gb300._lib import DYC_EINVAL
    kt = np.uint32 if kb == 4 else np.uint64
    n = 9000
    host = np.array([0, 4096, 5000, 5000, n], np.uint32)
    bad = np.array([0, 4096, 5000, 0, n], np.uint32)
    S = dg.DyCuckooSet([20000] * 4, key_bytes=kb)
    rng = np.random.default_rng(kb)
    for r in range(12):  # several keys: the fault needs one in table 3's first bins
        k = rng.integers(1, 1 << 31, n).astype(kt)
        k[5000:] = k[0]
        args = [to_dev(a) for a in (bad, np.ones(n, np.uint8), k, k)]
        with pytest.raises(dg.DycError) as ei:
            S.apply(*args, h_offsets=host)
        assert ei.value.status == DYC_EINVAL, ei.value
    torch.cuda.synchronize()
    # the set still serves batches with good offsets
    S.close()
    S = dg.DyCuckooSet([20000] * 4, key_bytes=kb)
    maps = [O.Map() for _ in range(4)]
    ops = rng.integers(0, 3, n).astype(np.uint8)
    out, bits = S.apply(to_dev(host), to_dev(ops), to_dev(k), to_dev(k), h_offsets=host)
    _check(S, maps, host, ops, k, k, out, bits, "good offsets")
    S.close()


def _two_sets(sizes, kb, **kw):
    import databases_gpu_gb300 as dg
    return dg.DyCuckooSet(sizes, key_bytes=kb, **kw), dg.DyCuckooSet(sizes, key_bytes=kb, **kw)


def _against_each(A, B, counts, draw, rounds, graph=False):
    """Rounds of counts[t] ops per table through the batched path and, table by
    table, through dyc_apply: equal results, sizes, capacities and contents."""
    import torch
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)
    n = int(off[-1])
    table = np.repeat(np.arange(len(counts)), counts)
    rng = np.random.default_rng(n)
    bufs = None
    for r in range(rounds):
        k = draw(rng, n, table).astype(np.uint32 if A.key_bytes == 4 else np.uint64)
        v = rng.integers(1, 1 << 31, n).astype(k.dtype)
        ops = rng.choice(np.array([0, 1, 2], np.uint8), size=n, p=[0.2, 0.6, 0.2])
        args = [to_dev(a) for a in (off, ops, k, v)]
        if bufs is None:
            bufs = args + [torch.empty_like(args[3]), torch.empty((n + 31) // 32, dtype=torch.int32, device="cuda")]
        else:
            for b, a in zip(bufs, args):
                b.copy_(a)
        oa, ba = A.apply(*bufs[:4], out=bufs[4], bits=bufs[5], h_offsets=off, graph=graph)
        ob, bb = B.apply(*args, h_offsets=off, each=True)
        assert bool((oa == ob).all()), "round %d: values" % r
        assert bool((ba == bb).all()), "round %d: bits" % r
        (sa, ca), (sb, cb) = A.sizes(), B.sizes()
        assert np.array_equal(sa, sb) and np.array_equal(ca, cb), "round %d: sizes" % r
    for t in range(0, len(counts), max(1, len(counts) // 50)):
        for x, y in zip(A.table(t).export(), B.table(t).export()):
            assert bool((torch.sort(x).values == torch.sort(y).values).all()), t


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("graph", [False, True])
def test_tables_with_few_ops_share_bins(kb, graph):
    """3000 tables, half without ops, the same few keys in all of them, and some
    tables of 700 to 5000 ops on few keys and on many: bins of many tables, of
    two, and of one; growing tables, so the counts of the upsize policy matter."""
    rng = np.random.default_rng(kb)
    counts = rng.integers(0, 6, 3000) * rng.integers(0, 2, 3000)
    counts[[7, 500, 501, 1400, 2999]] = [700, 5000, 896, 2500, 1793]
    A, B = _two_sets([16] * 3000, kb)

    def draw(rng, n, table):
        few = rng.integers(1, 4, n)
        many = rng.integers(1, 1 << 31, n)
        return np.where(np.isin(table, [500, 2999]), many, few)

    _against_each(A, B, counts, draw, 3, graph)
    A.close()
    B.close()


@pytest.mark.parametrize("kb", [4, 8])
def test_overfull_bins_of_several_tables(kb):
    """A key that repeats 3000 times in one table whose bin it shares with the
    ops of 40 others, some with the same key; and more than 1024 (table, key)
    pairs in overfull bins."""
    counts = [3] * 20 + [3000] + [5] * 20 + [6000] + [1] * 800 + [4000]
    A, B = _two_sets([64] * len(counts), kb)

    def draw(rng, n, table):
        k = np.where(rng.random(n) < 0.2, rng.integers(1, 1 << 31, n), 77)
        return np.where((table == 41) & (rng.random(n) < 0.5), rng.integers(1, 2000, n), k)

    _against_each(A, B, counts, draw, 3)
    A.close()
    B.close()


@pytest.mark.parametrize("kb", [4, 8])
def test_a_table_with_more_bins_than_a_block_counts(kb):
    """One table gets 4.2 million ops, more than 4096 bins' worth: a tile's ops
    beyond those take their places one by one. Some keys are popular."""
    counts = [10, 4200000, 0, 3000]
    A, B = _two_sets([64, 1 << 22, 64, 64], kb)

    def draw(rng, n, table):
        return np.where(rng.random(n) < 0.1, rng.integers(1, 20, n), rng.integers(1, 1 << 31, n))

    _against_each(A, B, counts, draw, 2)
    A.close()
    B.close()


def test_scratch_follows_the_batch_and_not_the_table_count():
    """1000 ops over 20000 tables: under 64 MB for the first batch (a batch takes
    some 200 bytes an op and 20 a table; a bin for every table took 330 MB)."""
    import torch
    import databases_gpu_gb300 as dg
    nt, n = 20000, 1000
    S = dg.DyCuckooSet([8] * nt, auto_resize=False)
    off = np.searchsorted(np.sort(np.random.default_rng(1).integers(0, nt, n)), np.arange(nt + 1)).astype(np.uint32)
    off[-1] = n
    args = [to_dev(a) for a in (off, np.ones(n, np.uint8), np.arange(1, n + 1, dtype=np.uint32),
                                np.arange(1, n + 1, dtype=np.uint32))]
    out, bits = torch.empty_like(args[3]), torch.empty(40, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    S.apply(*args, out=out, bits=bits, h_offsets=off)
    free1, _ = torch.cuda.mem_get_info()
    assert free0 - free1 < 64 << 20
    sizes, _ = S.sizes()
    assert int(sizes.sum()) == n
    S.close()
