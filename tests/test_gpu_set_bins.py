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
