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
