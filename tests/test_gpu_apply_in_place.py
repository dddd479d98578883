"""dyc_apply with its results written over the key array (equal widths) and
apart from it: the same results, all equal to the oracle's map. Sizes around the small-batch kernel's bins and its largest batch. A matmul
on another stream holds most SMs meanwhile, so that a batch's blocks do not run
side by side."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import assert_same_contents, to_dev, to_host, unique_u32, unique_u64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("where", ["keys", "apart"])
@pytest.mark.parametrize("n", [385, 4096, 32768, 40000])
def test_results_over_the_inputs(kb, where, n):
    import torch
    import databases_gpu_gb300 as dg
    rng = np.random.default_rng(n + kb)
    kt = np.uint32 if kb == 4 else np.uint64
    pool = (unique_u32 if kb == 4 else unique_u64)(2 * n, seed=n).astype(kt)
    t = dg.DyCuckoo(8 * n, key_bytes=kb, value_bytes=kb)
    m = O.Map()
    a = torch.randn(4096, 4096, device="cuda", dtype=torch.bfloat16)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for step in range(6):
        k = pool[rng.integers(0, 2 * n, n)]
        k[rng.random(n) < 0.01] = 0
        v = rng.integers(1, 1 << 31, n).astype(kt)
        ops = rng.integers(0, 3, n).astype(np.uint8)
        dk, dv, do = to_dev(k), to_dev(v), to_dev(ops)
        out = dk if where == "keys" else torch.empty_like(dv)
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            for _ in range(30):
                b = a @ a
        out, bits = t.apply(do, dk, dv, out=out)
        ov, oh = m.apply(ops, k.astype(np.uint64), v.astype(np.uint64))
        assert np.array_equal(dg.unpack_bits(bits, n), oh), step
        assert np.array_equal(to_host(out, kb).astype(np.uint64), ov), step
        assert_same_contents(t, m, "step %d" % step)
    torch.cuda.synchronize()
    t.close()
