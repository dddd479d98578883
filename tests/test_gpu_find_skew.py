"""Large finds of 8-byte keys choose whether buckets go through the L1 by the
keys that repeat in a sample: batches of one key, of few, of skewed and of distinct keys, at the
batch size where the choice begins and above it. Whole numbers: all equal."""
import numpy as np
import pytest

from tests.helpers import to_dev, to_host, unique_u32, unique_u64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb,bucket", [(4, 128), (8, 128), (4, 64), (8, 64), (4, 32)])
@pytest.mark.parametrize("n", [(1 << 21) + 5, (1 << 23) - 31])
def test_skewed_finds_match(kb, bucket, n):
    import databases_gpu_gb300 as dg
    rng = np.random.default_rng(n + kb)
    pool = (unique_u32 if kb == 4 else unique_u64)(1 << 18, seed=kb)
    half = pool.size // 2
    present = np.arange(pool.size) < half
    value = rng.integers(1, 1 << 31, pool.size).astype(pool.dtype)
    t = dg.DyCuckoo(half * 2, key_bytes=kb, value_bytes=kb, bucket_bytes=bucket)
    t.insert(to_dev(pool[:half]), to_dev(value[:half]))
    for step in range(2):  # the second pass after a change of every value
        if step:
            value = value ^ np.array(0x5A5A5A, pool.dtype)
            t.insert(to_dev(pool[:half]), to_dev(value[:half]))
        for j in (np.zeros(n, np.int64), rng.integers(0, 3, n) * (half - 1),
                  np.minimum(rng.zipf(1.2, n), pool.size) - 1,
                  np.arange(n) % pool.size):
            k = pool[j]
            k[::1013] = 0
            hit = present[j] & (k != 0)
            out, bits = t.find(to_dev(k))
            assert np.array_equal(dg.unpack_bits(bits, n), hit)
            assert np.array_equal(to_host(out, kb), np.where(hit, value[j], 0))
    t.close()
