"""The host-array calls on memory that the program registered itself
(cudaHostRegister), which is used in place as allocated pinned memory is."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import unique_u32, unique_u64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("n", [33, 100001])
def test_registered_arrays_match_oracle(kb, n):
    import torch
    import databases_gpu_gb300 as dg
    rt = torch.cuda.cudart()
    kt = np.uint32 if kb == 4 else np.uint64
    rng = np.random.default_rng(n + kb)
    page = 4096
    raw = np.zeros(8 * n * 8 + 64 * page, np.uint8)
    base = -raw.ctypes.data % page
    arrays = [raw[base + i * (2 * n * 8 // page + 8) * page:][: n * kb].view(kt) for i in range(3)]
    bits = raw[base + 3 * (2 * n * 8 // page + 8) * page:][: (n + 31) // 32 * 4].view(np.uint32)
    regs = []
    for a in arrays + [bits]:
        assert int(rt.cudaHostRegister(a.ctypes.data, a.nbytes, 0)) == 0
        regs.append(a.ctypes.data)
    try:
        pool = (unique_u32 if kb == 4 else unique_u64)(2 * n, seed=n).astype(kt)
        t = dg.DyCuckoo(4 * n + 1024, key_bytes=kb, value_bytes=kb)
        m = O.Map()
        k, v, out = arrays
        k[:] = pool[rng.integers(0, n, n)]
        v[:] = rng.integers(1, 1 << 31, n)
        t.insert_host(k, v)
        m.insert(k.astype(np.uint64), v.astype(np.uint64))
        k[:] = pool[rng.integers(0, 2 * n, n)]
        t.find_host(k, out, bits)
        ov, oh = m.find(k.astype(np.uint64))
        assert np.array_equal(out.astype(np.uint64), ov)
        assert np.array_equal(np.unpackbits(bits.view(np.uint8), bitorder="little")[:n], oh)
        cnt = t.erase_host(k, bits)
        _, eh = m.erase(k.astype(np.uint64))
        assert cnt == int(eh.sum())
        assert np.array_equal(np.unpackbits(bits.view(np.uint8), bitorder="little")[:n], eh)
        t.close()
    finally:
        for p in regs:
            rt.cudaHostUnregister(p)
