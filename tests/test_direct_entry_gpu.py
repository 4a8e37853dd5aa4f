"""`vteb_split_kv_decode` for one sequence whose splits hold whole tiles: tensor-map copies over a cache whose rows the
stride gives, 16-byte copies where the stride is 0."""
import ctypes

import numpy as np
import pytest

from oracle import attention_oracle as orc
from vte_b200.bridge.cuda_runtime import ATTN_COMPACT, ATTN_NO_TENSOR_MAPS


@pytest.mark.gpu
@pytest.mark.parametrize("compact", [ATTN_COMPACT, 0], ids=["compact", "full"])
@pytest.mark.parametrize("heads", [(12, 2, 128), (8, 2, 256), (32, 8, 64)], ids=str)
def test_one_sequence_of_whole_tiles(cuda_runtime, heads, compact):
    """Lengths that end inside a tile, with a tile and with the cache.  The copies' kind does not change a bit.
    Bound: fp32 sums of at most 512 probabilities of 22 bits with values N(0, 1): 512^0.5 * 2^-22 * 4.5 / 2 < 1e-5."""
    rt = cuda_runtime
    Hq, Hkv, D = heads
    S, C = 512, 3
    rng = np.random.default_rng([Hq, D])
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    q, k, v = f16(1, Hq, D), f16(1, S, Hkv, D), f16(1, S, Hkv, D)
    bufs = []

    def dev(arr):
        bufs.append(rt.safe_malloc(arr.nbytes, "direct entry output"))
        rt.safe_memcpy_host_to_device(bufs[-1], arr, "direct entry output")
        return bufs[-1]

    try:
        dq, dk, dv, work = dev(q), dev(k), dev(v), dev(np.zeros(4, np.int32))
        dout = dev(np.zeros((1, Hq, D), np.float32))
        pm, pl, po = (dev(np.zeros((Hq, C, w), np.float32)) for w in (1, 1, D))
        for n in (1, 100, 192, 193, 500, 512):
            off = np.array([n - 1], dtype=np.int32)
            doff = dev(off)
            got = []
            for stride, flags in ((S * Hkv * D, 0), (0, 0), (S * Hkv * D, ATTN_NO_TENSOR_MAPS)):
                rt.split_kv_decode(dq, dk, dv, doff, dout, True, pm, pl, po, work, 1, Hq, Hkv, D, D ** -0.5, stride, C, 0,
                                   flags | compact)
                rt.check_status(work)
                out = np.zeros((1, Hq, D), dtype=np.float32)
                rt.safe_memcpy_device_to_host(out, dout, "direct entry output")
                got.append(out)
            assert np.max(np.abs(got[0] - orc.decode_attention(q, k, v, off))) <= 1e-5, n
            assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2]), n
    finally:
        for p in bufs:
            rt.safe_free(p, "direct entry cleanup")


@pytest.mark.gpu
def test_a_failed_call_does_not_fail_the_next(cuda_runtime):
    """A failure is reported by the call that had it; a launch that is checked by the last error reports its own only."""
    rt, p = cuda_runtime, ctypes.c_void_p()
    assert rt._lib.vteb_malloc(ctypes.byref(p), 1 << 50) != 0          # a petabyte: refused at once
    x = rt.safe_malloc(4096, "last error test output")
    try:
        rt.fill_normal_f16(x, 2048, 1)
        rt.stream_synchronize()
    finally:
        rt.safe_free(x, "last error test cleanup")
