"""The kernels with the reference's launch geometry at the sizes where a turn of their walk ends: lengths around
one position, one turn of a warp and one turn of a block, for every head width, with caches on and off 16-byte
boundaries (the two forms of the loads).

Bound of the fp16 outputs: half an ulp of the value (2^-11 of it, 2^-25 below fp16's normal range) plus 1e-5 for
the fp32 sums (values of N(0, 1) rows averaged over at most 700 positions, |out| <= 4; observed below 2e-6)."""
import ctypes

import numpy as np
import pytest

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 513, 700]


NAMED = ("flash_attention_kernel", "flash_attention_split_kv_partial_kernel")
SHORT = ("vteb_flash_attention_many_kernel", "vteb_split_kv_partial_compat_short_kernel")


@pytest.mark.parametrize("skew", [0, 4], ids=["aligned", "8-byte"])
@pytest.mark.parametrize("builds, heads", [(NAMED, h) for h in ((12, 2, 128), (6, 2, 64), (16, 1, 128), (4, 2, 256))] +
                         [(NAMED, h) for h in ((30, 2, 64), (8, 2, 256))] +          # grids of the build between few and many
                         [(SHORT, h) for h in ((12, 2, 128), (6, 2, 64), (4, 2, 256))],
                         ids=lambda x: str(x) if isinstance(x[0], int) else "named" if x is NAMED else "short")
def test_unsplit_and_split_walks_at_turn_boundaries(cuda_runtime, codegen, builds, heads, skew):
    rt = cuda_runtime
    Hq, Hkv, D = heads
    B, S, C = len(LENGTHS), 700, 3
    rng = np.random.default_rng([Hq, D])
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    q, k, v, kn, vn = f16(B, Hq, D), f16(B, S, Hkv, D), f16(B, S, Hkv, D), f16(B, Hkv, D), f16(B, Hkv, D)
    off = np.array(LENGTHS, dtype=np.int32) - 1
    k_ref, v_ref = k.copy(), v.copy()
    orc.kv_cache_append(kn, vn, k_ref, v_ref, off)
    ref = orc.decode_attention(q, k_ref, v_ref, off)
    arch, bufs = rt.get_gpu_architecture(), []

    def dev(arr, pad=0):
        p = rt.safe_malloc(arr.nbytes + 2 * pad, "walk test output")
        bufs.append(p)
        at = ctypes.c_void_p(p.value + 2 * pad)
        rt.safe_memcpy_host_to_device(at, np.ascontiguousarray(arr), "walk test output")
        return at

    def host(arr, at):
        rt.safe_memcpy_device_to_host(arr, at, "walk test output")
        return arr
    try:
        dq, dkn, dvn, doff = dev(q), dev(kn), dev(vn), dev(off)
        dk, dv = dev(k, skew), dev(v, skew)
        dout = dev(np.zeros((B, Hq, D), np.float16))
        vp, ci, cf = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
        stride, scale = S * Hkv * D, 1.0 / np.sqrt(D)
        _, unsplit = codegen.load_kernel_safe(rt, 'flash_attention', arch, builds[0])
        rt.launch_kernel(unsplit, (B, Hq, 1), (D, 1, 1),
                         [dq, dkn, dvn, dk, dv, dout, ci(1), ci(Hq), ci(Hkv), ci(D), cf(scale), doff, ci(stride)], 2 * D * 4)
        rt.synchronize()
        out = host(np.zeros((B, Hq, D), np.float16), dout).astype(np.float32)
        assert np.all(np.abs(out - ref) <= np.abs(ref) * 2.0 ** -11 + 2.0 ** -25 + 1e-5)
        assert np.array_equal(host(np.zeros_like(k), dk), k_ref) and np.array_equal(host(np.zeros_like(v), dv), v_ref)
        # the same caches, now with the new rows in them, cut into three splits
        dm, dl = dev(np.zeros((B, Hq, C), np.float32)), dev(np.zeros((B, Hq, C), np.float32))
        do = dev(np.zeros((B, Hq, C, D), np.float32))
        _, partial = codegen.load_kernel_safe(rt, 'flash_attention_split_kv_partial', arch, builds[1])
        rt.launch_kernel(partial, (B, Hq, C), (D, 1, 1),
                         [dq, dk, dv, dm, dl, do, ci(Hq), ci(Hkv), ci(D), cf(scale), doff, ci(stride), ci(C)], 2 * D * 4)
        rt.synchronize()
        pm, pl = host(np.zeros((B, Hq, C), np.float32), dm), host(np.zeros((B, Hq, C), np.float32), dl)
        po = host(np.zeros((B, Hq, C, D), np.float32), do)
        rm, rl, _ = orc.split_kv_partial(q, k_ref, v_ref, off, scale, C)
        live = rm > -1e29
        assert np.array_equal(pm[~live], rm[~live]) and np.all(pl[~live] == 0) and np.all(po[~live] == 0)
        assert np.allclose(pm[live], rm[live], atol=1e-5, rtol=1e-5) and np.allclose(pl[live], rl[live], rtol=1e-4)
        assert np.max(np.abs(orc.split_kv_reduce(pm, pl, po) - ref)) <= 1e-5
    finally:
        for p in bufs:
            rt.safe_free(p, "walk test cleanup")


@pytest.mark.parametrize("D", [64, 128, 256])
def test_an_infinite_value_in_the_newest_row_stays_infinite(cuda_runtime, codegen, D):
    """The newest row's weight is positive, so an infinite value in it gives an infinite output in that channel and
    leaves the others finite, also where the rows past the end fill up a turn."""
    rt = cuda_runtime
    Hq, Hkv, S, lengths = 2, 1, 160, [1, 5, 33, 129]
    B = len(lengths)
    rng = np.random.default_rng(D)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    q, k, v, kn, vn = f16(B, Hq, D), f16(B, S, Hkv, D), f16(B, S, Hkv, D), f16(B, Hkv, D), f16(B, Hkv, D)
    vn[:, :, 3] = np.inf
    off, bufs = np.array(lengths, dtype=np.int32) - 1, []

    def dev(arr):
        bufs.append(rt.safe_malloc(arr.nbytes, "infinite row test output"))
        rt.safe_memcpy_host_to_device(bufs[-1], np.ascontiguousarray(arr), "infinite row test output")
        return bufs[-1]
    try:
        dq, dk, dv, dkn, dvn, doff, dout = (dev(x) for x in (q, k, v, kn, vn, off, np.zeros((B, Hq, D), np.float16)))
        ci, cf = ctypes.c_int, ctypes.c_float
        _, unsplit = codegen.load_kernel_safe(rt, 'flash_attention', rt.get_gpu_architecture(), 'flash_attention_kernel')
        rt.launch_kernel(unsplit, (B, Hq, 1), (D, 1, 1), [dq, dkn, dvn, dk, dv, dout, ci(1), ci(Hq), ci(Hkv), ci(D),
                                                          cf(1.0 / np.sqrt(D)), doff, ci(S * Hkv * D)], 2 * D * 4)
        rt.synchronize()
        out = np.zeros((B, Hq, D), np.float16)
        rt.safe_memcpy_device_to_host(out, dout, "infinite row test output")
        assert np.all(out[:, :, 3] == np.inf) and np.all(np.isfinite(np.delete(out, 3, axis=2)))
    finally:
        for p in bufs:
            rt.safe_free(p, "infinite row test cleanup")
