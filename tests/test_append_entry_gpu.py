"""`vteb_kv_cache_append` followed by a programmatic `vteb_split_kv_decode`: the split reads offsets and older rows
ahead of its dependency wait, so what stands in front of the append has to be complete by then."""
import ctypes

import numpy as np
import pytest

from oracle import attention_oracle as orc
from vte_b200.bridge.cuda_runtime import ATTN_BALANCED, ATTN_COMPACT, ATTN_PROGRAMMATIC

APPENDS = 3          # before every attention, so that a row written two launches earlier is an older row for the split
STEPS = 24


@pytest.mark.gpu
@pytest.mark.parametrize("offsets_by_launch", [True, False], ids=["offsets-by-launch", "offsets-final"])
@pytest.mark.parametrize("heads, start, splits, flags, n_ctas", [
    ((12, 2, 128), [40], 2, ATTN_COMPACT, 0),                    # crosses the ends of tiles of 32 and of splits
    ((8, 2, 256), [7], 3, ATTN_COMPACT, 0),
    ((32, 8, 64), [1, 60, 17, 200, 31], 32, ATTN_BALANCED, 0),   # goes to clusters
    ((32, 8, 64), [1, 60, 17, 200, 31], 32, ATTN_BALANCED, 148), # equal shares
    ((28, 4, 128), [1, 60, 17, 200, 31], 32, 0, 0),              # work queue, full shape
], ids=["compact-128", "compact-256", "clusters-64", "balanced-64", "queue-128"])
def test_appends_then_programmatic_attention(cuda_runtime, codegen, heads, start, splits, flags, n_ctas, offsets_by_launch):
    """Every step appends three positions and attends, with nothing but launches between the steps.  Either a launch
    right in front of each append writes the offsets, or every append has offsets of its own.  Bound: fp32 sums of at
    most 272 probabilities of 22 bits with values N(0, 1), as in the tests of the same kernels."""
    rt = cuda_runtime
    Hq, Hkv, D = heads
    B, S = len(start), 288
    rng = np.random.default_rng([Hq, D, B])
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    k, v = f16(B, S, Hkv, D), f16(B, S, Hkv, D)
    q, knew, vnew = f16(STEPS, B, Hq, D), f16(STEPS * APPENDS, B, Hkv, D), f16(STEPS * APPENDS, B, Hkv, D)
    pad = -(-B // 4) * 4                                         # offsets in whole 16-byte words
    offs = np.zeros((STEPS * APPENDS, pad), dtype=np.int32)
    for i in range(STEPS * APPENDS):
        offs[i, :B] = np.array(start, dtype=np.int32) + i
    bufs = []

    def dev(arr=None, nbytes=0):
        p = rt.safe_malloc(arr.nbytes if arr is not None else nbytes, "append test output")
        bufs.append(p)
        if arr is not None:
            rt.safe_memcpy_host_to_device(p, arr, "append test output")
        else:
            rt.safe_memset(p, nbytes, "append test output")
        return p.value

    copy = codegen.load_kernel_safe(rt, "decode_attention", rt.get_gpu_architecture(), "vteb_stage_copy_kernel")[1]
    vp, ci = ctypes.c_void_p, ctypes.c_int
    try:
        dk, dv, dq, dkn, dvn, doffs = (dev(x) for x in (k, v, q, knew, vnew, offs))
        cur = dev(nbytes=pad * 4)
        out = dev(nbytes=STEPS * B * Hq * D * 4)
        pm, pl, po = dev(nbytes=B * Hq * splits * 4), dev(nbytes=B * Hq * splits * 4), dev(nbytes=B * Hq * splits * D * 4)
        work = dev(nbytes=16)
        row = B * Hkv * D * 2
        for step in range(STEPS):
            for a in range(step * APPENDS, (step + 1) * APPENDS):
                off = doffs + a * pad * 4
                if offsets_by_launch:
                    rt.launch_kernel(copy, (1, 1, 1), (32, 1, 1), [vp(off), vp(cur), ci(pad // 4)])
                    off = cur
                rt.kv_cache_append(dkn + a * row, dvn + a * row, dk, dv, off, B, Hkv, D, S * Hkv * D)
            rt.split_kv_decode(dq + step * B * Hq * D * 2, dk, dv, off, out + step * B * Hq * D * 4, True, pm, pl, po, work,
                               B, Hq, Hkv, D, D ** -0.5, S * Hkv * D, splits, 0, flags | ATTN_PROGRAMMATIC, n_ctas)
        rt.check_status(work)
        got = np.zeros((STEPS, B, Hq, D), dtype=np.float32)
        rt.safe_memcpy_device_to_host(got, ctypes.c_void_p(out), "append test output")
        kr, vr = np.zeros_like(k), np.zeros_like(v)
        rt.safe_memcpy_device_to_host(kr, ctypes.c_void_p(dk), "append test output")
        rt.safe_memcpy_device_to_host(vr, ctypes.c_void_p(dv), "append test output")
    finally:
        for p in bufs:
            rt.safe_free(p, "append test cleanup")
    for step in range(STEPS):
        for a in range(step * APPENDS, (step + 1) * APPENDS):
            orc.kv_cache_append(knew[a], vnew[a], k, v, offs[a, :B])
        ref = orc.decode_attention(q[step], k, v, offs[(step + 1) * APPENDS - 1, :B])
        assert np.max(np.abs(got[step] - ref)) <= 1e-5, step
    assert np.array_equal(kr, k) and np.array_equal(vr, v)
