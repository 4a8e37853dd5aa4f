"""More than eight query heads per KV head: the split kernel's `wide` build, where a group is cut into equal runs
of at most eight heads that read the same staged rows."""
import ctypes

import numpy as np
import pytest

from oracle import attention_oracle as orc
from vte_b200.bridge.cuda_runtime import FastPlan, load_library
from vte_b200.core.split_kv_attention import WIDE_SCRATCH_BYTES, choose_split_count

# (heads, consumer heads per KV head): groups of 9 to 64, every head width, one and several KV heads per item
WIDE = [((32, 2, 128), 2), ((48, 1, 128), 6), ((36, 4, 64), 3), ((20, 2, 64), 2), ((64, 1, 64), 8), ((64, 1, 256), 8),
        ((24, 2, 256), 2)]
LENGTHS = [1, 2, 15, 16, 17, 31, 33, 64, 65, 127, 129, 500, 900]


def test_plan_covers_groups_with_an_equal_cut(built_library):
    lib = load_library(str(built_library))
    plan = FastPlan()
    for (hq, hkv, d), nv in WIDE:
        assert lib.vteb_split_kv_plan_wide(hq, hkv, d, ctypes.byref(plan)) == 0
        assert plan.ok == 1 and plan.hg * nv <= 8 and plan.hg * plan.n_hgroups == hkv
        assert plan.threads == 320 and plan.nstages >= 2 and plan.smem_bytes <= 227 * 1024 and plan.tile % 16 == 0
        # the same rows staged as for a group of eight, so the copies' boxes and alignment are the tested ones
        assert (plan.hg * d) % 64 == 0
    for hq, hkv, d in [(16, 2, 128), (22, 2, 128), (13, 1, 64), (72, 1, 128), (32, 2, 96), (33, 2, 128)]:
        assert lib.vteb_split_kv_plan_wide(hq, hkv, d, ctypes.byref(plan)) == 0 and plan.ok == 0


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [len(LENGTHS), 1], ids=["ragged", "one"])
@pytest.mark.parametrize("heads", [h for h, _ in WIDE], ids=str)
def test_wide_groups_match_the_oracle(cuda_runtime, codegen, heads, batch):
    """Equal shares over a ragged batch, the append among the launches; one sequence through the work queue, and
    unsplit where the context is short.  Bound: fp32 sums of at most 900 probabilities that carry 22 bits (and 2^-25
    of the reference at least), values N(0, 1): 900^0.5 * 2^-25 * 4.5 < 5e-6, twice that for the order of the sums."""
    from vte_b200.core.decode_executor import DecodeAttentionExecutor
    Hq, Hkv, D = heads
    rng = np.random.default_rng([Hq, D, batch])
    meta = {"attention.head_count": Hq, "attention.head_count_kv": Hkv, "attention.key_length": D}
    lengths = [LENGTHS] if batch > 1 else [[n] for n in (900, 17, 1)]
    S = 928
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    k, v = f16(batch, S, Hkv, D), f16(batch, S, Hkv, D)
    for capacity in ((S,) if batch > 1 else (S, 64)):
        ex = DecodeAttentionExecutor(cuda_runtime, codegen, meta, batch, capacity, 1, with_append=True, wide=True)
        try:
            assert ex.dispatcher.wide and ex.dispatcher.split_kernel_name == f"vteb_split_kv_partial_wide_d{D}_kernel"
            for lens in lengths:
                if max(lens) > capacity:
                    continue
                q, kn, vn = f16(batch, Hq, D), f16(batch, Hkv, D), f16(batch, Hkv, D)
                off = np.array(lens, dtype=np.int32) - 1
                kr, vr = k[:, :capacity].copy(), v[:, :capacity].copy()
                ex.upload_layer(0, q, kr, vr)
                ex.upload_new_kv(0, kn, vn)
                out = ex.execute_decode_batch(off)[0]
                orc.kv_cache_append(kn, vn, kr, vr, off)
                assert np.max(np.abs(out - orc.decode_attention(q, kr, vr, off))) <= 1e-5
        finally:
            ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("heads, batch, capacity, longest", [((64, 1, 256), 13, 4096, 700), ((48, 1, 128), 200, 64, 64)],
                         ids=["fewer splits for the scratch limit", "more unsplit items than SMs"])
def test_wide_batches_at_the_limits_match_the_oracle(cuda_runtime, codegen, heads, batch, capacity, longest):
    """The balanced partition with its splits cut to the scratch limit; the work queue with more items than CTAs.
    Bound as above."""
    from vte_b200.core.decode_executor import DecodeAttentionExecutor
    Hq, Hkv, D = heads
    rng = np.random.default_rng([Hq, batch])
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    q, k, v = f16(batch, Hq, D), f16(batch, capacity, Hkv, D), f16(batch, capacity, Hkv, D)
    off = rng.integers(0, longest, size=batch).astype(np.int32)
    off[0], off[-1] = longest - 1, 0
    ex = DecodeAttentionExecutor(cuda_runtime, codegen, {"attention.head_count": Hq, "attention.head_count_kv": Hkv,
                                                         "attention.key_length": D}, batch, capacity, 1, wide=True)
    try:
        d = ex.dispatcher
        if d.balanced:
            assert d.max_chunks * batch * Hq * (D + 2) * 4 <= WIDE_SCRATCH_BYTES < (d.max_chunks + 1) * batch * Hq * (D + 2) * 4
        else:
            assert d.max_chunks == 1 and batch > cuda_runtime.get_num_cus()
        ex.upload_layer(0, q, k, v)
        out = ex.execute_decode_batch(off)[0]
    finally:
        ex.cleanup()
    assert np.max(np.abs(out - orc.decode_attention(q, k, v, off))) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("heads", [(32, 2, 128), (36, 4, 64), (24, 2, 256)], ids=str)
def test_wide_keeps_weights_far_below_the_maximum(cuda_runtime, codegen, heads):
    """Every sixteenth position carries all of the weight and values of zero, the others lie 30 octaves under it and
    make up the whole output.  Bound, relative: a probability of 2^-30 is held to 2^-43, so within 2^-14, and scores of
    30 octaves in fp32 cost 2e-6; four times that."""
    from vte_b200.core.decode_executor import DecodeAttentionExecutor
    Hq, Hkv, D = heads
    rng = np.random.default_rng([Hq, D, 30])
    meta = {"attention.head_count": Hq, "attention.head_count_kv": Hkv, "attention.key_length": D}
    for capacity, lens in ((64, [61]), (928, [900, 100, 17])):
        B = len(lens)
        q = np.ones((B, Hq, D), np.float16)
        k = np.zeros((B, capacity, Hkv, D), np.float16)
        k[:, ::16] = np.float16(30 * np.log(2) / np.sqrt(D))
        v = (rng.random((B, capacity, Hkv, D), dtype=np.float32) + 0.5).astype(np.float16)
        v[:, ::16] = 0
        off = np.array(lens, dtype=np.int32) - 1
        ex = DecodeAttentionExecutor(cuda_runtime, codegen, meta, B, capacity, 1, wide=True)
        try:
            assert ex.dispatcher.wide
            ex.upload_layer(0, q, k, v)
            out = ex.execute_decode_batch(off)[0]
        finally:
            ex.cleanup()
        ref = orc.decode_attention(q, k, v, off, dtype=np.float64)
        assert np.max(np.abs(out / ref - 1)) <= 2.5e-4


@pytest.mark.gpu
@pytest.mark.parametrize("heads", [(32, 2, 128), (36, 4, 64), (64, 1, 64), (24, 2, 256)], ids=str)
def test_wide_keeps_infinite_values(cuda_runtime, codegen, heads):
    """Every weight is positive, so an infinite value gives an infinite output in its channel, whatever sign the low
    part of the weight has, and leaves the others finite; both signs give NaN.  The newest row also fills the masked
    rows of the last tile."""
    from vte_b200.core.decode_executor import DecodeAttentionExecutor
    Hq, Hkv, D = heads
    rng = np.random.default_rng([Hq, D, 7])
    meta = {"attention.head_count": Hq, "attention.head_count_kv": Hkv, "attention.key_length": D}
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    for capacity, lens in ((64, [1]), (64, [61]), (928, [900, 1, 17, 112])):
        B = len(lens)
        q, k, v = f16(B, Hq, D), f16(B, capacity, Hkv, D), f16(B, capacity, Hkv, D)
        for b, n in enumerate(lens):
            v[b, n - 1, :, 3] = np.inf                      # the newest row
            v[b, n // 2, :, D - 2] = -np.inf                # a row of its own
            v[b, : n : 5, :, 9] = np.inf                    # many rows of a channel
            v[b, 0, :, 40], v[b, n - 1, :, 40] = np.inf, (-np.inf if n > 1 else np.inf)
        off = np.array(lens, dtype=np.int32) - 1
        ex = DecodeAttentionExecutor(cuda_runtime, codegen, meta, B, capacity, 1, wide=True)
        try:
            assert ex.dispatcher.wide
            ex.upload_layer(0, q, k, v)
            out = ex.execute_decode_batch(off)[0]
        finally:
            ex.cleanup()
        several = np.array(lens) > 1
        assert np.all(out[:, :, 3] == np.inf) and np.all(out[:, :, 9] == np.inf) and np.all(out[:, :, D - 2] == -np.inf)
        assert np.all(np.isnan(out[several][:, :, 40])) and np.all(out[~several][:, :, 40] == np.inf)
        rest = np.delete(np.arange(D), [3, 9, 40, D - 2])
        v[~np.isfinite(v)] = 0
        ref = orc.decode_attention(q, k, v, off)
        assert np.max(np.abs(out[:, :, rest] - ref[:, :, rest])) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("f32", [True, False], ids=["fp32", "fp16"])
@pytest.mark.parametrize("heads", [(32, 2, 128), (36, 4, 64), (64, 1, 64), (24, 2, 256)], ids=str)
def test_wide_stores_to_an_output_of_any_alignment(cuda_runtime, codegen, heads, f32):
    """An output that starts one element behind an aligned address, unsplit and combined: the same bits as aligned."""
    from vte_b200.core.decode_executor import DecodeAttentionExecutor
    Hq, Hkv, D = heads
    rng = np.random.default_rng([Hq, D, 4])
    meta = {"attention.head_count": Hq, "attention.head_count_kv": Hkv, "attention.key_length": D}
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    for capacity, lens in ((64, [61, 3]), (928, [900, 17])):
        q, k, v = f16(2, Hq, D), f16(2, capacity, Hkv, D), f16(2, capacity, Hkv, D)
        off = np.array(lens, dtype=np.int32) - 1
        outs = []
        for skip in (0, 4 if f32 else 2):
            ex = DecodeAttentionExecutor(cuda_runtime, codegen, meta, 2, capacity, 1, output_f32=f32, wide=True)
            try:
                assert ex.dispatcher.wide
                ex.tensor_mapping["blk.0.attention.output"] += skip
                ex.upload_layer(0, q, k, v)
                ex.execute_decode_batch(off, read_output=False)
                cuda_runtime.synchronize()
                raw = np.zeros(ex.out_bytes, dtype=np.uint8)
                cuda_runtime.safe_memcpy_device_to_host(raw, ctypes.c_void_p(ex.out_all.ptr + skip), "attention output")
                outs.append(raw.view(np.float32 if f32 else np.float16).reshape(2, Hq, D))
            finally:
                ex.cleanup()
        assert np.array_equal(outs[0], outs[1])
        assert np.max(np.abs(outs[0] - orc.decode_attention(q, k, v, off))) <= (1e-5 if f32 else 2e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [1, 5])
def test_wide_reads_offsets_behind_the_launch_in_front(cuda_runtime, codegen, batch):
    """A dispatcher's launches under programmatic launch, three appends and an attention per step, with a launch in
    front of each append that writes the offsets: right for the reference-geometry kernels, so right for `wide`."""
    from vte_b200.core.split_kv_attention import SplitKVAttentionDispatcher
    from vte_b200.bridge.memory import SlabAllocator
    rt, (Hq, Hkv, D), S, steps = cuda_runtime, (32, 2, 128), 288, 16
    rng = np.random.default_rng(batch)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    k, v = f16(batch, S, Hkv, D), f16(batch, S, Hkv, D)
    q, kn, vn = f16(steps, batch, Hq, D), f16(3 * steps, batch, Hkv, D), f16(3 * steps, batch, Hkv, D)
    offs = np.zeros((3 * steps, 8), dtype=np.int32)
    offs[:, :batch] = np.arange(3 * steps)[:, None] + np.array([40, 1, 200, 61, 15][:batch])
    alloc = SlabAllocator(rt, rt.get_real_mem_info()[1], requested_pool_size=64 << 20)
    alloc.initialize()
    bufs = []

    def dev(arr):
        bufs.append(rt.safe_malloc(arr.nbytes, "wide order output"))
        rt.safe_memcpy_host_to_device(bufs[-1], arr, "wide order output")
        return bufs[-1].value
    try:
        d = SplitKVAttentionDispatcher(rt, codegen, {"attention.head_count": Hq, "attention.head_count_kv": Hkv,
                                                     "attention.key_length": D}, allocator=alloc, context_length=S,
                                       batch_size=batch, output_f32=True, wide=True)
        assert d.wide
        dk, dv, dq, dkn, dvn, doffs = (dev(x) for x in (k, v, q, kn, vn, offs))
        cur, dout = dev(np.zeros(8, np.int32)), dev(np.zeros((steps, batch, Hq, D), np.float32))
        copy = codegen.load_kernel_safe(rt, "decode_attention", rt.get_gpu_architecture(), "vteb_stage_copy_kernel")[1]
        vp, ci, row = ctypes.c_void_p, ctypes.c_int, batch * Hkv * D * 2
        d._get_kernels()
        rt.synchronize()
        for step in range(steps):
            for a in range(3 * step, 3 * step + 3):
                rt.launch_kernel(copy, (1, 1, 1), (32, 1, 1), [vp(doffs + a * 32), vp(cur), ci(2)])
                rt.programmatic_launch = True
                launches = d.build_launches(0, {
                    "blk.0.q_proj.output": dq + step * batch * Hq * D * 2, "blk.0.k_proj.output": dkn + a * row,
                    "blk.0.v_proj.output": dvn + a * row, "blk.0.kv_cache.k": dk, "blk.0.kv_cache.v": dv,
                    "blk.0.attention.output": dout + step * batch * Hq * D * 4,
                    "kv_batch_stride_elements": S * Hkv * D}, cur, batch=batch)
                for fn, args, grid, block, smem in launches[:1] if a % 3 < 2 else launches:
                    rt.launch_kernel_recorded(fn, args, grid, block, smem)
                rt.programmatic_launch = False
        rt.check_status(d.work_ptr)
        out = np.zeros((steps, batch, Hq, D), np.float32)
        rt.safe_memcpy_device_to_host(out, ctypes.c_void_p(dout), "wide order output")
    finally:
        rt.programmatic_launch = False
        for p in bufs:
            rt.safe_free(p, "wide order cleanup")
        alloc.cleanup()
    for step in range(steps):
        for a in range(3 * step, 3 * step + 3):
            orc.kv_cache_append(kn[a], vn[a], k, v, offs[a, :batch])
        ref = orc.decode_attention(q[step], k, v, offs[3 * step + 2, :batch])
        assert np.max(np.abs(out[step] - ref)) <= 1e-5, step


@pytest.mark.gpu
def test_wide_only_where_the_split_layout_is_open(cuda_runtime, codegen):
    from vte_b200.bridge import CudaSafetyError
    from vte_b200.core.split_kv_attention import SplitKVAttentionDispatcher
    meta = {"attention.head_count": 32, "attention.head_count_kv": 2, "attention.key_length": 128}
    make = lambda m=meta, **kw: SplitKVAttentionDispatcher(cuda_runtime, codegen, m, context_length=4096, **kw)
    assert make(batch_size=8).wide and make(batch_size=8).balanced and make().wide and not make().balanced
    for kw in ({"num_splits": 16}, {"fixed_chunk_size": 32}, {"compat": True}):
        d = make(batch_size=8, **kw)
        assert d.compat and not d.wide and not d.balanced
    assert not make(dict(meta, **{"attention.head_count": 22})).wide              # 11 heads have no equal cut
    for batch in (2, 13, 64, 1024):                                               # scratch stays within its limit
        d = make(dict(meta, **{"attention.head_count": 64, "attention.head_count_kv": 1, "attention.key_length": 256}), batch_size=batch)
        other = choose_split_count(cuda_runtime.get_num_cus(), batch, 1, 4096)
        assert d.max_chunks <= max(other, WIDE_SCRATCH_BYTES // (batch * 64 * 258 * 4))
        assert d.wide == d.balanced and (d.wide or d.max_chunks == other)
    for kw in ({"fuse_rope": True}, {"fuse_append": True}, {"emit_state": True}):
        with pytest.raises(CudaSafetyError):
            make(**kw)
