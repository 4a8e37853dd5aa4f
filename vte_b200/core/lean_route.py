"""Launch lists of a captured decode step from the kernels with one work item per CTA (csrc/kernels/lean_decode.cuh).

`SplitKVAttentionDispatcher.build_launches` keeps the reference's append / partial / reduce layout, whose pieces a
caller may replace, reorder or read back.  A step that an executor captures as a whole owes nobody that layout, so the
executor may take a shorter one for it: one launch a layer (`cluster`), in which the parts of a (sequence, KV head) are a
thread-block cluster that merges its states through shared memory and which appends the step's K and V rows itself.
"""
from __future__ import annotations

import ctypes
import math

from ..bridge.cuda_runtime import ClusterGrid
from ..bridge.errors import CudaSafetyError

FLAG_PREFETCH_Q = 8
FLAG_WAIT_FIRST = 32
FLAG_ROWS_FINAL = 64


def cluster_kernel_name(group: int, head_dim: int) -> str:
    return f"vteb_decode_cluster_{'2_' if group > 8 else ''}d{head_dim}_kernel"


class LeanRoute:
    """`parts` CTAs per (sequence, KV head): one launch a layer (`cluster`), or split and combine."""

    def __init__(self, dispatcher, parts: int, append: bool, cluster: bool):
        d = self.d = dispatcher
        self.parts, self.append, self.cluster = int(parts), bool(append), bool(cluster)
        self.plan = d.hip.lean_plan(d.num_q_heads, d.num_kv_heads, d.head_dim, self.parts, d.context_length, self.cluster)
        if not self.plan.ok:
            raise CudaSafetyError(f"{self.parts} CTAs per (sequence, KV head) are not covered for this geometry")
        load = lambda symbol: d.codegen.load_kernel_safe(d.hip, 'decode_attention', d.hip.get_gpu_architecture(), symbol)[1]
        if self.cluster:
            self.function = load(cluster_kernel_name(d.num_q_heads // d.num_kv_heads, d.head_dim))
        else:
            self.function = load(f"vteb_split_kv_lean_d{d.head_dim}_kernel")
            self.combine = load('vteb_split_kv_combine_small_kernel' if self.parts <= 32 else
                                'vteb_split_kv_combine_f32_kernel' if d.output_f32 else 'vteb_split_kv_combine_f16_kernel')

    def launches(self, layer: int, tensor_mapping: dict, kv_offset_ptr: int, batch: int):
        d = self.d
        vp, ci, cf = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
        attention_scale = d.metadata.get('attention_scale')
        scale = float(attention_scale) if attention_scale else 1.0 / math.sqrt(d.head_dim)
        ptr = lambda name: d._resolve_ptr(tensor_mapping, name)
        q, out = ptr(f'blk.{layer}.q_proj.output'), ptr(f'blk.{layer}.attention.output')
        k_cache, v_cache = d._resolve_kv_cache_ptrs(layer, tensor_mapping)
        stride = int(tensor_mapping.get('kv_batch_stride_elements', 0))
        d._validate(batch, q, k_cache, v_cache, out, kv_offset_ptr, stride)
        k_new, v_new = (ptr(f'blk.{layer}.k_proj.output'), ptr(f'blk.{layer}.v_proj.output')) if self.append else (0, 0)
        flags = (0 if self.append else FLAG_ROWS_FINAL) | (FLAG_PREFETCH_Q if d.hip.programmatic_launch else 0)
        rope = [vp(0), vp(0), ci(-1), ci(0)]
        if d.fuse_rope:
            rope = [vp(ptr('rope_cos')), vp(ptr('rope_sin')), ci(d.rope_type), ci(d.rotary_dim)]
        Hq, Hkv, D, N = d.num_q_heads, d.num_kv_heads, d.head_dim, self.parts
        out_kind = 2 if d.output_f32 else 1
        next_k = next_v = 0
        partials = [vp(0), vp(0), vp(0)]
        if not self.cluster:
            partials = [vp(p.ptr) for p in d.partial_buffers]
            next_k, next_v = d._resolve_kv_cache_ptrs(layer + 1, tensor_mapping)
        args = [vp(q), vp(k_cache), vp(v_cache), *partials, ci(Hq), ci(Hkv), ci(D), cf(scale), vp(kv_offset_ptr), ci(stride),
                ci(N), vp(k_new), vp(v_new), vp(out), ci(out_kind), ci(flags), ci(self.plan.depth), vp(d.work_ptr + 4),
                vp(next_k if next_v else 0), vp(next_v if next_k else 0)] + rope
        dims = (batch * Hkv * N, 1, 1)
        split = (self.function, args, ClusterGrid(dims, N) if self.cluster else dims, (self.plan.threads, 1, 1), self.plan.smem_bytes)
        if self.cluster:
            return [split]
        rows, slices = batch * Hq, D // 32
        args = [*partials, vp(out), ci(Hq), ci(D), ci(N)]
        if N <= 32:
            return [split, (self.combine, args + [ci(out_kind), vp(d.work_ptr), ci(rows), ci(1)],
                            ((rows * slices + 7) // 8, 1, 1), (256, 1, 1), 0)]
        return [split, (self.combine, args + [ci(slices), vp(d.work_ptr)], (rows * slices, 1, 1), (256, 1, 1), min(N, 256) * 4)]


# Estimated microseconds a layer, by which a route is chosen.  Fitted to 1,536 steps of 12 head geometries, 1 to 64
# sequences of 130 to 80,000 positions (the shortest down to a twentieth of the longest) in caches with room for 1 to 2.5
# times the longest, every route timed on each: the choice is within 1.6 % of the best route on the whole, takes 0.63 times
# as long as the dispatcher's launches, and at most 1.17 times (more than 1.05 in 8 of them).
_PER_POSITION = {64: 0.0038, 128: 0.0065, 256: 0.0145}      # K and V of one KV head through one CTA, alone on its SM
_TWO_RUNS = 1.34                                            # nine to sixteen query heads per KV head
_LONGEST, _MEAN = 0.75, 0.5                                 # of a batch, as shares of the cache's capacity
_ONE = 0.92                                                 # the same for one sequence
CLUSTER_PARTS = (2, 3, 4, 5, 6, 8, 9, 12, 16)              # more than 8 only where the device has room for such clusters
LEAN_SPLIT_MAX_CONTEXT = 131072


def _dispatcher_us(batch: int, cache_bytes: float, append: bool) -> float:
    return (7.2 if batch == 1 else 12.7) + cache_bytes / 5.8e6 + (2.0 if append else 0.0)


def _cluster_us(parts: int, pairs: int, resident: int, positions: float, per_position: float, num_sms: int, cache_bytes: float) -> float:
    """`resident` clusters run at once, one wave after the other; CTAs that share an SM share its load rate.  The stream
    of all of them and the stream of one CTA overlap (a smooth maximum)."""
    waves = -(-pairs // resident)
    one = per_position * max(1.0, min(pairs, resident) * parts / num_sms) * positions / parts * waves * (0.9 if waves > 1 else 1.0)
    return 3.4 + 0.21 * math.log2(parts) + 3.5 * (waves - 1) + ((cache_bytes / 6.1e6) ** 3.4 + one ** 3.4) ** (1 / 3.4)


def _split_us(parts: int, positions: float, head_dim: int, cache_bytes: float) -> float:
    return 5.2 + 0.0125 * head_dim + max(cache_bytes / 12e6, 0.57 * _PER_POSITION[head_dim] * positions / parts)


def choose_lean_route(d, append: bool) -> tuple:
    """(CTAs per (sequence, KV head), whether they are a cluster) for a dispatcher's geometry; (0, False): its own launches.

    Clusters win wherever latency counts: a layer is one dependent launch of 3.3 us instead of two or three (7.1).  They
    lose to the dispatcher's equal shares where a batch streams for tens of microseconds, because a cluster's CTAs stay
    with their sequence, and to split and combine for one long sequence, whose parts fill the GPU."""
    Hq, Hkv, D, batch, context = d.num_q_heads, d.num_kv_heads, d.head_dim, d.batch_size, d.context_length
    if D not in _PER_POSITION or Hq % Hkv:
        return 0, False
    group, pairs, positions = Hq // Hkv, batch * Hkv, (_ONE if batch == 1 else _LONGEST) * context
    cache_bytes = 4.0 * D * pairs * (_ONE if batch == 1 else _MEAN) * context
    per_position = _PER_POSITION[D] * (_TWO_RUNS if group > 8 else 1.0)
    best, route = 0.95 * _dispatcher_us(batch, cache_bytes, append), (0, False)
    function = None
    for parts in CLUSTER_PARTS:
        plan = d.hip.lean_plan(Hq, Hkv, D, parts, context, True)
        if not plan.ok or _cluster_us(parts, pairs, pairs, positions, per_position, 1 << 30, cache_bytes) >= best:
            continue                                        # not even with an SM for every CTA
        if function is None:
            function = d.codegen.load_kernel_safe(d.hip, 'decode_attention', d.hip.get_gpu_architecture(), cluster_kernel_name(group, D))[1]
        resident = d.hip.max_active_clusters(function, parts, plan.threads, plan.smem_bytes)
        if resident < 1:
            continue
        us = _cluster_us(parts, pairs, resident, positions, per_position, d.num_sms, cache_bytes)
        if us < best:
            best, route = us, (parts, True)
    parts = d.num_sms // Hkv
    if (batch == 1 and context <= LEAN_SPLIT_MAX_CONTEXT and 1 < parts <= d.max_chunks and
            d.hip.lean_plan(Hq, Hkv, D, parts, context, False).ok and _split_us(parts, positions, D, cache_bytes) < best):
        route = parts, False
    return route


UNSPLIT_MIN_CAPACITY = 256          # cache positions a sequence, by the stride; above them flash_attention_kernel goes to clusters


def _unsplit_parts(hip, kernels: dict, name: str, Hq: int, Hkv: int, D: int, pairs: int, capacity: int):
    """(parts, plan), or (0, None).  Sizes alone decide, so `kernels` remembers a thousand of them."""
    known = kernels.setdefault("parts", {})
    key = (Hq, Hkv, D, pairs, capacity)
    if key not in known:
        if len(known) >= 1024:
            known.clear()
        best = (math.inf, 0, None)
        for parts in CLUSTER_PARTS:
            plan = hip.lean_plan(Hq, Hkv, D, parts, capacity, True)
            if not plan.ok or hip.max_active_clusters(kernels[name], parts, plan.threads, plan.smem_bytes) < pairs:
                continue
            us = _cluster_us(parts, pairs, pairs, _LONGEST * capacity, _PER_POSITION[D], hip.get_num_cus(), 0.0)
            if us < best[0]:
                best = (us, parts, plan)
        known[key] = best[1:]
    return known[key]


def unsplit_as_clusters(hip, kernels: dict, args: list, grid, block):
    """flash_attention_kernel's launch (13 arguments, grid (batch, query heads, 1), block (head_dim)) as a launch of the
    cluster kernels, (function, args, grid, block, shared_mem), or None where its own builds serve it.

    Its geometry has one block walk a whole sequence; a cluster per (sequence, KV head) has as many SMs on it as the grid
    leaves and reads K and V once for the group.  us a layer, plain stream order, builds / clusters: four sequences of 12
    heads on 2 of 128, 64 positions 4.8 / 5.3, 200: 5.9 / 5.3, 600: 8.6 / 5.4, 1,500: 15.3 / 6.3, 4,000: 43 / 9.6.  So:
    caches with room for more than 256 positions (512 with two runs of query heads: 6.5 us at the least), and no more
    pairs than clusters run at once (a second wave costs more than short sequences take: 64 sequences of 200 positions
    19 / 21, of 64 8 / 17)."""
    if len(args) != 13:
        return None
    value = lambda a: a if isinstance(a, int) else getattr(a, "value", None) or 0
    q, k, v, k_cache, v_cache, out, _, Hq, Hkv, D, scale, offsets, stride = (value(a) for a in args)
    batch = int(grid[0])
    if (D not in _PER_POSITION or Hkv <= 0 or Hq <= 0 or Hq % Hkv or stride <= 0 or stride % 8 or (q | k | v | k_cache | v_cache) % 16 or
            tuple(int(x) for x in grid) != (batch, Hq, 1) or tuple(int(x) for x in block) != (D, 1, 1)):
        return None
    group, pairs, capacity = Hq // Hkv, batch * Hkv, stride // (Hkv * D)
    name = cluster_kernel_name(group, D)
    if name not in kernels or capacity <= UNSPLIT_MIN_CAPACITY * (2 if group > 8 else 1):
        return None
    parts, plan = _unsplit_parts(hip, kernels, name, Hq, Hkv, D, pairs, capacity)
    if not parts:
        return None
    vp, ci, cf = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    lean = [vp(q), vp(k_cache), vp(v_cache), vp(0), vp(0), vp(0), ci(Hq), ci(Hkv), ci(D), cf(scale), vp(offsets), ci(stride), ci(parts),
            vp(k), vp(v), vp(out), ci(1), ci(FLAG_WAIT_FIRST), ci(plan.depth), vp(0), vp(0), vp(0), vp(0), vp(0), ci(-1), ci(0)]
    return kernels[name], lean, ClusterGrid((pairs * parts, 1, 1), parts), (plan.threads, 1, 1), plan.smem_bytes
