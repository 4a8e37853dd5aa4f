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
from .split_kv_attention import UNSPLIT_MAX_CONTEXT

FLAG_PREFETCH_Q = 8
FLAG_WAIT_FIRST = 32
FLAG_ROWS_FINAL = 64
FLAG_KEEP = 128


SPLIT, CLUSTER, HALF = 0, 1, 2      # kinds of route: split and combine; clusters; clusters of blocks of half the warps


def cluster_kernel_name(kind: int, group: int, head_dim: int) -> str:
    return f"vteb_decode_cluster_{'half_' if kind == HALF else ''}{'2_' if group > 8 else ''}d{head_dim}_kernel"


class LeanRoute:
    """`parts` CTAs per (sequence, KV head): one launch a layer (CLUSTER, HALF), or split and combine."""

    def __init__(self, dispatcher, parts: int, kind: int, append: bool):
        d = self.d = dispatcher
        self.parts, self.kind, self.append, self.cluster = int(parts), int(kind), bool(append), kind != SPLIT
        self.plan = d.hip.lean_plan(d.num_q_heads, d.num_kv_heads, d.head_dim, self.parts, d.context_length, kind)
        if not self.plan.ok:
            raise CudaSafetyError(f"{self.parts} CTAs per (sequence, KV head) are not covered for this geometry")
        if not self.cluster and self.parts > d.max_chunks:      # the partial buffers hold max_chunks a row
            raise CudaSafetyError(f"{self.parts} splits, the partial buffers have room for {d.max_chunks}")
        load = lambda symbol: d.codegen.load_kernel_safe(d.hip, 'decode_attention', d.hip.get_gpu_architecture(), symbol)[1]
        self.name = (cluster_kernel_name(kind, d.num_q_heads // d.num_kv_heads, d.head_dim) if self.cluster
                     else f"vteb_split_kv_lean_d{d.head_dim}_kernel")
        self.function, self._resident = load(self.name), None
        if not self.cluster:
            self.combine = load('vteb_split_kv_combine_small_kernel' if self.parts <= 32 else
                                'vteb_split_kv_combine_f32_kernel' if d.output_f32 else 'vteb_split_kv_combine_f16_kernel')

    def pays(self, longest: int, total: int) -> bool:
        """Whether a step whose longest sequence has `longest` positions, and all together `total`, is estimated shorter on
        this route than in the dispatcher's launches.  A route is chosen by capacity, but its CTAs stay with their sequence: one
        long sequence among short ones takes as long as its parts, where equal shares spread it over the GPU (32 sequences of
        12 heads on 2 of 128, one of 32,768 positions, 31 of 500: 71 us a layer in clusters, 29)."""
        d = self.d
        if not self.cluster or d.context_length <= UNSPLIT_MAX_CONTEXT:
            return True
        us = lambda kind, parts, resident: d.hip.lean_step_estimate(kind, parts, d.num_q_heads, d.num_kv_heads, d.head_dim, d.batch_size,
                                                                    d.context_length, longest, total, resident)
        if self._resident is None:
            self._resident = d.hip.max_active_clusters(self.function, self.parts, self.plan.threads, self.plan.smem_bytes)
        return us(self.kind, self.parts, self._resident) <= us(-1, 0, 0) + (LEAST_APPEND_US if self.append else 0.0)

    def pays_up_to(self) -> int:
        """A length up to which the route pays whatever the other sequences have."""
        batch, lo, hi = self.d.batch_size, 0, self.d.context_length
        while lo < hi:
            mid = (lo + hi + 1) // 2
            if self.pays(mid, mid + batch - 1) and self.pays(mid, mid * batch):
                lo = mid
            else:
                hi = mid - 1
        return lo

    def launches(self, layer: int, tensor_mapping: dict, kv_offset_ptr: int, batch: int, keep: tuple = (0, 0)):
        """`keep`: where the kernel leaves a copy of Q and of the offsets, for a layer whose partials may be asked for."""
        d = self.d
        vp, ci, cf = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
        attention_scale = d.metadata.get('attention_scale')
        scale = float(attention_scale) if attention_scale else 1.0 / math.sqrt(d.head_dim)
        ptr = lambda name: d._resolve_ptr(tensor_mapping, name)
        q, out = ptr(f'blk.{layer}.q_proj.output'), ptr(f'blk.{layer}.attention.output')
        k_cache, v_cache = d._resolve_kv_cache_ptrs(layer, tensor_mapping)
        stride = int(tensor_mapping.get('kv_batch_stride_elements', 0))
        d._validate(batch, q, k_cache, v_cache, out, kv_offset_ptr, stride)
        k_new = v_new = 0
        if self.append:
            k_new, v_new = ptr(f'blk.{layer}.k_proj.output'), ptr(f'blk.{layer}.v_proj.output')
            if not k_new or not v_new:                     # null means to the kernels that the row is in the cache already
                raise CudaSafetyError(f"layer {layer}: the new K / V rows could not be resolved (null)")
            if (k_new | v_new) % 16:                       # 16-byte loads; an append launch takes rows of any alignment
                return d.build_launches(layer, tensor_mapping, kv_offset_ptr, batch)
        flags = (0 if self.append else FLAG_ROWS_FINAL) | (FLAG_PREFETCH_Q if d.hip.programmatic_launch else 0)
        rope = d._rope_arguments(tensor_mapping) if d.fuse_rope else [vp(0), vp(0), ci(-1), ci(0)]
        Hq, Hkv, D, N = d.num_q_heads, d.num_kv_heads, d.head_dim, self.parts
        out_kind = 2 if d.output_f32 else 1
        next_k = next_v = 0
        partials = [vp(0), vp(0), vp(0)]
        if not self.cluster:
            partials = [vp(p.ptr) for p in d.partial_buffers]
            next_k, next_v = d._next_caches(layer, tensor_mapping)
        if keep[0]:
            next_k, next_v = keep
            flags |= FLAG_KEEP
        args = [vp(q), vp(k_cache), vp(v_cache), *partials, ci(Hq), ci(Hkv), ci(D), cf(scale), vp(kv_offset_ptr), ci(stride),
                ci(N), vp(k_new), vp(v_new), vp(out), ci(out_kind), ci(flags), ci(self.plan.depth), vp(d.work_ptr + 4),
                vp(next_k), vp(next_v)] + rope
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


CLUSTER_PARTS = (2, 3, 4, 5, 6, 8, 9, 12, 16)              # more than 8 only where the device has room for such clusters
LEAN_SPLIT_MAX_CONTEXT = 131072
SPLIT_ALONE_BYTES = 24 << 20                               # K and V rows in a cache up to which it pays without an append
APPEND_US = 2.0                                            # the append launch that the other routes have,
LEAST_APPEND_US = 1.5                                      # at the least,
SMALL_APPEND_US = 0.5                                      # in front of the one launch of a small cache
MARGIN = 0.95                                              # a route has to be estimated this much below the dispatcher's launches


def cluster_options(hip, load, Hq: int, Hkv: int, D: int, batch: int, context: int, below: float):
    """(estimated us, kind, parts, function, plan, clusters at once) of every cluster route estimated `below` that many
    us.  `load(name)` loads a kernel; None where it is not to be had."""
    for kind in (CLUSTER, HALF):
        function = None
        for parts in CLUSTER_PARTS:
            plan = hip.lean_plan(Hq, Hkv, D, parts, context, kind)
            if not plan.ok or hip.lean_estimate(kind, parts, Hq, Hkv, D, batch, context, batch * Hkv) >= below:
                continue                                   # not even with room for all clusters at once
            function = function or load(cluster_kernel_name(kind, Hq // Hkv, D))
            if function is None:
                break
            resident = hip.max_active_clusters(function, parts, plan.threads, plan.smem_bytes)
            us = hip.lean_estimate(kind, parts, Hq, Hkv, D, batch, context, resident)
            if resident > 0 and us < below:
                yield us, kind, parts, function, plan, resident


def choose_lean_route(d, append: bool) -> tuple:
    """(CTAs per (sequence, KV head), kind) for a dispatcher's geometry; (0, 0): its own launches.  The estimates and what
    they are fitted to: csrc/kernels/lean_decode.cuh.

    Clusters win wherever latency counts: a layer is one dependent launch of 3.3 us instead of two or three (7.1).  They
    lose to the dispatcher's equal shares where a batch streams for a hundred microseconds, because a cluster's CTAs stay
    with their sequence, and to split and combine for one long sequence, whose parts fill the GPU.  Up to
    UNSPLIT_MAX_CONTEXT positions the dispatcher's layer is one launch too, and many clusters take longer to start than
    its CTAs: 64 sequences of 32 heads on 8 of 64, room for 16 positions 4.9 us, in clusters 15.9.

    Split and combine of one KV head a CTA, where there is no append launch to save, us / the dispatcher's: 12 heads on 2 of
    128, 32,768 positions 9.6 / 10.3, 32 on 8 of 64 15.4 / 16.4; 8 on 2 of 256, 8,192: 8.2 / 8.7, 16,384: 12.3 / 11.9; 16 on 4
    of 64, 16,384: 7.7 / 8.2, 32,768: 12.3 / 10.8."""
    Hq, Hkv, D, batch, context = d.num_q_heads, d.num_kv_heads, d.head_dim, d.batch_size, d.context_length
    if Hkv <= 0 or Hq % Hkv or D not in (64, 128, 256):
        return 0, 0
    best, route = MARGIN * (d.hip.lean_estimate(-1, 0, Hq, Hkv, D, batch, context, 0) + (APPEND_US if append else 0.0)), (0, 0)
    load = lambda name: d.codegen.load_kernel_safe(d.hip, 'decode_attention', d.hip.get_gpu_architecture(), name)[1]
    for us, kind, parts, _, _, resident in cluster_options(d.hip, load, Hq, Hkv, D, batch, context, best):
        if us < best:
            best, route, clusters = us, (parts, kind), resident
    if context <= UNSPLIT_MAX_CONTEXT and route[0]:
        us = lambda kind, parts, resident: d.hip.lean_step_estimate(kind, parts, Hq, Hkv, D, batch, context, context, batch * context, resident)
        return route if us(route[1], route[0], clusters) <= MARGIN * (us(-1, 0, 0) + (SMALL_APPEND_US if append else 0.0)) else (0, 0)
    parts = d.num_sms // Hkv
    if not append and (D == 256 or D == 64 and Hkv < 8) and context * Hkv * D * 4 > SPLIT_ALONE_BYTES:
        return route
    if (batch == 1 and context <= LEAN_SPLIT_MAX_CONTEXT and 1 < parts <= d.max_chunks and d.hip.lean_plan(Hq, Hkv, D, parts, context, SPLIT).ok
            and d.hip.lean_estimate(SPLIT, parts, Hq, Hkv, D, 1, context, 0) < best):
        route = parts, SPLIT
    return route


UNSPLIT_MIN_CAPACITY = 256          # cache positions a sequence, by the stride; above them flash_attention_kernel goes to clusters


def _unsplit_option(hip, kernels: dict, Hq: int, Hkv: int, D: int, pairs: int, capacity: int):
    """(us, parts, function, plan), parts 0 where no clusters hold all pairs at once.  Sizes alone decide, so `kernels`
    remembers a thousand of them."""
    known = kernels.setdefault("parts", {})
    key = (Hq, Hkv, D, pairs, capacity)
    if key not in known:
        if len(known) >= 1024:
            known.clear()
        options = cluster_options(hip, kernels.get, Hq, Hkv, D, pairs // Hkv, capacity, math.inf)
        known[key] = min(((us, parts, function, plan) for us, _, parts, function, plan, resident in options if resident >= pairs),
                         key=lambda o: o[0], default=(0.0, 0, None, None))
    return known[key]


def unsplit_as_clusters(hip, kernels: dict, args: list, grid, block, status: int = 0):
    """flash_attention_kernel's launch (13 arguments, grid (batch, query heads, 1), block (head_dim)) as a launch of the
    cluster kernels, (function, args, grid, block, shared_mem), or None where its own builds serve it.  `status`: where a
    launch reports a wait that ran out.

    Its geometry has one block walk a whole sequence; a cluster per (sequence, KV head) has as many SMs on it as the grid
    leaves and reads K and V once for the group.  us a layer, plain stream order, builds / clusters: four sequences of 12
    heads on 2 of 128, 64 positions 4.8 / 5.3, 200: 5.9 / 5.3, 600: 8.6 / 5.4, 1,500: 15.3 / 6.3, 4,000: 43 / 9.6 (the clusters 0.6 less
    since they set themselves up ahead of their wait).  So:
    caches with room for more than 256 positions (512 with two runs of query heads: 6.5 us at the least), and no more
    pairs than clusters run at once (a second wave costs more than short sequences take: 64 sequences of 200 positions
    19 / 21, of 64 8 / 17).  The host sees the room, not the lengths: a sequence of up to about 100 positions (150 of 256-wide
    heads, 200 with two runs) in such a cache takes longer than its own builds, 4.9 us instead of 3.3 (one position), 4.6 (64)
    and 4.4 (128).  One CTA alone for those gave 4.1 to 4.4, and 0.25 more to every longer one."""
    if len(args) != 13:
        return None
    value = lambda a: a if isinstance(a, int) else getattr(a, "value", None) or 0
    q, k, v, k_cache, v_cache, out, _, Hq, Hkv, D, scale, offsets, stride = (value(a) for a in args)
    batch = int(grid[0])
    if (D not in (64, 128, 256) or Hkv <= 0 or Hq <= 0 or Hq % Hkv or stride <= 0 or stride % 8 or (q | k | v | k_cache | v_cache) % 16 or
            tuple(int(x) for x in grid) != (batch, Hq, 1) or tuple(int(x) for x in block) != (D, 1, 1)):
        return None
    group, pairs, capacity = Hq // Hkv, batch * Hkv, stride // (Hkv * D)
    if capacity <= UNSPLIT_MIN_CAPACITY * (2 if group > 8 else 1):
        return None
    _, parts, function, plan = _unsplit_option(hip, kernels, Hq, Hkv, D, pairs, capacity)
    if not parts:
        return None
    vp, ci, cf = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    lean = [vp(q), vp(k_cache), vp(v_cache), vp(0), vp(0), vp(0), ci(Hq), ci(Hkv), ci(D), cf(scale), vp(offsets), ci(stride), ci(parts),
            vp(k), vp(v), vp(out), ci(1), ci(FLAG_WAIT_FIRST), ci(plan.depth), vp(status), vp(0), vp(0), vp(0), vp(0), ci(-1), ci(0)]
    return function, lean, ClusterGrid((pairs * parts, 1, 1), parts), (plan.threads, 1, 1), plan.smem_bytes
