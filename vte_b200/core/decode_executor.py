"""Decode-step driver for the attention path: one captured CUDA graph per step.

The attention-only counterpart of `HIPGraphExecutor` / `BatchedHIPGraphExecutor`
(vte/core/hip_graph_executor.py:504-819, vte/core/batched_hip_graph_executor.py:
231-292): it owns the per-layer buffers an executor would hand the dispatcher
(`blk.{l}.q_proj.output`, `blk.{l}.k_proj.output`, `blk.{l}.v_proj.output`,
`blk.{l}.attention.output`, `blk.{l}.kv_cache.k/.v`,
`kv_batch_stride_elements`), records every layer's launches from
`SplitKVAttentionDispatcher.build_launches` into one graph
(hip_graph_executor.py:635-651), and replays it per token after rewriting the
device array of per-sequence kv offsets from a staging buffer
(hip_graph_executor.py:772-789; batched: batched_hip_graph_executor.py:276-285).
Unlike the reference's batched executor it admits ragged context lengths.
"""
from __future__ import annotations

import ctypes
import types
from typing import Optional

import numpy as np

from ..bridge.cuda_runtime import HostStep, StepArgs
from ..bridge.errors import CudaSafetyError
from ..bridge.memory import MemoryRegion, SlabAllocator
from ..config import ENV_NO_PDL, env_flag
from .lean_route import LeanRoute, choose_lean_route
from .split_kv_attention import FLAG_DIRECT_OUTPUT, SplitKVAttentionDispatcher
from .step_route import StepRoute, one_launch_pays


def _round_up(x: int, m: int) -> int:
    return (x + m - 1) // m * m


# Staging copies of an end-to-end step up to this size are launches (build_io_graph).  Measured, copy nodes against
# launches, a step of 12 query heads: 3 KB of Q 34.2 / 27.1 us, 84 KB (28 layers) 182 / 173, 336 KB 289 / 284;
# of 32 heads of 64: 1.8 MB 730 / 730, 7 MB 2,099 / 2,104.
STAGE_COPY_MAX_BYTES = 1 << 20


# Staging slots for the offsets of steps in flight.  With one slot and an event a step the event alone took 2.5 us of a
# queued step of 97 (28 layers, one sequence of 1,531 positions).
OFFSET_SLOTS = 64

STEP_OFFSETS = 64       # sequences whose offsets may be among the arguments of a step of one launch (kStepOffsets in csrc/kernels/step_decode.cuh)
NOT_SIDE_BY_SIDE = "one launch for all layers: a layer reads or writes what another writes, or has pointers that are not 16-byte aligned"


class DecodeAttentionExecutor:
    _step, _one_launch, _direct, _closed = None, False, (), False
    _graph_kept = _io_kept = None
    _recorded_step = ()

    def __init__(self, hip, codegen, metadata: dict, batch_size: int, context_length: int, n_layers: int, *,
                 n_kv_buffers: Optional[int] = None, num_splits: Optional[int] = None, output_f32: bool = True,
                 use_graph: bool = True, programmatic: Optional[bool] = None, compat: bool = False,
                 with_append: bool = False, fixed_chunk_size=None, min_chunk: Optional[int] = None,
                 strict_empty_splits: bool = False, allocator: Optional[SlabAllocator] = None,
                 emit_state: bool = False, per_layer_hook=None, prefetch_next_layer: bool = True,
                 fused_combine: Optional[bool] = None, variant: str = "auto", rope: str = "off",
                 rope_theta: float = 1e6, tensor_maps: bool = True, fuse_append: bool = False,
                 balanced: Optional[bool] = None, wide: Optional[bool] = None, lean: Optional[tuple] = None,
                 one_launch: Optional[bool] = None):
        self.hip = hip
        if lean is not None and lean[0] and (compat or strict_empty_splits or emit_state or fused_combine):
            raise CudaSafetyError("a route of lean_route.py has no compat kernels, empty-split partials, shard states or fused combine")
        # nothing that the caller has asked for ties the step to the dispatcher's own launches
        open_layout = not (num_splits or compat or strict_empty_splits or emit_state or fused_combine or balanced is not None or
                           wide is not None) and (fixed_chunk_size is None and min_chunk is None and variant == "auto" and
                                                  tensor_maps and prefetch_next_layer)
        if one_launch and (lean is not None or not open_layout or not use_graph):
            raise CudaSafetyError("one launch for all layers takes no split layout, partials, shard states or shapes of the caller's, "
                                  "and no step without a graph")
        # rope: "off" = Q and K arrive rotated; "separate" = the reference's standalone rotation
        # launch runs before the append (rotating the projections in place); "fused" = the append
        # rotates K and the split kernel rotates Q.  Either way the step includes the append.
        # "fused-append": as "fused", and the split kernel also does the append (no append launch).
        if rope not in ("off", "separate", "fused", "fused-append"):
            raise CudaSafetyError(f"rope must be off, separate, fused or fused-append, not {rope!r}")
        self.rope = rope
        if rope != "off":
            with_append = True
        self.metadata = dict(metadata)
        self.B = int(batch_size)
        self.S = int(context_length)
        self.L = int(n_layers)
        self.n_kv = int(n_kv_buffers or n_layers)   # distinct KV buffers; layers cycle through them
        if not (1 <= self.n_kv <= self.L):
            raise CudaSafetyError(f"n_kv_buffers {self.n_kv} outside 1..{self.L}")
        self.Hq = int(metadata.get('attention.head_count', 12))
        self.Hkv = int(metadata.get('attention.head_count_kv', 2))
        self.D = int(metadata.get('attention.key_length', 128))
        self.output_f32 = bool(output_f32)
        self.use_graph = bool(use_graph)
        self.programmatic = (not env_flag(ENV_NO_PDL)) if programmatic is None else bool(programmatic)
        self.with_append = bool(with_append)
        self.emit_state = bool(emit_state)          # outputs are [B, Hq, D + 2] fp32 shard states
        self.per_layer_hook = per_layer_hook        # called as hook(layer) after a layer's launches are recorded
        self.launch_rewriter = None                 # optional: rewriter(layer, launches) -> launches, before recording
        self.kv_batch_stride = self.S * self.Hkv * self.D
        if self.kv_batch_stride >= 2 ** 31:
            raise CudaSafetyError("one sequence's cache exceeds 2^31 elements: the kernel ABI's stride is an int")

        out_elem = 4 if self.output_f32 else 2
        self.kv_bytes = self.B * self.kv_batch_stride * 2           # one K (or V) cache of one layer
        self.q_bytes = self.B * self.Hq * self.D * 2
        self.kvnew_bytes = self.B * self.Hkv * self.D * 2
        self.out_bytes = self.B * self.Hq * self.D * out_elem
        if self.emit_state:
            self.out_bytes = self.B * self.Hq * (self.D + 2) * 4

        self._owns_allocator = allocator is None
        if allocator is None:
            need = (2 * self.n_kv * (self.kv_bytes + 256) + self.L * (self.q_bytes + 2 * self.kvnew_bytes
                    + self.out_bytes + 1024) + (64 << 20) + 4 * self.B + 4096 + (4 * self.S * self.D + 4096 if rope != "off" else 0))
            free_b, total_b = hip.get_real_mem_info()
            allocator = SlabAllocator(hip, total_b, requested_pool_size=need)
            allocator.initialize()
        self.allocator = allocator
        A = allocator.allocate
        # Every layer's Q, then the kv offsets, in one allocation; every layer's output, then the
        # dispatcher's work words (ticket, status), in another: an end-to-end step is then one copy in
        # and one copy out, and the status word comes back with the results.
        self._q_tail = _round_up(self.L * self.q_bytes, 256)
        self._out_tail = _round_up(self.L * self.out_bytes, 256)
        self.q_all = A(self._q_tail + _round_up(4 * self.B, 256), "q_proj.output.all", MemoryRegion.ACTIVATIONS)
        self.out_all = A(self._out_tail + 256, "attention.output.all", MemoryRegion.ACTIVATIONS)
        self.offsets = types.SimpleNamespace(ptr=self.q_all.ptr + self._q_tail, size=4 * self.B)
        self.dispatcher = SplitKVAttentionDispatcher(
            hip, codegen, self.metadata, allocator=allocator, context_length=self.S, batch_size=self.B,
            num_splits=num_splits, fixed_chunk_size=fixed_chunk_size, compat=compat, min_chunk=min_chunk,
            output_f32=self.output_f32, strict_empty_splits=strict_empty_splits, emit_state=self.emit_state,
            prefetch_next_layer=prefetch_next_layer, fused_combine=fused_combine, variant=variant,
            fuse_rope=rope in ("fused", "fused-append"), fuse_append=(rope == "fused-append" or fuse_append), tensor_maps=tensor_maps,
            work_ptr=self.out_all.ptr + self._out_tail, balanced=balanced, wide=wide)

        # lean: (CTAs per (sequence, KV head), kind) of a route of lean_route.py; (0, 0) never, None where one pays and
        # the caller has asked for nothing that the dispatcher's own launches have and these have not.
        self._lean = lean if lean is not None else None if open_layout else (0, 0)
        self._route, self._forced_route = None, lean is not None
        # one_launch: the whole step in one launch over all layers (step_route.py); None where it may and pays, False: a launch
        # list per layer, in which a layer starts when the one in front of it is done, True: refused where it may not
        self._one_launch = one_launch if one_launch is not None else None if lean is None and open_layout else False
        self._step, self._direct, self._host_step = None, [], None
        # where lengths can make the dispatcher's launches the shorter ones: a step of those is captured beside the route's, and
        # each step takes one by its longest and total length; up to _route_pays_to positions it is the route's in any case
        self._route_pays_to, self._on_route, self._launches = self.S, True, (0, 0)
        self._plain_graph_exec = self._plain_io_graph_exec = None
        # what partials of a routed step can be had from: the last layer's Q and offsets as the step saw them, the names it
        # was captured with (each graph's, and the last step's), and whether the partial buffers are still to be filled
        self._kept, self._kept_names, self._partials_due = None, None, False
        self.k_cache = [A(self.kv_bytes, f"kv_cache.k.{i}", MemoryRegion.KV_CACHE) for i in range(self.n_kv)]
        self.v_cache = [A(self.kv_bytes, f"kv_cache.v.{i}", MemoryRegion.KV_CACHE) for i in range(self.n_kv)]
        # all layers' Q (and outputs) are contiguous so one copy moves a whole step's worth
        self.knew_all = A(self.L * self.kvnew_bytes, "k_proj.output.all", MemoryRegion.ACTIVATIONS)
        self.vnew_all = A(self.L * self.kvnew_bytes, "v_proj.output.all", MemoryRegion.ACTIVATIONS)

        self.tensor_mapping = {'kv_batch_stride_elements': self.kv_batch_stride}
        for l in range(self.L):
            self.tensor_mapping[f'blk.{l}.q_proj.output'] = self.q_all.ptr + l * self.q_bytes
            self.tensor_mapping[f'blk.{l}.k_proj.output'] = self.knew_all.ptr + l * self.kvnew_bytes
            self.tensor_mapping[f'blk.{l}.v_proj.output'] = self.vnew_all.ptr + l * self.kvnew_bytes
            self.tensor_mapping[f'blk.{l}.attention.output'] = self.out_all.ptr + l * self.out_bytes
            self.tensor_mapping[f'blk.{l}.kv_cache.k'] = self.k_cache[l % self.n_kv]
            self.tensor_mapping[f'blk.{l}.kv_cache.v'] = self.v_cache[l % self.n_kv]

        if self.rope != "off":
            from ..workloads import build_rope_cache
            rope_type = int(self.metadata.get('rope_type', 0))
            width = int(self.metadata.get('rotary_dim', self.D)) if rope_type == 2 else self.D
            cos, sin = build_rope_cache(self.S, width, float(rope_theta))
            self.rope_cos = A(cos.nbytes, "rope_cos", MemoryRegion.ACTIVATIONS)
            self.rope_sin = A(sin.nbytes, "rope_sin", MemoryRegion.ACTIVATIONS)
            hip.safe_memcpy_host_to_device(ctypes.c_void_p(self.rope_cos.ptr), cos, "rope_cos upload")
            hip.safe_memcpy_host_to_device(ctypes.c_void_p(self.rope_sin.ptr), sin, "rope_sin upload")
            self.tensor_mapping['rope_cos'] = self.rope_cos
            self.tensor_mapping['rope_sin'] = self.rope_sin

        # pinned staging: offsets, a step's Q, a step's outputs
        self._stage_q = hip.host_alloc(self._q_tail + _round_up(4 * self.B, 256))          # Q of every layer, then the offsets
        self._stage_offsets = ctypes.c_void_p(self._stage_q.value + self._q_tail)
        self._stage_out = hip.host_alloc(self._out_tail + 256)                               # outputs, then the work words
        ctypes.memset(self._stage_out.value, 0, self._out_tail + 256)
        # kv offsets of device-side steps: a ring of staging slots, each half marked by one event when its last copy is
        # enqueued and waited for when its first slot comes up again
        self._offset_ring = hip.host_alloc(OFFSET_SLOTS * _round_up(4 * self.B, 256))
        self._offset_slot, self._offset_events = 0, [None, None]
        self.codegen = codegen
        self._copy_fn = None            # staging copies as launches
        self._graph_exec = None
        self._io_graph_exec = None      # staging copies + the layers' launches + the output copy, as one graph
        self._stage_event = None        # recorded after a step's staging copies; the next step waits for it
        self._stage_in_flight = False
        self.kernel_launches_per_step = 0

    # ---- data movement helpers ----------------------------------------------------
    def upload_layer(self, layer: int, q: np.ndarray, k_cache: Optional[np.ndarray] = None,
                     v_cache: Optional[np.ndarray] = None):
        """Host -> device of one layer's Q [B,Hq,D] and (optionally) its caches
        [B,max_seq,Hkv,D], all fp16."""
        self.hip.safe_memcpy_host_to_device(ctypes.c_void_p(self.q_all.ptr + layer * self.q_bytes),
                                            np.ascontiguousarray(q, dtype=np.float16), "q upload")
        if k_cache is not None:
            self.upload_cache(layer % self.n_kv, k_cache, v_cache)

    def upload_cache(self, buf: int, k_cache: np.ndarray, v_cache: np.ndarray):
        if buf == (self.L - 1) % self.n_kv:
            self._fill_partials()
        for dst, src in ((self.k_cache[buf], k_cache), (self.v_cache[buf], v_cache)):
            src = np.ascontiguousarray(src, dtype=np.float16)
            if src.shape != (self.B, self.S, self.Hkv, self.D):
                raise CudaSafetyError(f"cache shape {src.shape} != {(self.B, self.S, self.Hkv, self.D)}")
            self.hip.safe_memcpy_host_to_device(ctypes.c_void_p(dst.ptr), src, "kv upload")

    def upload_new_kv(self, layer: int, k_new: np.ndarray, v_new: np.ndarray):
        self.hip.safe_memcpy_host_to_device(ctypes.c_void_p(self.knew_all.ptr + layer * self.kvnew_bytes),
                                            np.ascontiguousarray(k_new, dtype=np.float16), "k_new upload")
        self.hip.safe_memcpy_host_to_device(ctypes.c_void_p(self.vnew_all.ptr + layer * self.kvnew_bytes),
                                            np.ascontiguousarray(v_new, dtype=np.float16), "v_new upload")

    def fill_cache_on_device(self, buf: int, seed: int, sigma: float = 1.0, outlier_prob: float = 0.0,
                             outlier_scale: float = 1.0):
        """Synthetic N(0, sigma) cache contents generated on the device."""
        if buf == (self.L - 1) % self.n_kv:
            self._fill_partials()
        n = self.B * self.kv_batch_stride
        self.hip.fill_normal_f16(ctypes.c_void_p(self.k_cache[buf].ptr), n, 2 * seed + 1, sigma, outlier_prob, outlier_scale)
        self.hip.fill_normal_f16(ctypes.c_void_p(self.v_cache[buf].ptr), n, 2 * seed + 2, sigma, outlier_prob, outlier_scale)

    def download_cache_rows(self, buf: int, b: int, n_rows: int):
        """(K, V) [n_rows, Hkv, D] fp16 of sequence b, for checking against the oracle."""
        row = self.Hkv * self.D
        k = np.empty((n_rows, self.Hkv, self.D), dtype=np.float16)
        v = np.empty_like(k)
        off = b * self.kv_batch_stride * 2
        self.hip.safe_memcpy_device_to_host(k, ctypes.c_void_p(self.k_cache[buf].ptr + off), "kv rows for output check")
        self.hip.safe_memcpy_device_to_host(v, ctypes.c_void_p(self.v_cache[buf].ptr + off), "kv rows for output check")
        assert k.nbytes == n_rows * row * 2
        return k, v

    # ---- graph ----------------------------------------------------------------------
    def _stage_copy(self, dst: int, src: int, nbytes: int, first: bool = False):
        """Record a staging copy as a launch.  Both ends are 256-byte aligned and padded to 256 bytes."""
        words = -(-nbytes // 16)
        programmatic, self.hip.programmatic_launch = self.hip.programmatic_launch, self.programmatic and not first
        try:
            self.hip.launch_kernel_recorded(self._copy_fn, [ctypes.c_void_p(src), ctypes.c_void_p(dst), ctypes.c_int(words)],
                                            (max(1, min(self.hip.get_num_cus(), -(-words // 256))), 1, 1), (256, 1, 1), 0)
        finally:
            self.hip.programmatic_launch = programmatic

    def layer_launches(self, layer: int, plain: bool = False):
        """What a step launches for a layer (without a rotation launch of its own); `plain`: in the dispatcher's launches."""
        if self._route is not None and not plain and self.dispatcher.offsets_final:
            last = layer == self.L - 1
            launches = self._route.launches(layer, self.tensor_mapping, self.offsets.ptr, self.B,
                                            (self._kept.ptr, self._kept.ptr + _round_up(self.q_bytes, 256)) if last else (0, 0))
            if last:
                self._kept_names = dict(self.tensor_mapping) if launches[0][0] is self._route.function else None
            return launches
        launches = self.dispatcher.build_launches(layer, self.tensor_mapping, self.offsets.ptr, batch=self.B)
        return launches if self.with_append or self.dispatcher.fuse_append else launches[1:]

    @property
    def route_name(self):
        """(kernel, CTAs per (sequence, KV head)) where the last captured step did not take the dispatcher's launches, else None;
        (kernel, 0) where it is one launch."""
        if self._recorded_step:
            return self._step.name, 0
        return (self._route.name, self._route.parts) if self._route is not None and self._on_route else None

    def _record_all(self, after_copy: bool = False, plain: bool = False, one_launch: Optional[list] = None, mirror: Optional[tuple] = None):
        """`one_launch`: what the one launch of all layers takes from the mapping, where it serves."""
        n = 0
        programmatic = self.hip.programmatic_launch
        self._recorded_step = self._record_step(one_launch, mirror) if one_launch else ()
        if one_launch:
            return len(self._recorded_step)
        # within a captured step of nothing but the layers' own launches, offsets and older rows do not change
        self.dispatcher.offsets_final = self.use_graph and self.per_layer_hook is None and self.launch_rewriter is None
        for l in range(self.L):
            launches = self.layer_launches(l, plain)
            if self.launch_rewriter is not None:
                launches = self.launch_rewriter(l, launches)
            if self.rope == "separate":
                launches = [self.dispatcher.build_rope_launch(self.tensor_mapping, self.offsets.ptr, batch=self.B,
                                                              layer_idx=l)] + launches
            for fn, args, grid, block, smem in launches:
                if after_copy and n == 0:
                    # the split kernel reads the kv offsets ahead of its dependency wait: plain stream order
                    # behind the launch that brings them
                    self.hip.programmatic_launch = False
                self.hip.launch_kernel_recorded(fn, args, grid, block, smem)
                n += 1
                self.hip.programmatic_launch = programmatic
            if self.per_layer_hook is not None:
                n += int(self.per_layer_hook(l) or 0)
        return n

    def _record_step(self, layers: list, mirror: Optional[tuple] = None) -> list:
        """Record the launches of a step without an order among its layers."""
        launches = self._step.launches(self.tensor_mapping, self.offsets.ptr, self.B, layers,
                                       (self._kept.ptr, self._kept.ptr + _round_up(self.q_bytes, 256)), mirror)
        self._kept_names = dict(self.tensor_mapping)
        for launch in launches:
            self.hip.launch_kernel_recorded(*launch)
        return launches

    def _serves_one_launch(self) -> Optional[list]:
        """What the one launch takes from the mapping of this moment, which may be another than the one it was chosen with; None where
        a step that is recorded now may not be one launch."""
        if self._step is None or self.per_layer_hook is not None or self.launch_rewriter is not None:
            return None
        layers = self._step.resolve(self.tensor_mapping)
        if self._step.serves(self.tensor_mapping, self.offsets.ptr, self.B, layers):
            return layers
        if self._one_launch:
            raise CudaSafetyError(NOT_SIDE_BY_SIDE)
        return None

    def _choose_route(self) -> Optional[list]:
        """Before a step is captured: whether its layers' launches are the dispatcher's own or a route of lean_route.py.  Where one
        launch for all of them has just been found to serve, what it takes from the mapping."""
        d = self.dispatcher
        if (self._route is not None or self._step is not None or self._lean == (0, 0) and not self._one_launch or not self.use_graph or
                self.per_layer_hook is not None or self.launch_rewriter is not None or not d.enabled or not hasattr(self.hip, 'lean_plan')):
            if self._one_launch and self._step is None:
                raise CudaSafetyError("one launch for all layers needs a captured step without a hook or a rewriter")
            return None
        d._allocate_scratch()                         # and the work words
        append = self.with_append or d.fuse_append
        if self._one_launch is not False:
            layers = self._choose_one_launch(append)
            if layers:
                return layers
        if self._lean is None:
            self._lean = choose_lean_route(d, append)
        if self._lean[0]:
            route = LeanRoute(d, *self._lean, append)
            try:
                self._kept = self.allocator.allocate(_round_up(self.q_bytes, 256) + _round_up(4 * self.B, 256), "attn_partials_source",
                                                     MemoryRegion.SCRATCH)
            except CudaSafetyError:
                if self._forced_route:
                    raise
                self._lean = (0, 0)                   # a caller's allocator with no room for it: the dispatcher's launches need none
                return None
            self._route = route
            if not self._forced_route:
                self._route_pays_to = route.pays_up_to()
        return None

    def _choose_one_launch(self, append: bool) -> Optional[list]:
        """Takes one launch for the step where its layers may run side by side and that pays."""
        d, forced, blocks = self.dispatcher, bool(self._one_launch), []
        if self.rope == "separate" or not hasattr(self.hip, 'step_plan') or (not forced and not one_launch_pays(d, self.L)):
            if forced:
                raise CudaSafetyError("one launch for all layers has no rotation launches")
            return None
        try:
            step = StepRoute(d, self.allocator, self.L, append)
            blocks.append(step.scratch)
            self._kept = self.allocator.allocate(_round_up(self.q_bytes, 256) + _round_up(4 * self.B, 256), "attn_partials_source",
                                                 MemoryRegion.SCRATCH)
            blocks.append(self._kept)
            layers = step.resolve(self.tensor_mapping)
            if not step.serves(self.tensor_mapping, self.offsets.ptr, self.B, layers):
                raise CudaSafetyError(NOT_SIDE_BY_SIDE)
        except CudaSafetyError:
            if forced:
                raise
            for block in blocks:
                self.allocator.free(block)
            self._kept = None
            return None
        self._step = step
        return layers

    def _require_open(self, staging: bool = False):
        """A cleaned-up executor has no staging memory, and device memory only where the caller's allocator holds it."""
        if self._closed and (staging or self._owns_allocator):
            raise CudaSafetyError("the executor has been cleaned up: its memory is gone")

    def build_decode_graph(self):
        """Capture all layers' launches once (hip_graph_executor.py:504-725)."""
        if self._graph_exec is not None:
            return
        self._require_open()
        self.hip.programmatic_launch = self.programmatic
        try:
            if not self.use_graph:
                n = len(self.dispatcher.build_launches(0, self.tensor_mapping, self.offsets.ptr, batch=self.B))
                n += 1 if self.rope == "separate" else 0
                self.kernel_launches_per_step = (n if (self.with_append or self.dispatcher.fuse_append) else n - 1) * self.L
                return
            one = self._choose_route() or self._serves_one_launch()
            self._graph_exec, n, self._graph_kept = self._capture(lambda: self._record_all(one_launch=one))
            self._direct = []
            if one and self.B <= STEP_OFFSETS:
                for fn, (captured,), grid, block, smem in self._recorded_step:
                    args = StepArgs.from_buffer_copy(captured)
                    args.offsets_here = 1
                    self._direct.append((args.offsets, self.hip.prepare_launch(fn, [args], grid, block, smem, self.programmatic)))
            plain = n
            if self._route_pays_to < self.S:
                self._plain_graph_exec, plain, _ = self._capture(lambda: self._record_all(plain=True))
            self._launches = n, plain
            self.kernel_launches_per_step = n
        finally:
            self.hip.programmatic_launch = False

    def _capture(self, record):
        """(executable graph, what `record` returns, the names that partials can be had with) of what `record` launches."""
        last, self._kept_names = self._kept_names, None
        self.hip.stream_begin_capture()
        try:
            n = record()
        finally:
            graph = self.hip.stream_end_capture()
            kept, self._kept_names = self._kept_names, last
        graph_exec = self.hip.graph_instantiate(graph)
        self.hip.graph_destroy(graph)
        return graph_exec, n, kept

    def _pick(self, offsets: np.ndarray, newest: int):
        """Which of two captured steps serves these offsets, the largest of which is `newest`."""
        self._on_route = newest < self._route_pays_to or self._route.pays(newest + 1, int(offsets.sum(dtype=np.int64)) + self.B)
        self.kernel_launches_per_step = self._launches[not self._on_route]

    def build_io_graph(self):
        """One graph for a whole end-to-end step: kv offsets and every layer's Q from pinned
        staging to the device, every layer's launches, every layer's output back to pinned
        staging.  Copies up to STAGE_COPY_MAX_BYTES are launches on the compute queue, larger ones
        copy nodes.  A step is then one graph launch instead of three copies and a launch (the
        reference stages its offsets with a separate copy before each launch,
        vte/core/hip_graph_executor.py:772-789)."""
        if self._io_graph_exec is not None or not self.use_graph:
            return
        self._require_open(staging=True)
        if self._copy_fn is None:                         # before the capture begins
            self._copy_fn = self.codegen.load_kernel_safe(self.hip, 'decode_attention', self.hip.get_gpu_architecture(),
                                                          'vteb_stage_copy_kernel')[1]
        one = self._choose_route() or self._serves_one_launch()
        self.hip.programmatic_launch = self.programmatic
        try:
            self._io_graph_exec, _, self._io_kept = self._capture(lambda: self._record_io(one_launch=one))
            if self._route_pays_to < self.S:
                self._plain_io_graph_exec, _, _ = self._capture(lambda: self._record_io(plain=True))
        finally:
            self.hip.programmatic_launch = False

    def _mirror(self):
        """Where the one launch of a step stores outputs and status for the host, or None where a copy has to bring them: with a
        launch list per layer, outputs large enough for a copy node, or a mapping that has them elsewhere.  28 layers of 32,768
        positions, queries from the host, with a copy launch / without: 176 / 170 us.  (Q taken from pinned memory by the CTAs
        that need it, without the copy in front: 186.)"""
        own = all(self.tensor_mapping.get(f'blk.{l}.attention.output') == self.out_all.ptr + l * self.out_bytes for l in range(self.L))
        if self._step is None or not own or self._out_tail > STAGE_COPY_MAX_BYTES or self.per_layer_hook is not None or self.launch_rewriter is not None:
            return None
        return self._stage_out.value, self._stage_out.value + self._out_tail + 4

    def _record_io(self, plain: bool = False, one_launch: Optional[list] = None):
        if max(self._q_tail, self._out_tail) <= STAGE_COPY_MAX_BYTES:
            mirror = self._mirror() if one_launch else None
            self._stage_copy(self.q_all.ptr, self._stage_q.value, self._q_tail + 4 * self.B, first=True)
            self._record_all(after_copy=True, plain=plain, one_launch=one_launch, mirror=mirror)
            if not mirror:
                self._stage_copy(self._stage_out.value, self.out_all.ptr, self._out_tail + 16)
        else:
            self.hip.memcpy_h2d_async(ctypes.c_void_p(self.q_all.ptr), self._stage_q, self._q_tail + 4 * self.B,
                                      "q and kv offsets staging")
            self._record_all(plain=plain, one_launch=one_launch)
            self.hip.memcpy_d2h_async(self._stage_out, ctypes.c_void_p(self.out_all.ptr), self._out_tail + 16,
                                      "attention output and status word")

    def _wait_for_staging(self):
        """The pinned Q staging may be rewritten only after the previous step's asynchronous copy has read it (a step
        enqueued with `read_output=False` returns before it ran)."""
        if self._stage_in_flight:
            self.hip.event_synchronize(self._stage_event)
            self._stage_in_flight = False

    def _mark_staging_copied(self):
        if self._stage_event is None:
            self._stage_event = self.hip.event_create()
        self.hip.event_record(self._stage_event)
        self._stage_in_flight = True

    def _checked_offsets(self, kv_offsets: np.ndarray):
        """(int32[B] offsets, the largest of them)"""
        off = np.ascontiguousarray(kv_offsets, dtype=np.int32)
        if off.shape != (self.B,):
            raise CudaSafetyError(f"kv_offsets shape {off.shape} != ({self.B},)")
        newest = int(off.max())
        if off.min() < 0 or newest >= self.S:
            raise CudaSafetyError(f"kv offset outside 0..{self.S - 1}")
        return off, newest

    def _leaves(self, names: Optional[dict]):
        """After a step: the names that its partials can be had with, None where they are in the partial buffers."""
        self._kept_names, self._partials_due = names, names is not None

    def _launch_with_offsets(self, off: np.ndarray):
        """A step of one launch, its offsets among the launch's arguments: neither a copy in front of the launch nor a graph around
        it.  us a step, a copy and a graph / this: 28 layers of one sequence of 1,531 positions 20.5 / 16.1, of 11,003 58.4 / 55.6,
        eight layers of 24,001 of 256-wide heads 74.7 / 71.9, of eight sequences of 32 heads on 2 55.0 / 51.7."""
        for offsets, launch in self._direct:
            ctypes.memmove(offsets, off.ctypes.data, off.nbytes)
            launch()
        self._leaves(self._graph_kept)

    def _update_staging_buffers(self, kv_offsets: np.ndarray):
        off, newest = self._checked_offsets(kv_offsets)
        if self._plain_graph_exec is not None:
            self._pick(off, newest)
        half, slot = divmod(self._offset_slot, OFFSET_SLOTS // 2)
        if slot == 0 and self._offset_events[half] is not None:
            self.hip.event_synchronize(self._offset_events[half])
        stage = ctypes.c_void_p(self._offset_ring.value + self._offset_slot * _round_up(4 * self.B, 256))
        ctypes.memmove(stage.value, off.ctypes.data, off.nbytes)
        self.hip.memcpy_h2d_async(ctypes.c_void_p(self.offsets.ptr), stage, off.nbytes, "kv_offsets")
        if slot == OFFSET_SLOTS // 2 - 1:
            if self._offset_events[half] is None:
                self._offset_events[half] = self.hip.event_create()
            self.hip.event_record(self._offset_events[half])
        self._offset_slot = (self._offset_slot + 1) % OFFSET_SLOTS

    def launch_step(self):
        """Enqueue one decode step (no host synchronisation)."""
        if self._closed:
            self._require_open()
        if self._graph_exec is not None:
            self.hip.graph_launch(self._graph_exec if self._on_route else self._plain_graph_exec)
            self._leaves(self._graph_kept if self._on_route else None)
        else:
            self.hip.programmatic_launch, self._kept_names = self.programmatic, None
            try:
                self._record_all(one_launch=self._serves_one_launch())
                self._leaves(self._kept_names)
            finally:
                self.hip.programmatic_launch = False

    def execute_decode_batch(self, kv_offsets: np.ndarray, q_host: Optional[np.ndarray] = None,
                             read_output: bool = True) -> Optional[np.ndarray]:
        """One decode step end to end: stage offsets (and, when given, every layer's
        Q [L,B,Hq,D] fp16) host -> device, replay the graph, read every layer's
        output back.  Returns [L,B,Hq,D] (fp32 or fp16)."""
        if self._closed:
            self._require_open(staging=True)
        self.build_decode_graph()
        nbytes = self.L * self.out_bytes
        if q_host is not None and read_output and self.use_graph:
            # the whole step as one graph launch
            self.build_io_graph()
            off = np.ascontiguousarray(kv_offsets, dtype=np.int32)
            if off.shape != (self.B,):
                raise CudaSafetyError(f"kv_offsets must be int32[{self.B}] within 0..{self.S - 1}")
            qh = np.ascontiguousarray(q_host, dtype=np.float16)
            if qh.nbytes != self.L * self.q_bytes:
                raise CudaSafetyError("q_host must be [L, B, Hq, D] fp16")
            self._wait_for_staging()
            if self._plain_io_graph_exec is not None:  # refused offsets pick nothing
                self._pick(*self._checked_offsets(off))
            if self._host_step is None:
                self._host_step = HostStep(self._stage_offsets.value, self._stage_q.value, self._stage_out.value, self._stage_out.value + self._out_tail + 4,
                                           self.L * self.q_bytes, nbytes, self.B, self.S)
            out = np.empty((self.L, self.B, self.Hq, self.D + 2 if self.emit_state else self.D),
                           dtype=np.float32 if (self.output_f32 or self.emit_state) else np.float16)
            # staging, graph, wait and the copy of the outputs, in one call
            done = self.hip.host_step(self._host_step, self._io_graph_exec if self._on_route else self._plain_io_graph_exec,
                                      off.ctypes.data, qh.ctypes.data, out.ctypes.data)
            self._leaves(self._io_kept if self._on_route else None)
            if not done:                              # the status word travelled with the outputs
                self.dispatcher_check()
                return self._output_array(nbytes)
            return out
        else:
            off = self._checked_offsets(kv_offsets)[0] if self._direct else self._update_staging_buffers(kv_offsets)
            if q_host is not None:
                qh = np.ascontiguousarray(q_host, dtype=np.float16)
                if qh.nbytes != self.L * self.q_bytes:
                    raise CudaSafetyError("q_host must be [L, B, Hq, D] fp16")
                self._wait_for_staging()
                ctypes.memmove(self._stage_q.value, qh.ctypes.data, qh.nbytes)
                self.hip.memcpy_h2d_async(ctypes.c_void_p(self.q_all.ptr), self._stage_q, qh.nbytes, "q staging")
                self._mark_staging_copied()
            if self._direct:
                self._launch_with_offsets(off)
            else:
                self.launch_step()
            if not read_output:
                return None
            self.hip.memcpy_d2h_async(self._stage_out, ctypes.c_void_p(self.out_all.ptr), nbytes, "attention output")
            self.hip.stream_synchronize()
        self.dispatcher_check()
        return self._output_array(nbytes)

    def _output_array(self, nbytes: int) -> np.ndarray:
        dt = np.float32 if (self.output_f32 or self.emit_state) else np.float16
        flat = np.frombuffer((ctypes.c_char * nbytes).from_address(self._stage_out.value), dtype=dt)
        return flat.reshape(self.L, self.B, self.Hq, self.D + 2 if self.emit_state else self.D).copy()

    execute_decode = execute_decode_batch

    def dispatcher_check(self):
        """Raise if a split kernel reported a timed-out wait."""
        if self.dispatcher.work_ptr and hasattr(self.hip, "check_status"):
            self.hip.check_status(ctypes.c_void_p(self.dispatcher.work_ptr))

    def _fill_partials(self):
        """Where the last step took a route without partials: its last layer's split launch, now, on the Q and offsets that
        the step left a copy of.  The layer's caches have to be the step's still."""
        if not self._partials_due:
            return
        self._partials_due = False
        d, ci, vp = self.dispatcher, ctypes.c_int, ctypes.c_void_p
        names = {**self._kept_names, f'blk.{self.L - 1}.q_proj.output': self._kept.ptr}
        fn, args, grid, block, smem = d.build_launches(self.L - 1, names, self._kept.ptr + _round_up(self.q_bytes, 256),
                                                       batch=self.B)[0 if d.fuse_append else 1]
        if len(args) > 13:                            # not the reference-geometry kernels
            args[15] = ci(args[15].value & ~FLAG_DIRECT_OUTPUT)
            args[21], args[22] = vp(0), ci(0)         # partials, no output
            if d.fuse_append:
                args[-2:] = [vp(0), vp(0)]            # the step has appended its row
        # the ticket is zero only behind a combine launch
        self.hip.memset_async(vp(d.work_ptr), 4, 0, "work ticket")
        self.hip.launch_kernel_recorded(fn, args, grid, block, smem)
        self.hip.memset_async(vp(d.work_ptr), 4, 0, "work ticket")
        self.hip.stream_synchronize()
        self.dispatcher_check()

    def read_partials(self):
        """(partial_m, partial_l [B,Hq,C], partial_o [B,Hq,C,D]) of the last layer of the last step.  Cache rows that the step
        read must not have been overwritten since by anything but this executor's own upload and fill methods."""
        self._fill_partials()
        pm, pl, po = self.dispatcher.partial_buffers
        C = self.dispatcher.max_chunks
        m = np.empty((self.B, self.Hq, C), dtype=np.float32)
        l = np.empty_like(m)
        o = np.empty((self.B, self.Hq, C, self.D), dtype=np.float32)
        self.hip.safe_memcpy_device_to_host(m, ctypes.c_void_p(pm.ptr), "partial output m")
        self.hip.safe_memcpy_device_to_host(l, ctypes.c_void_p(pl.ptr), "partial output l")
        self.hip.safe_memcpy_device_to_host(o, ctypes.c_void_p(po.ptr), "partial output o")
        return m, l, o

    def cleanup(self):
        self._closed = True
        self._direct, self._host_step = [], None          # launches on device memory and staging memory that go below
        if self._stage_event is not None:
            self.hip.event_destroy(self._stage_event)
            self._stage_event = None
            self._stage_in_flight = False
        if self._graph_exec is not None:
            self.hip.graph_exec_destroy(self._graph_exec)
            self._graph_exec = None
        if self._io_graph_exec is not None:
            self.hip.graph_exec_destroy(self._io_graph_exec)
            self._io_graph_exec = None
        for graph_exec in (self._plain_graph_exec, self._plain_io_graph_exec):
            if graph_exec is not None:
                self.hip.graph_exec_destroy(graph_exec)
        self._plain_graph_exec = self._plain_io_graph_exec = None
        for i, event in enumerate(self._offset_events):
            if event is not None:
                self.hip.event_synchronize(event)
                self.hip.event_destroy(event)
                self._offset_events[i] = None
        for p in (self._stage_q, self._stage_out, self._offset_ring):
            if p is not None and p.value:
                self.hip.host_free(p)
        self._stage_offsets = self._stage_q = self._stage_out = self._offset_ring = None
        if self._owns_allocator:
            self.allocator.cleanup()
