"""A captured decode step as one launch over all its layers (csrc/kernels/step_decode.cuh).

An executor's step gets every layer's projections before it starts: `execute_decode_batch` is handed Q of all layers at once,
or finds the projections in the step's buffers.  Where nothing that one layer writes is read by another, the layers are as
independent of one another as the sequences of a batch, and the positions of all of them are shared out over the GPU together.
A step with work between its layers (`per_layer_hook`, `launch_rewriter`), with layers that share a cache which they append
to, or with a mapping that hands one layer's output to another keeps a launch list per layer.
"""
from __future__ import annotations

import ctypes
import math

from ..bridge.cuda_runtime import StepArgs, StepLayer
from ..bridge.errors import CudaSafetyError
from ..bridge.memory import MemoryRegion


class StepRoute:
    """The launches of a whole step: one for every 64 layers."""

    def __init__(self, dispatcher, allocator, n_layers: int, append: bool, hg: int = 0):
        d = self.d = dispatcher
        self.layers, self.append, self.ctas = int(n_layers), bool(append), d.num_sms
        self.plan = d.hip.step_plan(d.num_q_heads, d.num_kv_heads, d.head_dim, d.batch_size, self.ctas, hg)
        if not self.plan.ok:
            raise CudaSafetyError("one launch for all layers does not cover this geometry or batch")
        self.name = f"vteb_decode_step_{'2_' if d.num_q_heads > 8 * d.num_kv_heads else ''}d{d.head_dim}_kernel"
        self.function = d.codegen.load_kernel_safe(d.hip, 'decode_attention', d.hip.get_gpu_architecture(), self.name)[1]
        # the boards on which CTAs leave their state of a run that goes on in the next one's share, then every CTA's count of launches
        boards = (self.plan.state_bytes + 255) // 256 * 256
        self.scratch = allocator.allocate(boards + 4 * self.ctas, "attn_step_boards", MemoryRegion.SCRATCH)
        self.launch_counts = self.scratch.ptr + boards
        d.hip.safe_memset(ctypes.c_void_p(self.scratch.ptr), boards + 4 * self.ctas, "attn_step_boards")

    def _layer(self, layer: int, mapping: dict):
        """(q, K cache, V cache, new K, new V, output) of a layer."""
        d = self.d
        ptr = lambda name: d._resolve_ptr(mapping, f'blk.{layer}.{name}')
        new = (ptr('k_proj.output'), ptr('v_proj.output')) if self.append else (0, 0)
        if self.append and not all(new):                   # null means to the kernel that the row is in the cache already
            raise CudaSafetyError(f"layer {layer}: the new K / V rows could not be resolved (null)")
        return (ptr('q_proj.output'), *d._resolve_kv_cache_ptrs(layer, mapping), *new, ptr('attention.output'))

    def resolve(self, mapping: dict) -> list:
        """What every layer reads and writes."""
        return [self._layer(layer, mapping) for layer in range(self.layers)]

    def serves(self, mapping: dict, kv_offset_ptr: int, batch: int, layers: list | None = None) -> bool:
        """Whether the layers of a mapping may run side by side: pointers that 16-byte accesses can take, and nothing that
        one part of the step writes overlaps with anything else in it."""
        d = self.d
        stride = int(mapping.get('kv_batch_stride_elements', 0))
        row = d.num_kv_heads * d.head_dim * 2
        q_bytes, new_bytes, cache_bytes = batch * d.num_q_heads * d.head_dim * 2, batch * row, ((batch - 1) * stride * 2 + d.context_length * row)
        spans = {(kv_offset_ptr, kv_offset_ptr + 4 * batch, False), (self.scratch.ptr, self.scratch.ptr + self.scratch.size, True)}
        sizes = (q_bytes, cache_bytes, cache_bytes, new_bytes, new_bytes, q_bytes * (2 if d.output_f32 else 1))
        written = (False, self.append, self.append, False, False, True)
        if stride % (row // 2) or stride < d.context_length * (row // 2):     # the caches are read as whole position rows
            return False
        writes = 1
        for pointers in self.resolve(mapping) if layers is None else layers:
            d._validate(batch, *(pointers[i] for i in (0, 1, 2, 5)), kv_offset_ptr, stride)
            if any(p % 16 for p in pointers):
                return False
            spans.update((p, p + n, w) for p, n, w in zip(pointers, sizes, written) if p)
            writes += sum(written)
        if d.fuse_rope:
            width = d.rotary_dim if d.rope_type == 2 else d.head_dim
            spans.update((a.value, a.value + 2 * width * d.context_length, False) for a in d._rope_arguments(mapping)[:2])
        if sum(w for _, _, w in spans) != writes:          # two writers of one place
            return False
        end_read = end_written = 0
        for lo, hi, w in sorted(spans):
            if lo < end_written or (w and lo < end_read):
                return False
            end_read, end_written = max(end_read, hi), max(end_written, hi if w else 0)
        return True

    def launches(self, mapping: dict, kv_offset_ptr: int, batch: int, layers: list, keep: tuple, host: tuple | None = None):
        """`layers`: what `resolve` found.  `keep`: where the last layer leaves a copy of its Q and of the offsets, from which its partials can be had.  `host`:
        pinned memory (outputs, one layer's after another's, and status word) that the kernel stores to as well."""
        d = self.d
        attention_scale = d.metadata.get('attention_scale')
        row = d.num_kv_heads * d.head_dim
        row_out = d.num_q_heads * d.head_dim * (4 if d.output_f32 else 2)
        # as far as `serves` has looked: the last sequence's room, not its stride, ends what a tile may read
        n_rows = int(mapping['kv_batch_stride_elements']) // row * (batch - 1) + d.context_length
        out = []
        for first in range(0, self.layers, self.plan.max_layers):
            n = min(self.plan.max_layers, self.layers - first)
            a = StepArgs()
            for i in range(n):
                q, k_cache, v_cache, k_new, v_new, output = layers[first + i]
                maps = (d.hip.kv_tensor_map(p, n_rows, row, self.plan.tile, self.plan.hg * d.head_dim // 64) for p in (k_cache, v_cache))
                a.layer[i] = StepLayer(*maps, q, k_cache, v_cache, k_new, v_new, output)
                if host:
                    a.layer[i].mirror = host[0] + (first + i) * batch * row_out
            a.kv_offsets, a.boards, a.launches, a.status = kv_offset_ptr, self.scratch.ptr, self.launch_counts, d.work_ptr + 4
            if host:
                a.status_mirror = host[1]
            a.keep_q, a.keep_offsets = keep
            a.keep_layer = n - 1 if first + n == self.layers else -1
            a.num_layers, a.batch, a.num_q_heads, a.num_kv_heads = n, batch, d.num_q_heads, d.num_kv_heads
            a.hg, a.hg_log2, a.wph, a.group = self.plan.hg, self.plan.hg_log2, self.plan.wph, d.num_q_heads // d.num_kv_heads
            a.groups, a.group_inv, a.fan = d.num_kv_heads // a.hg, -(-65536 // a.group), self.plan.fan
            a.kv_batch_stride, a.out_kind = int(mapping.get('kv_batch_stride_elements', 0)), 2 if d.output_f32 else 1
            a.rope_type = -1
            if d.fuse_rope:
                a.rope_cos, a.rope_sin, a.rope_type, a.rotary_dim = (x.value for x in d._rope_arguments(mapping))
            a.scale = float(attention_scale) if attention_scale else 1.0 / math.sqrt(d.head_dim)
            out.append((self.function, [a], (self.ctas, 1, 1), (self.plan.threads, 1, 1), self.plan.smem_bytes))
        return out


ONE_LAUNCH_BYTES = 600e6            # K and V of a step from which it pays with two layers too
# Share of a cache's room that sizes are judged by where lengths are not known yet: what the caches of the measured steps hold, one
# sequence and a batch of unequal ones.  Only `large` below depends on it, not whether four layers and more are one launch.
IN_USE_ALONE, IN_USE_BATCH = 0.72, 0.5


def one_launch_pays(d, layers: int) -> bool:
    """Whether a step of `layers` layers goes to one launch rather than to a launch list per layer, by sizes that do not change.

    us a step behind a flushed L2, append included, launches per layer / one launch, over 7 head geometries, 1 to 64 sequences, room for
    300 to 262,144 positions, 1 to 100 % of it in use; 448 sizes for each count of layers (252 for six), fill by fill:
      six 1.10 to 5.0 times as fast (mean 1.99), five 0.96 to 3.8 (1.58), four 0.96 to 3.3 (1.44): always.  Below 1 are 2 % of four and 1 % of
        five layers: 64 sequences of 300 of 32 heads on 2 of 128 half full 51 / 53, 64 of 8,192 of 8 heads on 8 half full 484 / 501;
      three 0.80 to 3.0 (1.26): batches of four and more with groups of up to eight, 0.91 to 3.0 (64 of 300 of 12 heads on 2 half full
        21 / 23, 16 of 32,768 of 8 on 8 1 % full 33 / 35); two or three sequences 0.86, one 0.80, wider groups 0.80;
      two 0.62 to 2.6 (1.07): not, but for large steps of heads wider than 64: 0.89 to 1.5 (8 heads on 8, 16 of 32,768 1 % full 24 / 26,
        half full 273 / 260), one sequence of 256-wide heads 0.93 to 1.0 and so not.
    One layer has nothing to share out that the launches per layer do not: 0.5 to 1.06.  Large steps of two or three layers of 64-wide
    heads gain nothing for sure: their arithmetic keeps up with HBM at full clocks only (64 ragged sequences of 32 heads on 8, two
    layers: 345 / 338 us on one machine, 353 / 364 on another)."""
    plan = d.hip.step_plan(d.num_q_heads, d.num_kv_heads, d.head_dim, d.batch_size, d.num_sms)
    if not plan.ok or layers < 2:
        return False
    if layers >= 4:
        return True
    in_use = IN_USE_ALONE if d.batch_size == 1 else IN_USE_BATCH
    large = layers * d.batch_size * d.context_length * d.num_kv_heads * d.head_dim * 4 * in_use >= ONE_LAUNCH_BYTES
    if large:
        return d.head_dim > 64 and not (layers == 2 and d.batch_size == 1 and d.head_dim == 256)
    return layers == 3 and d.batch_size >= 4 and d.num_q_heads <= 8 * d.num_kv_heads
