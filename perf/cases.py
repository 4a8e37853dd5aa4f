"""The decode-attention work this package is used for, as measurable cases.

Four ways in, all public:

  host     `DecodeAttentionExecutor.execute_decode_batch(offsets, q)`: a decode step whose queries come from the
           host and whose outputs go back there.
  step     `execute_decode_batch(offsets, read_output=False)`: a decode step inside a program that keeps its
           activations on the device; projections are in the step's buffers, outputs stay on the device.
  call     `CudaRuntime.kv_cache_append` + `CudaRuntime.split_kv_decode`: one layer at a time through the C ABI, with
           the caller's own tensors and scratch and no graph, as a plugin calls it.
  unsplit  `flash_attention_kernel` under its reference name and launch geometry, one launch per layer in a captured
           graph, as the reference's batched executor records it.

A step's route says what it contains: "attend" (the row of the newest position is in the cache already), "append"
(append launch, then attention), "rope" (the append rotates K, the split kernel rotates Q), "rope_append" (rotation
and append inside the split kernel).  Caches hold `capacity` positions per sequence; the sequences' lengths lie in
[ctx_min, ctx_max] and follow from the case alone.
"""
import ctypes
import math

import numpy as np
import torch

from vte_b200.bridge import CudaRuntime
from vte_b200.bridge.cuda_runtime import ATTN_BALANCED, ATTN_COMPACT, ATTN_COMPAT, ATTN_PROGRAMMATIC
from vte_b200.compiler import CodegenEngine
from vte_b200.core.decode_executor import DecodeAttentionExecutor
from vte_b200.core.split_kv_attention import balanced_split_count, choose_split_count


def _case(name, mode, batch, heads, capacity, ctx_min, ctx_max, layers, route="attend", f32=True, rotary_dim=0,
          sigma=1.0, outliers=False):
    q_heads, kv_heads, head_dim = heads
    c = {"mode": mode, "batch": batch, "q_heads": q_heads, "kv_heads": kv_heads, "head_dim": head_dim,
         "capacity": capacity, "ctx_min": ctx_min, "ctx_max": ctx_max, "layers": layers, "route": route, "f32": f32,
         "rotary_dim": rotary_dim, "sigma": sigma, "outliers": outliers}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call there is: one layer, one sequence, half a thousand positions, from the host and back
        _case("host_one_layer_512", "host", 1, (12, 2, 128), 512, 512, 512, 1),
        # an ordinary chat: a cache with room for 4,096 positions, about a third of it in use, projections on the
        # device, the append as a launch of its own; fp16 outputs for the next projection
        _case("chat_28_layers_1531", "step", 1, (12, 2, 128), 4096, 1531, 1531, 28, "append", f32=False),
        # a long document, rotation and append folded into the attention launches; an odd length
        _case("document_28_layers_11003", "step", 1, (12, 2, 128), 16384, 11003, 11003, 28, "rope_append"),
        # the headline configuration end to end: 32,768 positions, 28 layers, queries from the host, outputs back
        _case("host_28_layers_32k", "host", 1, (12, 2, 128), 32768, 32768, 32768, 28),
        # a serving batch of ragged sequences of 8 x 64-wide heads
        _case("batch64_ragged_64wide", "step", 64, (32, 8, 64), 16384, 1024, 16384, 2),
        # the share of such a batch that one of eight GPUs serves, with the append
        _case("batch8_ragged_64wide", "step", 8, (32, 8, 64), 16384, 1024, 16384, 10, "append", f32=False),
        # ragged long contexts of 256-wide heads with outliers in the caches
        _case("batch16_ragged_256wide", "step", 16, (8, 2, 256), 65536, 2048, 65536, 1, sigma=0.5, outliers=True),
        # one sequence of 256-wide heads of which the first 64 channels are rotated; an odd length
        _case("one_256wide_24001", "step", 1, (8, 2, 256), 32768, 24001, 24001, 8, "rope", rotary_dim=64),
        # the largest: one sequence of a million positions
        _case("million_positions", "step", 1, (12, 2, 128), 1048576, 1048576, 1048576, 4),
        # many query heads on few KV heads (sixteen to one), a small batch
        _case("batch8_group16", "step", 8, (32, 2, 128), 4096, 500, 4096, 8, "append", f32=False),
        # the reference's own batched decode: four sequences, the unsplit kernel for every layer
        _case("unsplit_batch4", "unsplit", 4, (12, 2, 128), 2048, 100, 1500, 28, "append", f32=False),
        # short ragged requests served layer by layer from a program with its own tensors, no graph
        _case("call_batch32_short", "call", 32, (28, 4, 128), 4096, 100, 4000, 1, "append", f32=False),
    ]


#: Head geometries of `draw`: the listed ones and their neighbours (no grouping, groups of 3, 7, 8).
_HEADS = [(12, 2, 128), (12, 2, 128), (32, 8, 64), (32, 8, 64), (8, 2, 256), (8, 2, 256), (28, 4, 128), (12, 4, 128),
          (16, 2, 128), (8, 8, 128), (32, 2, 128)]
_MOST_BYTES = 2.0e9     # cache bytes one drawn pass may read


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    mode = rng.choices(["step", "host", "call", "unsplit"], [5, 2, 2, 1])[0]
    heads = rng.choice(_HEADS)
    position = 4 * heads[1] * heads[2]                      # bytes of one cached position, K and V
    route = rng.choice(["attend", "append", "append", "rope", "rope_append"])
    if mode == "host":
        route = "attend"
    elif mode in ("call", "unsplit"):
        route = "append"
    elif heads[0] // heads[1] > 8 and route.startswith("rope"):
        route = "append"                                    # rotation inside the attention needs groups of at most 8
    rotary = 64 if route.startswith("rope") and heads[2] == 256 else 0
    f32 = mode != "unsplit" and rng.random() < 0.5
    if mode == "unsplit":
        batch, longest = rng.randint(1, 8), _log(rng, 64, 2048)
    elif heads[0] // heads[1] > 8:
        batch, longest = _log(rng, 1, 16), _log(rng, 128, 8192)
    elif mode != "call" and rng.random() < 0.5:
        batch, longest = 1, _log(rng, 128, 524288 if route in ("attend", "append") else 65536)
    else:
        batch, longest = _log(rng, 2, 64), _log(rng, 256, 32768)
    while batch > 1 and batch * longest * position > _MOST_BYTES:
        batch = max(1, batch // 2)
    shortest = longest if batch == 1 else max(1, int(longest * rng.uniform(0.05, 1.0)))
    capacity = longest if rng.random() < 0.3 else min(1048576, _round_up(int(longest * rng.uniform(1.0, 2.5)), 256))
    if mode == "call":
        layers = 1
    else:
        layers = min(28, _log(rng, 1, 28), max(1, int(_MOST_BYTES / (batch * longest * position))))
        layers = min(layers, max(1, int(8e9 / (batch * capacity * position))))
        if mode == "unsplit":
            layers = min(layers, 8)
    return _case(None, mode, batch, heads, capacity, shortest, longest, layers, route, f32, rotary)


def _round_up(x, m):
    return (x + m - 1) // m * m


def _lengths(case):
    """int32[batch] sequence lengths, uniform in [ctx_min, ctx_max]; they depend on the case only."""
    rng = np.random.default_rng([case["batch"], case["ctx_min"], case["ctx_max"]])
    return rng.integers(case["ctx_min"], case["ctx_max"] + 1, size=case["batch"]).astype(np.int32)


_shared = {}


def _runtime():
    """The program's one runtime and kernel loader."""
    if not _shared:
        rt = CudaRuntime(device_index=0)
        rt.initialize()
        _shared["rt"], _shared["codegen"] = rt, CodegenEngine()
    return _shared["rt"], _shared["codegen"]


class _Executor:
    """An executor and its device memory, which outlives every view of it."""

    def __init__(self, *args, **kw):
        self.ex = DecodeAttentionExecutor(*args, **kw)

    def __del__(self):
        if hasattr(self, "ex"):
            self.ex.cleanup()


class _DeviceArray:
    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _view(owner, ptr, shape, dtype):
    """A torch view of an executor's device memory; the tensor holds on to its owner."""
    typestr = {torch.float16: "<f2", torch.float32: "<f4"}[dtype]
    return torch.as_tensor(_DeviceArray(owner, ptr, tuple(shape), typestr), device="cuda")


def _fill_cache(x, case, gen):
    x.normal_(0.0, case["sigma"], generator=gen)
    if case["outliers"]:
        for part in x.view(-1).split(1 << 26):
            part[torch.rand(part.shape, device="cuda", generator=gen) < 0.01] *= 20.0


class _State:
    """What a program holds between steps."""
    graph = None

    def __del__(self):
        if self.graph is not None:
            _shared["rt"].graph_exec_destroy(self.graph)


def prepare(case, seed):
    rt, codegen = _runtime()
    s = _State()
    s.mode, s.rt = case["mode"], rt
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s.lengths = _lengths(case)
    s.offsets = s.lengths - 1
    (_prepare_executor if s.mode in ("host", "step") else _prepare_tensors)(s, case, gen, seed, rt, codegen)
    torch.cuda.synchronize()
    return s


def _prepare_executor(s, case, gen, seed, rt, codegen):
    B, Hq, Hkv, D, L = case["batch"], case["q_heads"], case["kv_heads"], case["head_dim"], case["layers"]
    meta = {"attention.head_count": Hq, "attention.head_count_kv": Hkv, "attention.key_length": D}
    if case["rotary_dim"]:
        meta.update(rope_type=2, rotary_dim=case["rotary_dim"])
    route = case["route"]
    owner = _Executor(rt, codegen, meta, B, case["capacity"], L, output_f32=case["f32"], with_append=(route == "append"),
                      rope={"rope": "fused", "rope_append": "fused-append"}.get(route, "off"))
    s.owner = owner
    s.executor = ex = owner.ex
    rows = []
    for i in range(ex.n_kv):
        for cache in (ex.k_cache[i], ex.v_cache[i]):
            x = _view(owner, cache.ptr, (B, case["capacity"], Hkv, D), torch.float16)
            _fill_cache(x, case, gen)
            rows += [x[b, int(s.offsets[b])] for b in range(B)]
    if s.mode == "host":
        s.q = np.random.default_rng(seed).standard_normal((L, B, Hq, D), dtype=np.float32).astype(np.float16)
        ex.build_io_graph()
        return
    _view(owner, ex.q_all.ptr, (L, B, Hq, D), torch.float16).normal_(generator=gen)
    _view(owner, ex.knew_all.ptr, (L, B, Hkv, D), torch.float16).normal_(generator=gen)
    _view(owner, ex.vnew_all.ptr, (L, B, Hkv, D), torch.float16).normal_(generator=gen)
    s.out = [_view(owner, ex.out_all.ptr, (L, B, Hq, D), torch.float32 if case["f32"] else torch.float16)]
    if route != "attend":
        s.out += rows[:60]                      # the newest rows of the caches are written by the step
    ex.build_decode_graph()


def _prepare_tensors(s, case, gen, seed, rt, codegen):
    B, Hq, Hkv, D, L, S = (case[k] for k in ("batch", "q_heads", "kv_heads", "head_dim", "layers", "capacity"))
    dt = torch.float32 if case["f32"] else torch.float16

    def new(*shape):
        return torch.empty(shape, dtype=torch.float16, device="cuda")
    s.layers, rows = [], []
    s.dev_offsets = torch.from_numpy(s.offsets).cuda()
    for _ in range(L):
        q, kn, vn = (new(B, h, D).normal_(generator=gen) for h in (Hq, Hkv, Hkv))
        kc, vc = new(B, S, Hkv, D), new(B, S, Hkv, D)
        _fill_cache(kc, case, gen)
        _fill_cache(vc, case, gen)
        out = torch.zeros(B, Hq, D, dtype=dt, device="cuda")
        s.layers.append((q, kn, vn, kc, vc, out))
        rows += [c[b, int(s.offsets[b])] for c in (kc, vc) for b in range(B)]
    s.out = [layer[5] for layer in s.layers] + rows[:64 - L]
    s.scale, s.stride = 1.0 / math.sqrt(D), S * Hkv * D
    s.dims = (B, Hq, Hkv, D)
    if s.mode == "unsplit":
        _, fn = codegen.load_kernel_safe(rt, "flash_attention", rt.get_gpu_architecture(), "flash_attention_kernel")
        vp, ci, cf = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
        torch.cuda.synchronize()
        rt.stream_begin_capture()
        for q, kn, vn, kc, vc, out in s.layers:
            args = [vp(t.data_ptr()) for t in (q, kn, vn, kc, vc, out)]
            args += [ci(1), ci(Hq), ci(Hkv), ci(D), cf(s.scale), vp(s.dev_offsets.data_ptr()), ci(s.stride)]
            rt.launch_kernel_recorded(fn, args, (B, Hq, 1), (D, 1, 1), 2 * D * 4)
        graph = rt.stream_end_capture()
        s.graph = rt.graph_instantiate(graph)
        rt.graph_destroy(graph)
        return
    # the caller's scratch and its choice of split count and flags, as the header describes them
    fast = Hq // Hkv <= 8
    sms = rt.get_num_cus()
    groups = rt.split_kv_plan(Hq, Hkv, D).n_hgroups if fast else Hkv
    if not fast:
        s.splits, s.flags = choose_split_count(sms, B, groups, S), ATTN_COMPAT
    elif B == 1:
        s.splits, s.flags = choose_split_count(sms, 1, groups, S), ATTN_PROGRAMMATIC | ATTN_COMPACT
    else:
        s.splits, s.flags = balanced_split_count(sms, B, groups), ATTN_PROGRAMMATIC | ATTN_BALANCED
    s.partials = [torch.zeros(B * Hq * s.splits * w, device="cuda") for w in (1, 1, D)]
    s.work = torch.zeros(4, dtype=torch.int32, device="cuda")
    s.f32 = case["f32"]


def run(s):
    if s.mode == "host":
        return s.executor.execute_decode_batch(s.offsets, s.q)
    if s.mode == "step":
        s.executor.execute_decode_batch(s.offsets, read_output=False)
        return s.out
    if s.mode == "unsplit":
        s.rt.graph_launch(s.graph)
        return s.out
    B, Hq, Hkv, D = s.dims
    off = s.dev_offsets.data_ptr()
    pm, pl, po = (t.data_ptr() for t in s.partials)
    for q, kn, vn, kc, vc, out in s.layers:
        s.rt.kv_cache_append(kn.data_ptr(), vn.data_ptr(), kc.data_ptr(), vc.data_ptr(), off, B, Hkv, D, s.stride)
        s.rt.split_kv_decode(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), off, out.data_ptr(), s.f32, pm, pl, po,
                             s.work.data_ptr(), B, Hq, Hkv, D, s.scale, s.stride, s.splits, 0, s.flags)
    return s.out


def work(case):
    """K and V once per KV head, Q in, outputs out, one offset per sequence; new rows in and out where appended."""
    B, Hq, Hkv, D, L = case["batch"], case["q_heads"], case["kv_heads"], case["head_dim"], case["layers"]
    positions = int(_lengths(case).astype(np.int64).sum())
    one = positions * Hkv * D * 4 + B * Hq * D * (2 + (4 if case["f32"] else 2)) + 4 * B
    if case["route"] != "attend":
        one += 2 * B * Hkv * D * (2 + 2) - B * Hkv * D * 4      # the newest row is read from the projections instead
    return {"bytes": L * one, "flops": L * 4 * positions * Hq * D}


def tolerance(case):
    # fp32 sums of fp16 products over up to a million positions; fp16 outputs are rounded once
    return {"rel": 2e-5, "max": 5e-4} if case["f32"] else {"rel": 5e-4, "max": 2e-3}
