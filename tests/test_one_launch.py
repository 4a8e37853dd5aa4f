"""A decode step as one launch over all its layers (core/step_route.py, csrc/kernels/step_decode.cuh): what may take it and
what does, on the CPU, and the kernels against the oracle where tiles, shares and runs meet."""
import ctypes
import re
from types import SimpleNamespace

import numpy as np
import pytest

from oracle import attention_oracle as orc
from tests.test_host_logic import FakeCodegen, FakeRuntime
from tests.test_lean_routes import FakeHip
from vte_b200.bridge.cuda_runtime import CudaRuntime, KvTensorMap, StepArgs, StepLayer, StepPlan, load_library
from vte_b200.bridge.errors import CudaRuntimeError, CudaSafetyError
from vte_b200.bridge.memory import SlabAllocator
from vte_b200.core.decode_executor import DecodeAttentionExecutor
from vte_b200.core.split_kv_attention import SplitKVAttentionDispatcher
from vte_b200.core.step_route import StepRoute, one_launch_pays


def step_plan(Hq, Hkv, D, batch, ctas=148, hg=0):
    plan = StepPlan()
    assert load_library().vteb_step_plan(Hq, Hkv, D, batch, ctas, hg, ctypes.byref(plan)) == 0
    return plan


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("group", [1, 7, 8, 9, 16, 17])
def test_plan_covers_what_the_kernels_do(built_library, group, D):
    assert ctypes.sizeof(StepLayer) == 320 and ctypes.sizeof(StepArgs) == 64 * 320 + 512 < 32764
    for Hkv in (1, 2, 3, 4, 6, 8, 12):
        for batch in (1, 64, 1024, 1025):
            p = step_plan(group * Hkv, Hkv, D, batch)
            assert bool(p.ok) == (group <= (8 if D == 256 else 16) and batch <= 1024)
            if not p.ok:
                continue
            warps = p.threads // 32 - 1
            assert Hkv % p.hg == 0 and p.hg == 1 << p.hg_log2 and p.hg * p.wph == warps // (2 if D == 256 else 1) and p.tile == 16 * p.wph <= 256
            assert (warps * 32) % (D // 8) == 0 and p.smem_bytes <= 227 * 1024
            assert 4 <= p.fan <= 16
            assert p.state_bytes == 148 * p.hg * group * (D // 2 + 1) * 16


def a_route(layers=3, append=True, heads=(12, 2, 128), batch=2, capacity=512, f32=False, **kw):
    """(route, mapping, offsets) over made-up addresses that do not overlap."""
    Hq, Hkv, D = heads
    d = object.__new__(SplitKVAttentionDispatcher)
    vars(d).update(num_q_heads=Hq, num_kv_heads=Hkv, head_dim=D, batch_size=batch, context_length=capacity, output_f32=f32, num_sms=148,
                   fuse_rope=False, rope_type=0, rotary_dim=D, hip=SimpleNamespace(step_plan=step_plan), **kw)
    r = object.__new__(StepRoute)
    vars(r).update(d=d, layers=layers, append=append, scratch=SimpleNamespace(ptr=0x1000, size=0x1000))
    m, at = {'kv_batch_stride_elements': capacity * Hkv * D}, 0x100000
    for l in range(layers):
        for name, size in (('q_proj.output', batch * Hq * D * 2), ('k_proj.output', batch * Hkv * D * 2), ('v_proj.output', batch * Hkv * D * 2),
                           ('kv_cache.k', batch * capacity * Hkv * D * 2), ('kv_cache.v', batch * capacity * Hkv * D * 2),
                           ('attention.output', batch * Hq * D * (4 if f32 else 2))):
            m[f'blk.{l}.{name}'] = at
            at += size                                           # back to back: what touches does not overlap
    return r, m, at


def test_layers_run_side_by_side_only_where_none_reads_what_another_writes(built_library):
    for append in (True, False):
        r, m, free = a_route(append=append)
        may = lambda **change: r.serves({**m, **{k.replace('__', '.'): v for k, v in change.items()}}, free, 2)
        assert may()
        assert not may(blk__1__q_proj__output=m['blk.0.attention.output'])                 # one layer's output is the next one's Q
        assert not may(blk__1__q_proj__output=m['blk.0.attention.output'] + 16)
        assert not may(blk__2__attention__output=m['blk.0.attention.output'])               # two writers
        assert not may(blk__2__attention__output=m['blk.2.q_proj.output'])                  # in place
        assert may(blk__2__q_proj__output=m['blk.0.q_proj.output'])                         # read twice
        assert may(blk__2__kv_cache__k=m['blk.0.kv_cache.k']) != append                     # a shared cache: read only
        assert not may(blk__2__kv_cache__k=m['blk.0.kv_cache.k'] + 1024) == append
        assert not may(blk__2__attention__output=free + 0x10008) and may(blk__2__attention__output=free + 0x10010)      # 16-byte stores
        assert may(blk__1__v_proj__output=free + 0x10008) != append
        assert not may(blk__0__attention__output=0x1800)                                    # the route's own scratch
        assert r.serves({**m, 'kv_batch_stride_elements': 512 * 256}, free, 2)
        for stride in (512 * 256 + 128, 511 * 256):                                          # no whole rows; shorter than the cache
            assert not r.serves({**m, 'kv_batch_stride_elements': stride}, free, 2)
        assert not r.serves(m, m['blk.1.attention.output'] + 64, 2)                          # offsets under an output
    with pytest.raises(CudaSafetyError, match="null"):
        r, m, free = a_route()
        r.serves({k: v for k, v in m.items() if k != 'blk.1.v_proj.output'}, free, 2)


def test_what_goes_to_one_launch(built_library):
    pays = lambda layers, *a: one_launch_pays(a_route(1, True, *a)[0].d, layers)
    assert pays(28, (12, 2, 128), 1, 4096) and pays(4, (16, 1, 64), 1, 64) and pays(4, (32, 2, 128), 1, 4096)
    assert pays(3, (8, 2, 256), 8, 4096) and not pays(3, (8, 2, 256), 1, 4096) and not pays(3, (32, 2, 128), 8, 4096)
    assert pays(2, (8, 8, 128), 64, 16384) and pays(3, (32, 8, 64), 8, 4096)
    assert not pays(2, (32, 8, 64), 64, 16384) and not pays(3, (32, 8, 64), 64, 16384) and not pays(2, (8, 8, 128), 8, 4096)
    assert not pays(1, (12, 2, 128), 1, 1 << 20)                   # one layer: nothing to share out
    assert not pays(28, (36, 2, 128), 1, 4096) and not pays(28, (18, 2, 256), 1, 4096) and not pays(28, (12, 2, 128), 1025, 64)


def test_few_layers_go_to_one_launch_only_where_none_of_their_lengths_loses_much(built_library):
    """Choices are made for the caches' room, before lengths are known: two or three sequences of three layers, and one of
    256-wide heads with two, were up to a seventh slower than the launches per layer for some or all lengths."""
    pays = lambda layers, *a: one_launch_pays(a_route(1, True, *a)[0].d, layers)
    assert not pays(2, (8, 2, 256), 1, 262144) and pays(2, (8, 2, 256), 16, 32768) and pays(3, (8, 2, 256), 1, 262144)
    for heads in ((8, 2, 256), (32, 8, 64), (12, 2, 128)):
        assert not pays(3, heads, 2, 4096) and not pays(3, heads, 3, 4096) and pays(3, heads, 4, 4096)
    assert pays(4, (32, 2, 128), 1, 8192) and pays(4, (8, 2, 256), 2, 4096)


class HostOnly(FakeRuntime, FakeHip):
    """A runtime whose launches are names in a list: nothing is dereferenced but pinned memory."""
    step_plan, programmatic_launch = staticmethod(step_plan), False

    def __init__(self):
        super().__init__()
        self.log, self.recording, self.maps, self.pinned = [], None, [], []

    def _names(self, launches): return [self.loaded[fn.value - 0x1001][1] for fn, *_ in launches]
    def launched(self):
        names, self.log = self._names(self.log), []
        return names
    def get_real_mem_info(self): return 180 << 30, 180 << 30
    def host_alloc(self, n):
        self.pinned.append(ctypes.create_string_buffer(n))
        return ctypes.c_void_p(ctypes.addressof(self.pinned[-1]))
    def stream_begin_capture(self): self.recording = []
    def stream_end_capture(self):
        graph, self.recording = self.recording, None
        return graph
    def launch_kernel_recorded(self, *launch): (self.log if self.recording is None else self.recording).append(launch)
    def graph_instantiate(self, graph): return graph
    def graph_launch(self, graph): self.log += graph
    def prepare_launch(self, *launch): return lambda: self.log.append(launch[:5])
    def host_step(self, step, graph, offsets, q, out):
        if not all(0 <= x < step.capacity for x in (ctypes.c_int * step.batch).from_address(offsets)):
            raise CudaSafetyError("kv_offsets out of range")
        self.log += graph
        return True
    def kv_tensor_map(self, ptr, n_rows, row_halves, box_rows, box_cols=0):
        self.maps.append((ptr, n_rows, row_halves))
        return KvTensorMap()
    def event_create(self): return ctypes.c_void_p(1)
    def _nothing(self, *a, **kw): return True
    graph_destroy = graph_exec_destroy = host_free = stream_synchronize = check_status = event_record = event_synchronize = _nothing
    event_destroy = memcpy_h2d_async = memcpy_d2h_async = memset_async = safe_memcpy_host_to_device = safe_memcpy_device_to_host = _nothing


def host_only(B=1, S=4096, L=4, heads=(12, 2, 128), **kw):
    rt = HostOnly()
    meta = {"attention.head_count": heads[0], "attention.head_count_kv": heads[1], "attention.key_length": heads[2]}
    return DecodeAttentionExecutor(rt, FakeCodegen(), meta, B, S, L, **kw), rt


@pytest.mark.parametrize("option", [dict(lean=(4, 1)), dict(lean=(0, 0)), dict(compat=True), dict(strict_empty_splits=True), dict(emit_state=True),
                                    dict(num_splits=8), dict(use_graph=False), dict(fused_combine=True), dict(balanced=True), dict(wide=False),
                                    dict(variant="full"), dict(min_chunk=64), dict(tensor_maps=False), dict(prefetch_next_layer=False)], ids=str)
def test_one_launch_refuses_what_it_would_drop(built_library, option):
    with pytest.raises(CudaSafetyError, match="one launch for all layers"):
        host_only(one_launch=True, **option)
    for fine in (dict(one_launch=True), option if "lean" not in option else dict(lean=(0, 0)), dict(one_launch=False, **option)):
        ex, rt = host_only(**fine)                                     # by itself neither is
        ex.execute_decode_batch(np.array([100], dtype=np.int32), read_output=False)
        assert (rt.launched() == ["vteb_decode_step_d128_kernel"]) == (fine == dict(one_launch=True))


@pytest.mark.parametrize("late", [dict(rope="separate"), dict(per_layer_hook=lambda layer: 0), dict(n_kv_buffers=2, with_append=True)], ids=str)
def test_one_launch_refuses_what_it_cannot_keep_in_order(built_library, late):
    ex, rt = host_only(one_launch=True, **late)
    with pytest.raises(CudaSafetyError, match="one launch for all layers"):
        ex.build_decode_graph()
    assert rt.launched() == []


def test_nothing_is_launched_after_cleanup(built_library):
    """The device memory of an executor with an allocator of its own is gone by then; the staging memory is in any case."""
    off, q = np.array([100], dtype=np.int32), np.zeros((4, 1, 12, 128), dtype=np.float16)
    ex, rt = host_only()
    ex.execute_decode_batch(off, read_output=False)
    ex.execute_decode_batch(off, q)
    assert rt.launched() == ["vteb_decode_step_d128_kernel", "vteb_stage_copy_kernel", "vteb_decode_step_d128_kernel"]
    ex.cleanup()
    for call in (lambda: ex.execute_decode_batch(off, read_output=False), lambda: ex.execute_decode_batch(off), lambda: ex.execute_decode_batch(off, q),
                 ex.launch_step, ex.build_decode_graph, ex.build_io_graph):
        with pytest.raises(CudaSafetyError, match="cleaned up"):
            call()
    assert rt.launched() == []
    rt = HostOnly()                                                    # a caller's allocator outlives the executor
    allocator = SlabAllocator(rt, 180 << 30, requested_pool_size=1 << 30)
    allocator.initialize()
    meta = {"attention.head_count": 12, "attention.head_count_kv": 2, "attention.key_length": 128}
    ex = DecodeAttentionExecutor(rt, FakeCodegen(), meta, 1, 4096, 4, allocator=allocator)
    ex.execute_decode_batch(off, read_output=False)
    ex.cleanup()
    rt.launched()
    ex.launch_step()
    ex.build_decode_graph()
    ex.launch_step()
    assert rt.launched() == ["vteb_decode_step_d128_kernel"] * 2
    with pytest.raises(CudaSafetyError, match="cleaned up"):
        ex.execute_decode_batch(off, read_output=False)
    assert rt.launched() == []


@pytest.mark.parametrize("tag", ["attn_step_boards", "attn_partials_source"])
@pytest.mark.parametrize("one", [None, True])
def test_an_allocator_without_room_keeps_the_launches_per_layer(built_library, tag, one):
    """Whichever of the two blocks of a one-launch step finds no room: what the other took is given back."""
    rt = HostOnly()
    allocator = SlabAllocator(rt, 180 << 30, requested_pool_size=1 << 30)
    allocator.initialize()
    allocate, taken, refused = allocator.allocate, [], []

    def without(size, name, region):
        if name == tag:
            refused.append(name)
            raise CudaSafetyError("slab exhausted")
        taken.append(allocate(size, name, region))
        return taken[-1]
    allocator.allocate = without
    meta = {"attention.head_count": 12, "attention.head_count_kv": 2, "attention.key_length": 128}
    ex = DecodeAttentionExecutor(rt, FakeCodegen(), meta, 1, 4096, 4, allocator=allocator, one_launch=one)
    if one:
        with pytest.raises(CudaSafetyError, match="exhausted"):
            ex.build_decode_graph()
        return
    ex.execute_decode_batch(np.array([100], dtype=np.int32), read_output=False)
    assert refused and ex._step is None and not ex._direct
    assert not any(n.startswith("vteb_decode_step") for n in rt.launched())
    assert [b.tag for b in taken if not b.in_use] == ([] if tag == "attn_step_boards" else ["attn_step_boards"])


@pytest.mark.parametrize("spare", [0, 1, 100, 4096])
def test_tiles_end_where_the_last_sequence_s_room_does(built_library, spare):
    """With a stride longer than the cache, the rows behind the last sequence may be anybody's: the maps end in front of them."""
    B, S = 3, 500
    ex, rt = host_only(B, S)
    row = 256
    ex.tensor_mapping['kv_batch_stride_elements'] = (S + spare) * row
    for l in range(ex.L):                                              # K of all layers, then V, in somebody else's memory
        for i, name in enumerate(("k", "v")):
            ex.tensor_mapping[f'blk.{l}.kv_cache.{name}'] = 0x5000_0000_0000 + (i * ex.L + l) * B * (S + spare) * row * 2
    ex.build_decode_graph()
    assert ex.route_name[0] == "vteb_decode_step_d128_kernel"
    step = [m for m in rt.maps if m[0] >= 0x5000_0000_0000]
    assert len(step) >= 2 * ex.L and all(n_rows == (B - 1) * (S + spare) + S and halves == row for _, n_rows, halves in step)


@pytest.mark.parametrize("one", [None, True])
def test_a_step_is_captured_for_the_mapping_of_its_time(built_library, one):
    """Between the capture of a device-side step and that of a step from the host, layer 1's Q becomes layer 0's output: layers
    that depend on one another take a launch list each, and partials are that list's own."""
    off, q = np.array([100], dtype=np.int32), np.zeros((4, 1, 12, 128), dtype=np.float16)
    ex, rt = host_only(output_f32=False, with_append=True, one_launch=one)
    ex.execute_decode_batch(off, read_output=False)
    assert rt.launched() == ["vteb_decode_step_d128_kernel"] and ex._partials_due
    ex.tensor_mapping['blk.1.q_proj.output'] = ex.tensor_mapping['blk.0.attention.output']
    if one:
        with pytest.raises(CudaSafetyError, match="another writes"):
            ex.execute_decode_batch(off, q)
        assert rt.launched() == []
        return
    ex.build_io_graph()
    assert ex._partials_due and ex.route_name is None
    ex.execute_decode_batch(off, q)
    names = rt.launched()
    assert not any(n.startswith("vteb_decode_step") for n in names) and names.count("kv_cache_append_kernel") == 4 and not ex._partials_due
    assert names[0] == names[-1] == "vteb_stage_copy_kernel"           # and the outputs are brought by a copy
    ex.execute_decode_batch(off, read_output=False)                    # the captured one
    assert rt.launched() == ["vteb_decode_step_d128_kernel"] and ex._partials_due
    ex, rt = host_only(output_f32=False)                               # a hook that came in between
    ex.execute_decode_batch(off, read_output=False)
    hooked, ex.per_layer_hook = [], lambda layer: hooked.append(layer)
    ex.execute_decode_batch(off, q)
    assert hooked == [0, 1, 2, 3] and not ex._partials_due


def test_a_refused_step_picks_no_launches(built_library):
    """A long sequence of two captured steps, route and dispatcher's launches: offsets out of range leave the choice as it was."""
    B, S, L = 32, 32768, 2
    ex, rt = host_only(B, S, L, one_launch=False)
    q, none, far = np.zeros((L, B, 12, 128), dtype=np.float16), np.zeros(B, dtype=np.int32), np.array([S] + [0] * (B - 1), dtype=np.int32)
    ex.build_decode_graph()
    ex.build_io_graph()
    assert ex._plain_io_graph_exec is not None
    ex.execute_decode_batch(none, read_output=False)
    before = ex._on_route, ex.route_name, ex.kernel_launches_per_step
    for call in (dict(q_host=q), dict(read_output=False)):
        with pytest.raises(CudaSafetyError):
            ex.execute_decode_batch(far, **call)
        assert (ex._on_route, ex.route_name, ex.kernel_launches_per_step) == before


def test_a_prepared_launch_is_refused_when_its_runtime_is_gone():
    """As every other launch is: its function is unloaded and its stream destroyed by then, while another runtime keeps the library going."""
    rt, launched = object.__new__(CudaRuntime), []
    vars(rt).update(_initialized=True, _panic=False, _props={"shared_mem_per_block": 49152}, _smem_optin_set={}, _stream=ctypes.c_void_p(1),
                    _lib=SimpleNamespace(vteb_launch=lambda *a: launched.append(a) or 0), _validate_launch=lambda *a: None)
    launch = rt.prepare_launch(ctypes.c_void_p(0x1001), [ctypes.c_int(1)], (1, 1, 1), (32, 1, 1))
    launch()
    assert len(launched) == 1
    rt._initialized = False
    with pytest.raises(CudaSafetyError):
        launch()
    rt._initialized, rt._panic = True, True
    with pytest.raises(CudaSafetyError, match="panic"):
        launch()
    assert len(launched) == 1


def kernel_source():
    from vte_b200.compiler.codegen import KERNEL_DIR
    return (KERNEL_DIR / "step_decode.cuh").read_text()


def test_boards_are_written_and_read_in_whole_tagged_words():
    """A value and the number that makes it valid are one scalar of one access on either side, ordered as relaxed ones are: the
    elements of a vector access have no order among themselves, and a plain store beside a relaxed load is a race."""
    src = kernel_source()
    assert "ulonglong2* boards;" in src and len(re.findall(r"= a\.boards \+", src)) == src.count("a.boards") == 2    # written, read
    assert "st.relaxed.gpu.global.v2.b64 [%0]" in src and "ld.relaxed.gpu.global.v2.b64 {%0, %1}" in src
    assert len(re.findall(r"store_entry\(to ", src)) == 3 and src.count("= load_entry(from_at[u])") == 2
    assert not re.search(r"\*to = |\bto\[[0-9D]|\*from_at|relaxed\S*\.v4", src)          # by no other access


def test_no_copy_outlives_its_block():
    """The warp that fetches stops where another gave up, whose tiles may have a copy under way to them, and waits for its last copies
    whoever it was; no row is appended that may not have come."""
    src = kernel_source()
    fetching = src[src.index("// ---- the tiles of the share"):src.index("// ---- Q of a run's heads")]
    assert re.search(r"!mbar_wait_bounded\(empty0 [^)]*\) \|\| \*abort_word != 0\)", fetching)
    assert re.search(r"\n        for \(int i = 1; i <= min\(sent, SLOTS\); \+\+i\) \{", fetching) and "if (!ok" not in fetching
    assert "if (lane < CPR && *abort_word == 0) {" in src


HEADS = [(12, 2, 128), (32, 8, 64), (8, 2, 256), (8, 8, 128), (7, 1, 128), (6, 3, 64), (8, 1, 256), (22, 2, 128), (32, 2, 128), (16, 1, 64)]
LENGTHS = [1, 15, 16, 17, 31, 33, 47, 48, 49, 64, 65, 95, 96, 97, 127, 128, 129, 257, 300]


def executor(rt, codegen, heads, B, S, L, **kw):
    meta = {"attention.head_count": heads[0], "attention.head_count_kv": heads[1], "attention.key_length": heads[2], **kw.pop("meta", {})}
    return DecodeAttentionExecutor(rt, codegen, meta, B, S, L, **{"one_launch": True, **kw})


@pytest.mark.gpu
@pytest.mark.parametrize("heads", HEADS)
@pytest.mark.parametrize("append", [True, False], ids=["append", "attend"])
@pytest.mark.parametrize("layers,lengths", [(1, LENGTHS), (3, LENGTHS), (3, [700]), (1, [5000]), (2, [1]), (5, [2049, 40])], ids=str)
def test_one_launch_matches_the_oracle(cuda_runtime, codegen, heads, append, layers, lengths):
    """Lengths at which a block, a warp's turn or a tile starts or ends; runs within a share and cut into 2 to 40 pieces (more
    than eight: merged in two steps); steps in turn on the same caches.  fp32 sums of fp16 products: 2e-5 of the result's norm;
    the newest rows are the projections' bits."""
    Hq, Hkv, D = heads
    B, S = len(lengths), max(lengths) + 3
    rng = np.random.default_rng(3)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    ex = executor(cuda_runtime, codegen, heads, B, S, layers, with_append=append)
    try:
        caches = [(f16(B, S, Hkv, D), f16(B, S, Hkv, D)) for _ in range(layers)]
        for step in range(2):
            off = np.array([min(n + step, S) for n in lengths], dtype=np.int32) - 1
            q, kn, vn = f16(layers, B, Hq, D), f16(layers, B, Hkv, D), f16(layers, B, Hkv, D)
            for l, (k, v) in enumerate(caches):
                for b in range(B):
                    k[b, off[b] + 1:], v[b, off[b] + 1:] = np.inf, np.nan            # nothing behind the end counts
                ex.upload_layer(l, q[l], k, v)
                ex.upload_new_kv(l, kn[l], vn[l])
            out = ex.execute_decode_batch(off)
            assert ex.kernel_launches_per_step == 1 and ex.route_name[0].startswith("vteb_decode_step_")
            for l, (k, v) in enumerate(caches):
                if append:
                    orc.kv_cache_append(kn[l], vn[l], k, v, off)
                ref = orc.decode_attention(q[l], np.where(np.isfinite(k), k, 0), np.where(np.isfinite(v), v, 0), off)
                assert np.linalg.norm(out[l] - ref) <= 2e-5 * np.linalg.norm(ref)
                for b in (0, B - 1):
                    got = ex.download_cache_rows(l, b, S)
                    assert all(np.array_equal(x.view(np.uint16), y[b].view(np.uint16)) for x, y in zip(got, (k, v)))
                for b in range(B):
                    k[b, off[b] + 1:], v[b, off[b] + 1:] = 0.5, 0.25
    finally:
        ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("heads", [(12, 2, 128), (32, 8, 64), (8, 2, 256), (22, 2, 128)])
@pytest.mark.parametrize("B", [31, 32, 33, 64, 65, 130])
def test_batches_of_more_sequences_than_a_warp_has_lanes(cuda_runtime, codegen, heads, B):
    """Lengths are added up 32 at a time; up to 64 offsets come with the launch, more from memory, through the captured step.  Several
    steps queued without a wait, each with offsets of its own and its rows to append; then the last one's outputs."""
    Hq, Hkv, D = heads
    S, L, rng = 150, 4, np.random.default_rng(B)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    ex = executor(cuda_runtime, codegen, heads, B, S, L, with_append=True)
    try:
        q, kn, vn = f16(L, B, Hq, D), f16(L, B, Hkv, D), f16(L, B, Hkv, D)
        caches = [(f16(B, S, Hkv, D), f16(B, S, Hkv, D)) for _ in range(L)]
        for l in range(L):
            ex.upload_layer(l, q[l], *caches[l])
            ex.upload_new_kv(l, kn[l], vn[l])
        first = rng.integers(0, S - 12, B).astype(np.int32)
        first[[0, B - 1]] = 0, S - 13
        for step in range(12):
            ex.execute_decode_batch(first + step, read_output=False)
        out = ex.execute_decode_batch(first + 12)
        assert len(ex._direct) == (B <= 64) and ex.route_name[1] == 0
        for l, (k, v) in enumerate(caches):
            for step in range(13):
                orc.kv_cache_append(kn[l], vn[l], k, v, first + step)
            ref = orc.decode_attention(q[l], k, v, first + 12)
            assert np.linalg.norm(out[l] - ref) <= 2e-5 * np.linalg.norm(ref)
            for b in {0, 1, min(32, B - 1), B - 1}:
                got = ex.download_cache_rows(l, b, S)
                assert all(np.array_equal(x.view(np.uint16), y[b].view(np.uint16)) for x, y in zip(got, (k, v)))
    finally:
        ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("heads", [(12, 2, 128), (32, 8, 64), (8, 2, 256), (22, 2, 128)])
def test_a_stride_longer_than_the_cache(cuda_runtime, codegen, heads):
    """Rows between one sequence's room and the next one's start, and behind the last one's, belong to others: neither counted nor touched."""
    Hq, Hkv, D = heads
    B, S, spare, L, rt = 3, 200, 7, 4, cuda_runtime
    rows = (B - 1) * (S + spare) + S
    rng = np.random.default_rng(4)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    ex, mine = executor(rt, codegen, heads, B, S, L, with_append=True), []
    try:
        off = np.array([S - 1, 100, S - 1], dtype=np.int32)
        q, kn, vn, data = f16(L, B, Hq, D), f16(L, B, Hkv, D), f16(L, B, Hkv, D), []
        ex.tensor_mapping['kv_batch_stride_elements'] = (S + spare) * Hkv * D
        for l in range(L):
            ex.upload_layer(l, q[l])
            ex.upload_new_kv(l, kn[l], vn[l])
            for name in ("k", "v"):
                x = f16(rows, Hkv, D)
                for b in range(B):
                    x[b * (S + spare) + S:(b + 1) * (S + spare)] = np.inf
                mine.append(rt.safe_malloc(x.nbytes, "kv cache"))
                rt.safe_memcpy_host_to_device(mine[-1], x, "kv upload")
                ex.tensor_mapping[f'blk.{l}.kv_cache.{name}'] = mine[-1].value
                data.append(x)
        out = ex.execute_decode_batch(off)
        assert ex.kernel_launches_per_step == 1
        for l in range(L):
            per_seq = lambda x: np.stack([x[b * (S + spare):b * (S + spare) + S] for b in range(B)])
            k, v = per_seq(data[2 * l]), per_seq(data[2 * l + 1])
            orc.kv_cache_append(kn[l], vn[l], k, v, off)
            ref = orc.decode_attention(q[l], k, v, off)
            assert np.linalg.norm(out[l] - ref) <= 2e-5 * np.linalg.norm(ref)
            for x, new, p in ((data[2 * l], kn[l], mine[2 * l]), (data[2 * l + 1], vn[l], mine[2 * l + 1])):
                for b in range(B):
                    x[b * (S + spare) + off[b]] = new[b]
                got = np.empty_like(x)
                rt.safe_memcpy_device_to_host(got, p, "kv rows for output check")
                assert np.array_equal(got.view(np.uint16), x.view(np.uint16))
    finally:
        ex.cleanup()
        for p in mine:
            rt.safe_free(p, "kv cache")


@pytest.mark.gpu
@pytest.mark.parametrize("heads,hg", [((32, 8, 64), 1), ((32, 8, 64), 2), ((12, 2, 128), 2), ((8, 8, 128), 4), ((16, 8, 64), 4)])
def test_heads_a_block_serves_at_once(cuda_runtime, codegen, heads, hg):
    """Other counts of KV heads a block than the plan chooses by itself."""
    Hq, Hkv, D = heads
    off, rng = np.array([0, 333, 499], dtype=np.int32), np.random.default_rng(6)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    q, k, v = f16(3, Hq, D), f16(3, 500, Hkv, D), f16(3, 500, Hkv, D)
    ex = executor(cuda_runtime, codegen, heads, 3, 500, 2)
    try:
        plan = cuda_runtime.step_plan
        ex.hip = ex.dispatcher.hip = type("Forced", (), {"__getattr__": lambda self, name: getattr(cuda_runtime, name),
                                                         "step_plan": staticmethod(lambda *a: plan(*a[:5], hg))})()
        for l in range(2):
            ex.upload_layer(l, q, k, v)
        out = ex.execute_decode_batch(off)
        assert ex._step.plan.hg == hg and ex.kernel_launches_per_step == 1
        ref = orc.decode_attention(q, k, v, off)
        assert all(np.linalg.norm(out[l] - ref) <= 2e-5 * np.linalg.norm(ref) for l in range(2))
    finally:
        ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("one", [None, False])
def test_a_step_with_its_own_offsets_is_not_captured(cuda_runtime, codegen, one):
    """Its offsets would be the replays' too: refused as a graph launch in a capture is, and the next step is right."""
    rt = cuda_runtime
    ex = executor(rt, codegen, (12, 2, 128), 1, 512, 4, one_launch=one)
    try:
        for l in range(4):
            ex.fill_cache_on_device(l, l + 1)
            ex.upload_layer(l, np.ones((1, 12, 128), dtype=np.float16))
        off = np.array([300], dtype=np.int32)
        good = ex.execute_decode_batch(off)
        rt.stream_begin_capture()
        with pytest.raises(CudaRuntimeError, match="900"):
            ex.execute_decode_batch(off - 1, read_output=False)
        try:
            graph = rt.stream_end_capture()
        except CudaRuntimeError:
            assert one is False                                        # a refused graph launch ends the capture
        else:
            assert one is None and rt.graph_node_count(graph) == 0
            rt.graph_destroy(graph)
        assert np.array_equal(ex.execute_decode_batch(off), good)
    finally:
        ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("heads", HEADS)
@pytest.mark.parametrize("layers,lengths", [(1, [17000]), (1, [2100]), (2, [9000])], ids=str)
def test_cut_runs_are_merged_once_or_twice(cuda_runtime, codegen, heads, layers, lengths):
    """Either side of eight tiles a CTA with no more states of a run than one merge takes: above it a run lies in up to 148 shares, whose
    states are merged in two steps.  fp32 sums: 2e-5 of the result's norm."""
    Hq, Hkv, D = heads
    B, S = len(lengths), max(lengths)
    rng = np.random.default_rng(21)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    ex = executor(cuda_runtime, codegen, heads, B, S, layers)
    try:
        data = [(f16(B, Hq, D), f16(B, S, Hkv, D), f16(B, S, Hkv, D)) for _ in range(layers)]
        for l in range(layers):
            ex.upload_layer(l, *data[l])
        off = np.array(lengths, dtype=np.int32) - 1
        for _ in range(2):
            out = ex.execute_decode_batch(off)
            for l in range(layers):
                ref = orc.decode_attention(*data[l], off)
                assert np.linalg.norm(out[l] - ref) <= 2e-5 * np.linalg.norm(ref)
    finally:
        ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("heads,meta", [((12, 2, 128), {}), ((8, 4, 64), dict(rope_type=1)), ((8, 2, 256), dict(rope_type=2, rotary_dim=64)),
                                        ((8, 2, 256), {}), ((16, 2, 128), dict(rope_type=2, rotary_dim=128))])
@pytest.mark.parametrize("rope", ["fused", "fused-append"])
def test_one_launch_rotates(cuda_runtime, codegen, heads, meta, rope):
    """Q and the newest K row rotated on the way: the oracle's outputs, and the oracle's bits in the cache."""
    Hq, Hkv, D = heads
    B, S, L = 3, 600, 3
    rng = np.random.default_rng(5)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    ex = executor(cuda_runtime, codegen, heads, B, S, L, rope=rope, meta=meta)
    rope_type, width = meta.get("rope_type", 0), meta.get("rotary_dim", D)
    cos, sin = orc.rope_tables(S, width, 1e6)
    try:
        off = np.array([0, 333, 599], dtype=np.int32)
        for l in range(L):
            q, k, v, kn, vn = f16(B, Hq, D), f16(B, S, Hkv, D), f16(B, S, Hkv, D), f16(B, Hkv, D), f16(B, Hkv, D)
            ex.upload_layer(l, q, k, v)
            ex.upload_new_kv(l, kn, vn)
            if l == L - 1:
                out = ex.execute_decode_batch(off)
        assert ex.kernel_launches_per_step == 1
        q, kn = orc.rope_step(q, kn, cos, sin, off, rope_type, width)
        orc.kv_cache_append(kn, vn, k, v, off)
        ref = orc.decode_attention(q, k, v, off)
        assert np.linalg.norm(out[L - 1] - ref) <= 2e-5 * np.linalg.norm(ref)
        for b in range(B):
            got = ex.download_cache_rows(L - 1, b, S)
            assert np.array_equal(got[0].view(np.uint16), k[b].view(np.uint16)) and np.array_equal(got[1].view(np.uint16), v[b].view(np.uint16))
    finally:
        ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("heads,B,S", [((12, 2, 128), 1, 8192), ((32, 8, 64), 4, 2048), ((8, 2, 256), 2, 4096), ((32, 2, 128), 2, 4096)])
def test_one_launch_is_as_exact_as_the_launches_per_layer(cuda_runtime, codegen, heads, B, S):
    """Both against 64-bit sums: the routes it takes the place of keep fp32 sums of fp16 products, at 1.5e-7 to 2.2e-7 of the norm or
    more; a tenth is allowed for the order of the sums."""
    Hq, Hkv, D = heads
    rng = np.random.default_rng(S)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    L, off = 2, np.full(B, S - 1, dtype=np.int32)
    data, error = [(f16(B, Hq, D), f16(B, S, Hkv, D), f16(B, S, Hkv, D)) for _ in range(L)], []
    ref = [orc.decode_attention(*x, off, dtype=np.float64) for x in data]
    for one in (True, False):
        ex = executor(cuda_runtime, codegen, heads, B, S, L, one_launch=one)
        try:
            for l in range(L):
                ex.upload_layer(l, *data[l])
            out = ex.execute_decode_batch(off)
            error.append(max(np.linalg.norm(out[l] - ref[l]) / np.linalg.norm(ref[l]) for l in range(L)))
        finally:
            ex.cleanup()
    assert error[0] <= 1.1 * error[1]


@pytest.mark.gpu
@pytest.mark.parametrize("heads", [(12, 2, 128), (32, 8, 64), (8, 2, 256), (32, 2, 128)])
def test_infinite_values_stay_infinite(cuda_runtime, codegen, heads):
    """An infinite V gives the infinities and NaNs of fp32 products, in columns of its own; the others are untouched."""
    Hq, Hkv, D = heads
    B, S, L = 2, 500, 3
    rng = np.random.default_rng(11)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    ex = executor(cuda_runtime, codegen, heads, B, S, L)
    try:
        off = np.array([S - 1, 40], dtype=np.int32)
        q, k, v = f16(B, Hq, D), f16(B, S, Hkv, D), f16(B, S, Hkv, D)
        v[0, 17, 0, 3], v[0, 400, 0, 5], v[1, 40, Hkv - 1, D - 1] = np.inf, -np.inf, np.inf
        for l in range(L):
            ex.upload_layer(l, q, k, v)
        out = ex.execute_decode_batch(off)
        ref = orc.decode_attention(q, k, v, off)
        assert np.isinf(ref).any()
        for l in range(L):
            assert np.array_equal(np.isposinf(out[l]), np.isposinf(ref)) and np.array_equal(np.isneginf(out[l]), np.isneginf(ref))
            fine = np.isfinite(ref)
            assert np.linalg.norm(out[l][fine] - ref[fine]) <= 2e-5 * np.linalg.norm(ref[fine])
    finally:
        ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("heads,meta,B,way", [
    ((12, 2, 128), {}, 2, dict(one_launch=True)), ((8, 4, 64), dict(rope_type=1), 2, dict(one_launch=True)),
    ((8, 2, 256), dict(rope_type=2, rotary_dim=64), 2, dict(one_launch=True)), ((16, 2, 128), dict(rope_type=2, rotary_dim=64), 2, dict(one_launch=True)),
    ((12, 2, 128), {}, 2, dict(lean=(8, 1))), ((8, 4, 64), dict(rope_type=1), 2, dict(lean=(4, 1))), ((8, 2, 256), {}, 2, dict(lean=(5, 2))),
    ((8, 2, 256), dict(rope_type=2, rotary_dim=64), 1, dict(lean=(20, 0)))], ids=str)
@pytest.mark.parametrize("rope", ["fused", "fused-append"])
def test_infinite_values_stay_infinite_under_a_rotation(cuda_runtime, codegen, heads, meta, B, way, rope):
    """The same where the kernel rotates Q itself, the newest row's V among the infinite ones."""
    Hq, Hkv, D = heads
    S, L = 500, 2
    rng = np.random.default_rng(12)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    ex = executor(cuda_runtime, codegen, heads, B, S, L, rope=rope, meta=meta, **{"one_launch": None, **way})
    rope_type, width = meta.get("rope_type", 0), meta.get("rotary_dim", D)
    try:
        off = np.array([S - 1, 40], dtype=np.int32)[:B]
        q, k, v, kn, vn = f16(B, Hq, D), f16(B, S, Hkv, D), f16(B, S, Hkv, D), f16(B, Hkv, D), f16(B, Hkv, D)
        v[0, 17, 0, 3], v[0, 400, 0, 5], v[0, :400:7, Hkv - 1, 9] = np.inf, -np.inf, np.inf
        vn[0, 0, 40], vn[B - 1, Hkv - 1, D - 1] = np.inf, -np.inf
        for l in range(L):
            ex.upload_layer(l, q, k, v)
            ex.upload_new_kv(l, kn, vn)
        out = ex.execute_decode_batch(off)
        assert ex.route_name is not None
        q, kn = orc.rope_step(q, kn, *orc.rope_tables(S, width, 1e6), off, rope_type, width)
        orc.kv_cache_append(kn, vn, k, v, off)
        ref = orc.decode_attention(q, k, v, off)
        fine = np.isfinite(ref)
        assert np.isposinf(ref).any() and np.isneginf(ref).any()
        for l in range(L):
            assert np.array_equal(np.isposinf(out[l]), np.isposinf(ref)) and np.array_equal(np.isneginf(out[l]), np.isneginf(ref))
            assert np.linalg.norm(out[l][fine] - ref[fine]) <= 2e-5 * np.linalg.norm(ref[fine])
    finally:
        ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(with_append=True), dict(rope="fused-append"), {}], ids=str)
def test_partials_after_one_launch_and_many_layers(cuda_runtime, codegen, kw):
    """70 layers are two launches; the partials of the last one are those of a launch list per layer, bit for bit."""
    heads, B, S, L = (12, 2, 128), 2, 200, 70
    Hq, Hkv, D = heads
    rng = np.random.default_rng(2)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    q, kn, vn = f16(L, B, Hq, D), f16(L, B, Hkv, D), f16(L, B, Hkv, D)
    caches, off, got = [(f16(B, S, Hkv, D), f16(B, S, Hkv, D)) for _ in range(L)], np.array([150, 199], dtype=np.int32), []
    for one in (True, False):
        ex = executor(cuda_runtime, codegen, heads, B, S, L, one_launch=one, output_f32=False, **kw)
        try:
            for l in range(L):
                ex.upload_layer(l, q[l], *caches[l])
                ex.upload_new_kv(l, kn[l], vn[l])
            out = ex.execute_decode_batch(off)
            assert not one or ex.kernel_launches_per_step == 2
            again = ex.execute_decode_batch(off, q)                  # from the host
            assert np.array_equal(out, again)
            for l in range(L):
                ex.upload_layer(l, q[L - 1 - l])                      # the next step's
            got.append((out, ex.read_partials()))
        finally:
            ex.cleanup()
    (a, pa), (b, pb) = got
    assert np.linalg.norm(a.astype(np.float64) - b) <= 5e-4 * np.linalg.norm(b.astype(np.float64))      # fp16 outputs, rounded once
    used = pb[1] > 0
    assert used.any() and np.array_equal(pa[1], pb[1]) and np.array_equal(pa[0][used], pb[0][used]) and np.array_equal(pa[2][used], pb[2][used])


@pytest.mark.gpu
@pytest.mark.parametrize("heads", [(12, 2, 128), (32, 8, 64), (8, 2, 256), (32, 2, 128)])
@pytest.mark.parametrize("f32,one", [(True, True), (False, True), (True, None), (False, None)])
def test_a_step_from_the_host_stores_its_outputs_there(cuda_runtime, codegen, heads, f32, one):
    """The bits of the same step on the device, in its buffers as well.  Outputs above the limit go through copy nodes, to the same bits."""
    from vte_b200.core import decode_executor as de
    Hq, Hkv, D = heads
    B, S, L = 3, 500, 5 if one else 2                         # two layers: clusters, a launch each
    rng = np.random.default_rng(8)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    got, caches = [], [(f16(B, S, Hkv, D), f16(B, S, Hkv, D)) for _ in range(L)]
    new = [(f16(B, Hkv, D), f16(B, Hkv, D)) for _ in range(L)]
    steps = [(f16(L, B, Hq, D), rng.integers(0, S, B).astype(np.int32)) for _ in range(3)]
    limit = de.STAGE_COPY_MAX_BYTES
    for way in ("device", "host", "copies"):
        de.STAGE_COPY_MAX_BYTES = 0 if way == "copies" else limit
        ex = executor(cuda_runtime, codegen, heads, B, S, L, output_f32=f32, with_append=not one, one_launch=one)
        try:
            for l in range(L):
                ex.upload_new_kv(l, *new[l])
                ex.upload_cache(l, *caches[l])
            mine = []
            for bad in (np.array([0, S, 1], dtype=np.int32), np.array([0, -1, 1], dtype=np.int32), np.zeros(B + 1, dtype=np.int32)):
                with pytest.raises(CudaSafetyError):
                    ex.execute_decode_batch(bad, steps[0][0])
                with pytest.raises(CudaSafetyError):
                    ex.execute_decode_batch(bad)
            for q, off in steps:
                if way == "device":
                    for l in range(L):
                        ex.upload_layer(l, q[l])
                mine.append(ex.execute_decode_batch(off, None if way == "device" else q))
                assert (ex._mirror() is None) == (way == "copies" or not one)
                left_q, left_off, left = np.empty_like(q), np.empty_like(off), np.empty_like(mine[-1])
                for to, at in ((left_q, ex.q_all.ptr), (left_off, ex.offsets.ptr), (left, ex.out_all.ptr)):
                    cuda_runtime.safe_memcpy_device_to_host(to, ctypes.c_void_p(at), "output")
                assert np.array_equal(left_q, q) and np.array_equal(left_off, off) and np.array_equal(left, mine[-1])
            got.append(mine)
        finally:
            ex.cleanup()
            de.STAGE_COPY_MAX_BYTES = limit
    for other in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(got[0], other))


@pytest.mark.gpu
def test_shared_caches_with_an_append_keep_their_order(cuda_runtime, codegen):
    """Layers that append to one cache depend on one another: a launch list per layer, and `one_launch` is refused."""
    for kw, name in ((dict(with_append=True), None), ({}, "vteb_decode_step_d128_kernel")):
        ex = executor(cuda_runtime, codegen, (12, 2, 128), 1, 600, 4, n_kv_buffers=2, one_launch=None, **kw)
        try:
            ex.build_decode_graph()
            assert (ex.route_name or ("",))[0] == name if name else not (ex.route_name or ("",))[0].startswith("vteb_decode_step")
        finally:
            ex.cleanup()
    ex = executor(cuda_runtime, codegen, (12, 2, 128), 1, 600, 4, n_kv_buffers=2, with_append=True)
    try:
        with pytest.raises(CudaSafetyError, match="another writes"):
            ex.build_decode_graph()
    finally:
        ex.cleanup()


@pytest.mark.gpu
def test_a_state_that_never_comes_is_reported(cuda_runtime, codegen):
    """One CTA's count of launches is set off by five, so its state carries another number than the CTA that finishes the run
    waits for: after 200,000 cycles the kernel gives up and says so, and the next step is right."""
    class Short:
        def load_kernel_safe(self, *a, **kw):
            return codegen.load_kernel_safe(*a, vteb_wait_limit_cycles=200000, **kw)
    ex = DecodeAttentionExecutor(cuda_runtime, Short(), {"attention.head_count": 12, "attention.head_count_kv": 2, "attention.key_length": 128},
                                 1, 4096, 4, one_launch=True)
    try:
        for l in range(4):
            ex.fill_cache_on_device(l, l + 1)
            ex.upload_layer(l, np.ones((1, 12, 128), dtype=np.float16))
        off = np.array([4095], dtype=np.int32)
        good = ex.execute_decode_batch(off)
        count = ctypes.c_void_p(ex._step.launch_counts)
        cuda_runtime.safe_memcpy_host_to_device(count, np.array([5], dtype=np.uint32), "launch count")
        with pytest.raises(CudaRuntimeError):
            ex.execute_decode_batch(off)
        with pytest.raises(CudaRuntimeError):
            ex.execute_decode_batch(off, np.ones((4, 1, 12, 128), dtype=np.float16))
        cuda_runtime.safe_memcpy_host_to_device(count, np.array([3], dtype=np.uint32), "launch count")
        assert np.array_equal(ex.execute_decode_batch(off), good)
    finally:
        ex.cleanup()
