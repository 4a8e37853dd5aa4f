"""Routes with one work item per CTA (core/lean_route.py): what is chosen, on the CPU, and the kernels against the oracle
where lengths, parts and blocks meet."""
import ctypes
import math

import numpy as np
import pytest

from oracle import attention_oracle as orc
from vte_b200.bridge.cuda_runtime import LeanPlan, load_library
from vte_b200.core.decode_executor import DecodeAttentionExecutor
from vte_b200.bridge.errors import CudaSafetyError
from vte_b200.core.lean_route import CLUSTER_PARTS, LEAN_SPLIT_MAX_CONTEXT, LeanRoute, choose_lean_route


def lean_plan(*a):
    plan = LeanPlan()
    assert load_library().vteb_lean_plan(*a, ctypes.byref(plan)) == 0
    return plan


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("group", [1, 6, 8, 9, 16, 17])
def test_plan_holds_exchange_rows_and_received_states(built_library, group, D):
    for parts in (1, 2, 7, 16, 17, 148):
        for kind in (0, 1, 2):
            for context in (1, 128, 129, 4096, 1 << 20):
                p, cluster = lean_plan(2 * group, 2, D, parts, context, kind), kind > 0
                covered = group <= (8 if D == 256 or not cluster else 16) and (not cluster or 2 <= parts <= 16) and not (kind == 2 and D == 64)
                assert bool(p.ok) == covered
                if not covered:
                    continue
                warps = p.threads // 32
                assert warps == (6 if D == 256 else 8) // (2 if kind == 2 else 1)
                assert p.threads % (D // 8) == 0 and 1 <= p.depth <= (2 if D == 256 else 3)
                assert p.depth * 64 * D >= group * (D + 8) * 4                   # a warp's exchange rows in its own blocks
                blocks = -(-(-(-context // parts)) // 16)
                assert p.depth * warps >= min(blocks, 3 * warps if D < 256 else 2 * warps)
                need = 128 + (2 if group > 8 else 1) * D * 16 + warps * p.depth * 64 * D
                need += -(-(group * D // 32) // parts) * parts * 144 if cluster else 0
                assert p.smem_bytes == need <= 225 * 1024


class FakeHip:
    lean_plan = staticmethod(lean_plan)
    lean_estimate = staticmethod(lambda *a: load_library().vteb_lean_estimate(*a, 148))
    lean_step_estimate = staticmethod(lambda *a: load_library().vteb_lean_step_estimate(*a))
    get_gpu_architecture = staticmethod(lambda: "sm_100a")

    @staticmethod
    def max_active_clusters(fn, cluster, threads, smem):
        """What a B200 says with one block an SM, and with two."""
        one = {2: 74, 3: 45, 4: 33, 5: 26, 6: 22, 8: 15, 9: 15, 12: 7, 16: 7}
        two = {2: 148, 3: 93, 4: 71, 5: 56, 6: 45, 8: 33, 9: 30, 12: 21, 16: 14}
        return (two if smem <= 112 * 1024 else one)[cluster]


class FakeDispatcher:
    def __init__(self, heads, batch, context):
        self.num_q_heads, self.num_kv_heads, self.head_dim = heads
        self.batch_size, self.context_length, self.num_sms, self.max_chunks = batch, context, 148, 148
        self.hip, self.codegen, self.output_f32 = FakeHip, self, True

    def load_kernel_safe(self, *a):
        return None, ctypes.c_void_p(1)


def test_the_route_follows_the_size(built_library):
    route = lambda *a: choose_lean_route(FakeDispatcher(*a), True)
    assert route((12, 2, 128), 1, 4096) == (16, 1)                # one short sequence
    assert route((12, 2, 128), 1, 16384) == (74, 0)               # one long one: split and combine over the whole GPU
    assert route((12, 2, 128), 1, LEAN_SPLIT_MAX_CONTEXT + 1) == (0, 0)
    alone = lambda *a: choose_lean_route(FakeDispatcher(*a), False)
    assert alone((12, 2, 128), 1, 32768) == (74, 0) and alone((32, 8, 64), 1, 32768) == (18, 0) and alone((8, 2, 256), 1, 10000)[1] == 0
    assert route((8, 2, 256), 1, 32768) == (74, 0) and alone((8, 2, 256), 1, 32768) == alone((16, 4, 64), 1, 32768) == (0, 0)
    assert route((32, 8, 64), 64, 16384) == (0, 0)                # a batch that streams: equal shares
    assert route((32, 2, 128), 8, 4096)[1] and route((12, 2, 128), 4, 2048)[1]
    assert route((8, 8, 128), 37, 624) == (2, 2)                  # many pairs: clusters of half blocks
    assert route((34, 2, 128), 4, 2048) == (0, 0)                 # seventeen query heads on a KV head
    assert route((32, 2, 256), 4, 2048) == (0, 0)                 # sixteen with 256-wide heads
    assert route((12, 2, 96), 4, 2048) == (0, 0)
    for batch in (1, 3, 17, 64):
        for context in (1, 130, 1000, 9000, 70000):
            parts, kind = route((28, 4, 128), batch, context)
            assert parts == 0 or (parts in CLUSTER_PARTS if kind else batch == 1 and parts == 37)


def test_both_sides_of_the_rule_agree():
    """The executors' choice is in Python, the direct entry point's in C++."""
    import re
    from pathlib import Path
    from vte_b200.core import lean_route
    csrc = Path(lean_route.__file__).resolve().parent.parent / "csrc"
    margin = re.search(r"kLeanMargin = ([\d.]+);", (csrc / "kernels" / "lean_decode.cuh").read_text()).group(1)
    parts = re.search(r"kParts\[\] = \{([\d, ]+)\}", (csrc / "cluster_choice.h").read_text()).group(1)
    assert float(margin) == lean_route.MARGIN and tuple(int(x) for x in parts.split(",")) == CLUSTER_PARTS


def test_small_caches_keep_the_one_launch_that_is_shorter(built_library):
    """Up to 128 positions the dispatcher's layer is one launch.  Timed, dispatcher / clusters, us: 64 sequences of 32 heads on
    8 of 64 3.1 / 14.1 (room for 16) and 6.4 / 16.2 (128), of 28 on 4 of 128 4.9 / 9.5, of 8 on 2 of 256 5.4 / 6.4; one
    sequence of 8 on 2 of 256 3.1 / 4.1; of 12 on 2 of 128 with room for 128 4.9 / 3.1, eight of 28 on 4 7.2 / 4.0."""
    route = lambda *a, append=False: choose_lean_route(FakeDispatcher(*a), append)
    for append in (False, True):
        for capacity in (16, 64, 128):
            assert route((32, 8, 64), 64, capacity, append=append) == (0, 0)
            assert route((28, 4, 128), 64, capacity, append=append) == (0, 0)
        assert route((8, 2, 256), 64, 16, append=append) == (0, 0) and route((8, 2, 256), 1, 16) == (0, 0)
        assert route((12, 2, 128), 1, 128, append=append)[1] and route((28, 4, 128), 8, 128, append=append)[1]


def chosen_route(heads, batch, capacity, append=True):
    d = FakeDispatcher(heads, batch, capacity)
    parts, kind = choose_lean_route(d, append)
    return LeanRoute(d, parts, kind, append)


def test_one_long_sequence_among_short_ones_leaves_the_clusters(built_library):
    """Timed, clusters / dispatcher, us a layer, append included: 71 / 29, 74 / 33, 46 / 37, 40 / 23; with all sequences
    short 6.8 / 14, 7.6 / 15, 5.5 / 15, 7.7 / 15."""
    for heads, batch, capacity, others in (((12, 2, 128), 32, 32768, 500), ((12, 2, 128), 16, 65536, 1000),
                                           ((28, 4, 128), 8, 32768, 500), ((8, 2, 256), 16, 16384, 400)):
        route = chosen_route(heads, batch, capacity)
        assert route.cluster
        assert not route.pays(capacity, capacity + (batch - 1) * others) and route.pays(others, batch * others)
        known = route.pays_up_to()
        assert others < known < capacity and route.pays(known, known + batch - 1) and route.pays(known, known * batch)
    for heads, batch, capacity in (((12, 2, 128), 8, 2048), ((28, 4, 128), 4, 4096), ((32, 2, 128), 8, 4096), ((12, 2, 128), 8, 128)):
        assert chosen_route(heads, batch, capacity).pays_up_to() == capacity       # no lengths for which they do not
    assert chosen_route((12, 2, 128), 1, 16384).pays_up_to() == 16384              # one sequence, split and combine


def test_a_forced_split_route_stays_within_the_partial_buffers(built_library):
    """Each (sequence, query head) has room for max_chunks partials: one sequence of up to 2,048 positions for 32."""
    d = FakeDispatcher((12, 2, 128), 1, 2048)
    d.max_chunks = 32
    assert LeanRoute(d, 32, 0, False).parts == 32 and LeanRoute(d, 16, 1, False).parts == 16
    for parts in (33, 37, 148):
        with pytest.raises(CudaSafetyError, match="room for 32"):
            LeanRoute(d, parts, 0, False)


def real_dispatcher(**kw):
    from tests import test_host_logic as host
    d = host.make_dispatcher(**{"context_length": 4096, "batch_size": 1, **kw})[0]
    d.hip.lean_plan, d.hip.programmatic_launch = lean_plan, False
    d._allocate_scratch()
    return d, {**host.mapping(stride=4096 * 256), "rope_cos": 0x7300_0000_0000, "rope_sin": 0x7300_0010_0000}


@pytest.mark.parametrize("kind", [0, 1])
def test_a_route_checks_the_rows_to_append(built_library, kind):
    """Null new rows would mean to the kernel that the row is in the cache already; rows that 16-byte loads cannot read
    go through an append launch where the step has one, and are refused where the caller left it out."""
    d, m = real_dispatcher()
    names = [fn_args[1] for fn_args in LeanRoute(d, 16, kind, True).launches(0, m, 0x7200_0000_0000, 1)[:1]]
    assert [a.value for a in names[0][13:15]] == [m['blk.0.k_proj.output'], m['blk.0.v_proj.output']]
    for name in ('blk.0.k_proj.output', 'blk.0.v_proj.output'):
        with pytest.raises(CudaSafetyError, match="null"):
            LeanRoute(d, 16, kind, True).launches(0, {k: v for k, v in m.items() if k != name}, 0x7200_0000_0000, 1)
        odd = {**m, name: m[name] + 2}
        got = LeanRoute(d, 16, kind, True).launches(0, odd, 0x7200_0000_0000, 1)
        assert [x[2:] for x in got] == [x[2:] for x in d.build_launches(0, odd, 0x7200_0000_0000, 1)] and len(got) == 3
        assert m[name] + 2 in [a.value for a in got[0][1][:2]]
        folded, _ = real_dispatcher(fuse_append=True)
        with pytest.raises(CudaSafetyError, match="16-byte aligned"):
            LeanRoute(folded, 16, kind, True).launches(0, odd, 0x7200_0000_0000, 1)


@pytest.mark.parametrize("kind", [0, 1])
def test_a_route_checks_the_rotation_s_tables(built_library, kind):
    d, m = real_dispatcher(fuse_rope=True)
    args = LeanRoute(d, 16, kind, True).launches(0, m, 0x7200_0000_0000, 1)[0][1]
    assert [a.value for a in args[22:24]] == [m['rope_cos'], m['rope_sin']]
    for name in ('rope_cos', 'rope_sin'):
        for bad in ({k: v for k, v in m.items() if k != name}, {**m, name: m[name] + 2}):
            with pytest.raises(CudaSafetyError, match="rope_cos / rope_sin"):
                LeanRoute(d, 16, kind, True).launches(0, bad, 0x7200_0000_0000, 1)


def test_a_route_looks_no_further_than_a_pool_for_the_next_layer_s_rows(built_library):
    """The L2 prefetch reads the next layer's caches by name only (a pool's last layer has none behind it), at 16 bytes."""
    d, m = real_dispatcher()
    ahead = lambda m: [a.value or 0 for a in LeanRoute(d, 16, 0, True).launches(0, m, 0x7200_0000_0000, 1)[0][1][20:22]]
    next_k, next_v = 0x7400_0000_0000, 0x7500_0000_0000
    assert ahead({**m, 'blk.1.kv_cache.k': next_k, 'blk.1.kv_cache.v': next_v}) == [next_k, next_v]
    pooled = {k: v for k, v in m.items() if 'kv_cache' not in k}
    for without in ({**pooled, 'KV Cache Pool': 0x7600_0000_0000}, {**m, 'blk.1.kv_cache.k': next_k},
                    {**m, 'blk.1.kv_cache.k': next_k, 'blk.1.kv_cache.v': next_v + 8}):
        assert ahead(without) == [0, 0]


@pytest.mark.parametrize("forced", [False, True])
def test_an_allocator_without_room_for_the_copy_of_q_keeps_the_dispatcher_s_launches(built_library, forced):
    from types import SimpleNamespace

    def full(size, tag, region):
        raise CudaSafetyError("slab exhausted")
    d, _ = real_dispatcher()
    for name in ("lean_estimate", "lean_step_estimate", "max_active_clusters"):
        setattr(d.hip, name, getattr(FakeHip, name))
    ex = object.__new__(DecodeAttentionExecutor)
    vars(ex).update(dispatcher=d, hip=d.hip, B=1, S=4096, q_bytes=3072, use_graph=True, per_layer_hook=None, launch_rewriter=None, with_append=True,
                    _route=None, _lean=(16, 1) if forced else None, _forced_route=forced, allocator=SimpleNamespace(allocate=full))
    if forced:
        with pytest.raises(CudaSafetyError, match="exhausted"):
            ex._choose_route()
    else:
        ex._choose_route()
        assert ex._route is None and ex._lean == (0, 0)


@pytest.mark.parametrize("option", ["compat", "strict_empty_splits", "emit_state", "fused_combine"])
def test_a_forced_route_refuses_what_it_would_drop(option):
    with pytest.raises(CudaSafetyError, match="lean_route"):
        DecodeAttentionExecutor(None, None, {}, 1, 256, 1, lean=(4, 1), **{option: True})


def test_the_unsplit_kernel_goes_to_clusters_where_they_pay(built_library):
    """Which launches of flash_attention_kernel do, and with which arguments; all others keep their own builds."""
    from vte_b200.compiler.signatures import CLUSTER_KERNELS, KERNEL_SIGNATURES
    from vte_b200.core.lean_route import unsplit_as_clusters
    hip = FakeHip()
    hip.get_num_cus = lambda: 148
    kernels = {name: name for name in CLUSTER_KERNELS}
    vp, ci = ctypes.c_void_p, ctypes.c_int

    def served(B=4, heads=(12, 2, 128), capacity=2048, grid=None, block=None, at=0, stride=None, **status):
        Hq, Hkv, D = heads
        args = [vp(0x1000 * (i + 1)) for i in range(6)] + [ci(1), ci(Hq), ci(Hkv), ci(D), ctypes.c_float(0.5), vp(0x9000),
                                                          ci(capacity * Hkv * D if stride is None else stride)]
        args[0] = vp(0x1000 + at)
        return unsplit_as_clusters(hip, kernels, args, grid or (B, Hq, 1), block or (D, 1, 1), **status)
    assert served(status=0x4440)[1][19].value == 0x4440
    fn, args, grid, block, smem = served()
    parts = args[12].value
    assert fn.startswith("vteb_decode_cluster_") and fn.endswith("d128_kernel") and parts in CLUSTER_PARTS and grid == (8 * parts, 1, 1) and grid.cluster == parts
    assert [isinstance(a, t) for a, t in zip(args, KERNEL_SIGNATURES[fn])] == [True] * len(KERNEL_SIGNATURES[fn]) and block in ((256, 1, 1), (128, 1, 1))
    assert [a.value for a in (args[0], args[1], args[2], args[13], args[14], args[15])] == [0x1000, 0x4000, 0x5000, 0x2000, 0x3000, 0x6000]
    assert args[16].value == 1 and args[17].value == 32 and args[9].value == 0.5 and args[11].value == 2048 * 256
    assert served(heads=(32, 2, 128))[0].endswith("2_d128_kernel") and served(B=74)[1][12].value == 2
    for refused in (dict(capacity=256), dict(capacity=512, heads=(32, 2, 128)), dict(B=75), dict(heads=(34, 2, 128)), dict(stride=0),
                    dict(stride=2048 * 256 + 4), dict(at=8), dict(grid=(4, 6, 1)), dict(block=(64, 1, 1)), dict(heads=(32, 2, 256)),
                    dict(heads=(12, 2, 96)), dict(grid=(4, 12, 2))):
        assert served(**refused) is None, refused


def test_a_wait_that_ran_out_is_raised_wherever_the_host_waits(built_library):
    """Launches whose arguments have no status word report to one of the runtime's: raised once, by whichever wait is next."""
    from vte_b200.bridge.cuda_runtime import CudaRuntime, ERR_DEVICE_STATUS
    from vte_b200.bridge.errors import CudaRuntimeError

    class FakeLib:
        def __getattr__(self, name):
            return lambda *a: 0
    rt = CudaRuntime(str(built_library))
    rt._lib, rt._initialized, rt._launch_status = FakeLib(), True, ctypes.c_int(0)
    for wait in (rt.synchronize, rt.stream_synchronize, lambda: rt.event_synchronize(ctypes.c_void_p(1))):
        wait()
        rt._launch_status.value = 4
        with pytest.raises(CudaRuntimeError, match="bounded wait") as e:
            wait()
        assert e.value.code == ERR_DEVICE_STATUS
        wait()


@pytest.mark.parametrize("off", [False, True])
def test_cluster_launches_of_the_unsplit_kernel_obey_the_programmatic_switch(built_library, monkeypatch, off):
    from vte_b200.bridge.cuda_runtime import CudaRuntime, LAUNCH_CLUSTER_SHIFT, LAUNCH_PROGRAMMATIC
    from vte_b200.compiler.signatures import CLUSTER_KERNELS
    monkeypatch.setenv("VTE_B200_NO_PDL", "1") if off else monkeypatch.delenv("VTE_B200_NO_PDL", raising=False)
    rt, flags = CudaRuntime(str(built_library)), []

    class FakeLib:
        def __getattr__(self, name):
            return lambda *a: flags.append(a[-1]) or 0 if name == "vteb_launch" else 0
    rt.get_num_cus, rt.max_active_clusters, rt.lean_plan = lambda: 148, FakeHip.max_active_clusters, lean_plan
    rt.lean_estimate = FakeHip.lean_estimate
    rt._lib, rt._initialized, rt._props = FakeLib(), True, {"max_threads_per_block": 1024, "shared_mem_per_block": 49152,
                                                            "shared_mem_per_block_optin": 232448}
    rt._clustered = {2: {name: ctypes.c_void_p(3) for name in CLUSTER_KERNELS}}
    vp, ci = ctypes.c_void_p, ctypes.c_int
    args = [vp(0x1000 * (i + 1)) for i in range(6)] + [ci(1), ci(12), ci(2), ci(128), ctypes.c_float(0.5), vp(0x9000), ci(2048 * 256)]
    rt.launch_kernel_recorded(vp(2), args, (4, 12, 1), (128, 1, 1), 1024)
    assert flags[0] >> LAUNCH_CLUSTER_SHIFT > 1 and flags[0] & LAUNCH_PROGRAMMATIC == (0 if off else LAUNCH_PROGRAMMATIC)


LENGTHS = [1, 15, 16, 17, 127, 128, 129, 255, 257, 385, 600]


@pytest.mark.gpu
@pytest.mark.parametrize("heads", [(12, 2, 128), (8, 8, 64), (8, 1, 256), (16, 1, 64), (22, 2, 128), (32, 2, 128)])
@pytest.mark.parametrize("route", [(2, 1), (5, 1), (16, 1), (3, 2), (16, 2), (37, 0)])
@pytest.mark.parametrize("append", [True, False], ids=["append", "attend"])
def test_lean_kernels_match_the_oracle(cuda_runtime, codegen, heads, route, append):
    """Every length at which a block, a warp's turn or a part starts or ends, two layers on one cache.  fp32 sums of fp16
    products: 2e-5 of the result's norm; the newest rows are the projections' bits."""
    Hq, Hkv, D = heads
    if not route[1] and Hq // Hkv > 8:
        pytest.skip("split and combine serve groups of up to eight heads")
    if route[1] == 2 and D == 64:
        pytest.skip("no half blocks of 64-wide heads")
    B = len(LENGTHS) if route[1] else 1
    rng = np.random.default_rng(7)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    S = 640
    ex = DecodeAttentionExecutor(cuda_runtime, codegen, {"attention.head_count": Hq, "attention.head_count_kv": Hkv,
                                                         "attention.key_length": D}, B, S, 2, n_kv_buffers=1,
                                 with_append=append, lean=route, **({} if route[1] else {"num_splits": 148}))
    try:
        q, k0, v0 = f16(2, B, Hq, D), f16(B, S, Hkv, D), f16(B, S, Hkv, D)
        kn, vn = f16(2, B, Hkv, D), f16(2, B, Hkv, D)
        for lengths in ([LENGTHS] if B > 1 else [[n] for n in LENGTHS]):
            off, k, v = np.array(lengths, dtype=np.int32) - 1, k0.copy(), v0.copy()
            for b, n in enumerate(lengths):
                k[b, n:], v[b, n:] = np.inf, np.nan                   # nothing behind the end counts
            ex.upload_cache(0, k, v)
            for l in range(2):
                ex.upload_layer(l, q[l])
                ex.upload_new_kv(l, kn[l], vn[l])
            out = ex.execute_decode_batch(off)
            assert ex.kernel_launches_per_step == (2 if route[1] else 4)
            for l in range(2):
                for b, n in enumerate(lengths):
                    if append:
                        k[b, n - 1], v[b, n - 1] = kn[l, b], vn[l, b]
                ref = orc.decode_attention(q[l], np.where(np.isfinite(k), k, 0), np.where(np.isfinite(v), v, 0), off)
                assert np.linalg.norm(out[l] - ref) <= 2e-5 * np.linalg.norm(ref)
            got_k, got_v = ex.download_cache_rows(0, 0, S)
            assert np.array_equal(got_k.view(np.uint16), k[0].view(np.uint16)) and np.array_equal(got_v.view(np.uint16), v[0].view(np.uint16))
    finally:
        ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("heads,S", [((32, 8, 64), 16384), ((8, 1, 64), 131072)])
def test_the_lean_split_is_as_exact_as_the_dispatcher_s(cuda_runtime, codegen, heads, S):
    """64-wide heads: no further from 64-bit sums than the launches that the route replaces (the products of the low parts
    of P chained with those of the high parts were, by 10 to 22 %)."""
    Hq, Hkv, D = heads
    rng = np.random.default_rng([0, S, Hq])
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    q, k, v, off = f16(1, Hq, D), f16(1, S, Hkv, D), f16(1, S, Hkv, D), np.array([S - 1], dtype=np.int32)
    ref, error = orc.decode_attention(q, k, v, off, dtype=np.float64), []
    for lean in ((148 // Hkv, 0), (0, 0)):
        ex = DecodeAttentionExecutor(cuda_runtime, codegen, {"attention.head_count": Hq, "attention.head_count_kv": Hkv,
                                                             "attention.key_length": D}, 1, S, 1, lean=lean)
        try:
            ex.upload_layer(0, q, k, v)
            error.append(np.linalg.norm(ex.execute_decode_batch(off)[0] - ref))
        finally:
            ex.cleanup()
    assert error[0] <= error[1]


@pytest.mark.gpu
@pytest.mark.parametrize("heads,B,S,route,kw", [
    ((12, 2, 128), 3, 700, (8, 1), {}), ((12, 2, 128), 1, 4096, (37, 0), dict(rope="fused-append")),
    ((12, 2, 128), 1, 4096, (16, 1), dict(rope="fused")), ((32, 8, 64), 5, 300, (3, 1), dict(with_append=True)),
    ((8, 2, 256), 4, 300, (5, 2), dict(fuse_append=True)), ((32, 2, 128), 4, 2048, (6, 1), dict(with_append=True))])
def test_partials_after_a_routed_step_are_the_step_s_own(cuda_runtime, codegen, heads, B, S, route, kw):
    """Bit for bit what the dispatcher's own launches leave, although Q, offsets, new rows and caches change between the
    step and the call; neither the outputs nor the caches change with the call, twice in a row."""
    Hq, Hkv, D = heads
    meta = {"attention.head_count": Hq, "attention.head_count_kv": Hkv, "attention.key_length": D}
    rng = np.random.default_rng(B)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    k, v, steps = f16(B, S, Hkv, D), f16(B, S, Hkv, D), []
    for _ in range(2):
        steps.append((f16(2, B, Hq, D), f16(2, B, Hkv, D), f16(2, B, Hkv, D), rng.integers(S // 2, S, B).astype(np.int32)))
    got = []
    for lean in (route, (0, 0)):
        ex = DecodeAttentionExecutor(cuda_runtime, codegen, meta, B, S, 2, n_kv_buffers=1, lean=lean, **kw)
        try:
            ex.upload_cache(0, k, v)

            def rows_and_q(q, kn, vn):
                for l in range(2):
                    ex.upload_layer(l, q[l])
                    ex.upload_new_kv(l, kn[l], vn[l])
            mine = []
            for i, (q, kn, vn, off) in enumerate(steps):
                rows_and_q(q, kn, vn)
                out = ex.execute_decode_batch(off)
                caches = ex.download_cache_rows(0, 0, S)
                rows_and_q(*steps[1 - i][:3])                        # the next step's inputs
                ex._update_staging_buffers(steps[1 - i][3])
                if i:
                    ex.upload_cache(0, v, k)
                partials = ex.read_partials()
                again = ex.read_partials()
                assert all(np.array_equal(a, b) for a, b in zip(partials, again))
                if not i:
                    left = np.empty_like(out)
                    cuda_runtime.safe_memcpy_device_to_host(left, ctypes.c_void_p(ex.out_all.ptr), "output")
                    assert np.array_equal(left, out)
                    assert all(np.array_equal(a, b) for a, b in zip(caches, ex.download_cache_rows(0, 0, S)))
                mine.append(partials)
            got.append(mine)
        finally:
            ex.cleanup()
    for a, b in zip(*got):
        m, l, o = zip(a, b)
        used = l[1] > 0
        assert used.any() and np.array_equal(used, l[0] > 0)
        assert np.array_equal(m[0][used], m[1][used]) and np.array_equal(l[0], l[1]) and np.array_equal(o[0][used], o[1][used])


@pytest.mark.gpu
@pytest.mark.parametrize("rope", ["off", "fused-append"])
@pytest.mark.parametrize("from_host", [False, True])
def test_each_step_takes_the_route_that_its_lengths_ask_for(cuda_runtime, codegen, rope, from_host):
    """Steps of one executor, long among short and all short in turn: the oracle's outputs, the newest rows, the step's own
    partials, and as many launches as the route has.  fp32 sums of fp16 products: 2e-5 of the result's norm."""
    heads, B, S, L = (8, 2, 256), 16, 16384, 2
    Hq, Hkv, D = heads
    rng = np.random.default_rng(2)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    k, v = np.zeros((B, S, Hkv, D), np.float16), np.zeros((B, S, Hkv, D), np.float16)
    k[:, :600], v[:, :600], k[3], v[3] = f16(B, 600, Hkv, D), f16(B, 600, Hkv, D), f16(S, Hkv, D), f16(S, Hkv, D)
    ex = DecodeAttentionExecutor(cuda_runtime, codegen, {"attention.head_count": Hq, "attention.head_count_kv": Hkv,
                                                         "attention.key_length": D}, B, S, L, n_kv_buffers=1, with_append=True, rope=rope)
    if rope != "off":
        cos, sin = orc.rope_tables(S, D, 1e6)
    try:
        ex.upload_cache(0, k, v)
        for step, longest in enumerate((500, S - 3, 500, S - 2)):
            q, kn, vn = f16(L, B, Hq, D), f16(L, B, Hkv, D), f16(L, B, Hkv, D)
            off = rng.integers(300, 500, B).astype(np.int32)
            off[3] = longest - 1
            for l in range(L):
                ex.upload_new_kv(l, kn[l], vn[l])
                ex.upload_layer(l, q[l])
            out = ex.execute_decode_batch(off, q if from_host else None)
            skewed = longest > 500
            assert (ex.route_name is None) == skewed
            assert ex.kernel_launches_per_step == (L * (2 if rope != "off" else 3) if skewed else L)
            for l in range(L):
                ql, kl = (q[l], kn[l]) if rope == "off" else orc.rope_step(q[l], kn[l], cos, sin, off, 0, D)
                orc.kv_cache_append(kl, vn[l], k, v, off)
                ref = orc.decode_attention(ql, k, v, off)
                assert np.linalg.norm(out[l] - ref) <= 2e-5 * np.linalg.norm(ref)
            m, lsum, o = ex.read_partials()
            w = np.exp(np.where(lsum > 0, m, -np.inf) - m.max(axis=2, keepdims=True))
            whole = (np.where(lsum > 0, w, 0)[..., None] * np.where((lsum > 0)[..., None], o, 0)).sum(axis=2) / (w * lsum).sum(axis=2)[..., None]
            assert np.linalg.norm(whole - out[L - 1]) <= 2e-5 * np.linalg.norm(out[L - 1])
        rows_k, rows_v = ex.download_cache_rows(0, 3, S - 1)
        assert np.array_equal(rows_k, k[3, :S - 1]) and np.array_equal(rows_v, v[3, :S - 1])
    finally:
        ex.cleanup()


@pytest.mark.gpu
def test_partials_of_more_items_than_sms_each_time(cuda_runtime, codegen):
    """256 work items, one split: the launch behind read_partials draws them from a queue, whose ticket is zero every time."""
    B, S, Hkv, D = 32, 128, 8, 256
    rng = np.random.default_rng(1)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    q, k, v = f16(B, Hkv, D), f16(B, S, Hkv, D), f16(B, S, Hkv, D)
    ex = DecodeAttentionExecutor(cuda_runtime, codegen, {"attention.head_count": Hkv, "attention.head_count_kv": Hkv,
                                                         "attention.key_length": D}, B, S, 1, lean=(2, 1))
    try:
        ex.upload_layer(0, q, k, v)
        for _ in range(3):
            off = rng.integers(0, S, B).astype(np.int32)
            out = ex.execute_decode_batch(off)[0]
            m, l, o = ex.read_partials()
            assert m.shape == (B, Hkv, 1)
            whole = o[:, :, 0] / l
            assert np.linalg.norm(whole - out) <= 2e-5 * np.linalg.norm(out)
            assert np.linalg.norm(out - orc.decode_attention(q, k, v, off)) <= 2e-5 * np.linalg.norm(out)
    finally:
        ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("rope_type,rotary", [(0, 0), (1, 0), (2, 32), (2, 64)])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("route", [(6, 1), (6, 2), (37, 0)], ids=["cluster", "half", "split"])
def test_rotation_in_the_lean_kernels_gives_the_separate_launch_s_bits(cuda_runtime, codegen, route, D, rope_type, rotary):
    """The rotated row in the cache is the standalone rotation's, bit for bit, and so are the outputs of the same route, which
    are the oracle's: fp32 sums of fp16 products, 2e-5 of the result's norm."""
    if route[1] == 2 and D == 64:
        pytest.skip("no half blocks of 64-wide heads")
    meta = {"attention.head_count": 12, "attention.head_count_kv": 2, "attention.key_length": D, "rope_type": rope_type}
    if rotary:
        meta["rotary_dim"] = rotary
    rng = np.random.default_rng(3)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    B, S, kw = (2, 300, {}) if route[1] else (1, 300, {"num_splits": 148})
    q, k, v, kn, vn = f16(B, 12, D), f16(B, S, 2, D), f16(B, S, 2, D), f16(B, 2, D), f16(B, 2, D)
    off, got = np.array([250, 16], dtype=np.int32)[:B], []
    cos, sin = orc.rope_tables(S, rotary or D, 1e6)
    q_rot, k_rot = orc.rope_step(q, kn, cos, sin, off, rope_type, rotary or D)
    ref_k, ref_v = k.copy(), v.copy()
    orc.kv_cache_append(k_rot, vn, ref_k, ref_v, off)
    ref = orc.decode_attention(q_rot, ref_k, ref_v, off)
    for rope in ("separate", "fused", "fused-append"):
        ex = DecodeAttentionExecutor(cuda_runtime, codegen, meta, B, S, 1, rope=rope, lean=route, **kw)
        try:
            ex.upload_layer(0, q, k, v)
            ex.upload_new_kv(0, kn, vn)
            out = ex.execute_decode_batch(off)
            assert ex.kernel_launches_per_step == (1 if route[1] else 2) + (rope == "separate")
            got.append((out, *ex.download_cache_rows(0, 0, 251)))
            m, l, o = ex.read_partials()                             # the split launch's, on demand
            assert np.isfinite(m).all() and l.max() > 0
        finally:
            ex.cleanup()
    assert np.linalg.norm(got[0][0][0] - ref) <= 2e-5 * np.linalg.norm(ref) and np.array_equal(got[0][1][250], k_rot[0])
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)


@pytest.mark.gpu
def test_an_infinite_value_stays_infinite_in_a_cluster(cuda_runtime, codegen):
    """As fp32 products give it: infinite where its weight is not zero, the other columns finite."""
    rng = np.random.default_rng(5)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    q, k, v = f16(1, 12, 128), f16(1, 200, 2, 128), f16(1, 200, 2, 128)
    v[0, 3, 0, 5], v[0, 199, 1, 7] = np.inf, -np.inf
    ex = DecodeAttentionExecutor(cuda_runtime, codegen, {"attention.head_count": 12, "attention.head_count_kv": 2,
                                                         "attention.key_length": 128}, 1, 200, 1, lean=(8, 1))
    try:
        ex.upload_layer(0, q, k, v)
        out = ex.execute_decode_batch(np.array([199], dtype=np.int32))[0, 0]
    finally:
        ex.cleanup()
    assert np.all(out[:6, 5] == np.inf) and np.all(out[6:, 7] == -np.inf)
    out[:6, 5], out[6:, 7] = 0, 0
    assert np.isfinite(out).all()


@pytest.mark.gpu
def test_a_cluster_kernel_refuses_a_launch_without_its_clusters(cuda_runtime, codegen):
    """The grid's clusters have to be the parts: otherwise the status word says so and nothing is written."""
    meta = {"attention.head_count": 12, "attention.head_count_kv": 2, "attention.key_length": 128}
    ex = DecodeAttentionExecutor(cuda_runtime, codegen, meta, 1, 256, 1, lean=(4, 1))
    try:
        ex._choose_route()
        fn, args, grid, block, smem = ex._route.launches(0, ex.tensor_mapping, ex.offsets.ptr, 1)[0]
        module = codegen.load_kernel_safe(cuda_runtime, 'decode_attention', cuda_runtime.get_gpu_architecture(), ex._route.name)[0]
        ex._update_staging_buffers(np.array([200], dtype=np.int32))
        cuda_runtime.launch_kernel_recorded(fn, args, tuple(grid), block, smem)
        with pytest.raises(Exception, match="bounded wait"):
            ex.dispatcher_check()
        # without a status word of its own: the runtime's, as launches of flash_attention_kernel get it, or the module's
        for word, wait in ((ctypes.addressof(cuda_runtime._launch_status), cuda_runtime.stream_synchronize),
                           (0, lambda: cuda_runtime.module_check_status(module))):
            wait()
            args[19] = ctypes.c_void_p(word)
            cuda_runtime.launch_kernel_recorded(fn, args, tuple(grid), block, smem)
            with pytest.raises(Exception, match="bounded wait"):
                wait()
            wait()
    finally:
        ex.cleanup()


@pytest.mark.gpu
@pytest.mark.parametrize("heads,B,S", [((12, 2, 128), 3, 700), ((28, 4, 128), 64, 300), ((8, 2, 256), 5, 1000), ((32, 8, 64), 7, 520)])
@pytest.mark.parametrize("f32", [True, False])
def test_balanced_calls_through_the_direct_entry_point(cuda_runtime, heads, B, S, f32):
    """Calls that go to clusters (64 sequences of four KV heads to more than run at once), behind an append, with an output
    aligned to its element only: the oracle's result, the scratch untouched.  fp16 outputs are rounded once."""
    from vte_b200.bridge.cuda_runtime import ATTN_BALANCED, ATTN_PROGRAMMATIC
    rt, (Hq, Hkv, D) = cuda_runtime, heads
    rng = np.random.default_rng(B)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    q, k, v, kn, vn = f16(B, Hq, D), f16(B, S, Hkv, D), f16(B, S, Hkv, D), f16(B, Hkv, D), f16(B, Hkv, D)
    off = rng.integers(1, S + 1, B).astype(np.int32) - 1
    off[0], off[1], off[2] = S - 1, 0, 0
    bufs, dt, C = [], np.float32 if f32 else np.float16, 8

    def dev(a):
        bufs.append(rt.safe_malloc(a.nbytes + 16, "direct entry output"))
        rt.safe_memcpy_host_to_device(bufs[-1], np.ascontiguousarray(a), "direct entry output")
        return bufs[-1]
    try:
        dq, dk, dv, dkn, dvn, doff, dout = (dev(x) for x in (q, k, v, kn, vn, off, np.zeros((B, Hq, D), dt)))
        out_at = ctypes.c_void_p(dout.value + np.dtype(dt).itemsize)
        mark = np.full(B * Hq * C * D, 7.0, np.float32)
        pm, pl, po, work = dev(mark[:B * Hq * C]), dev(mark[:B * Hq * C]), dev(mark), dev(np.zeros(4, np.int32))
        stride = S * Hkv * D
        for _ in range(2):
            rt.kv_cache_append(dkn, dvn, dk, dv, doff, B, Hkv, D, stride)
            rt.split_kv_decode(dq, dk, dv, doff, out_at, f32, pm, pl, po, work, B, Hq, Hkv, D, 1 / math.sqrt(D), stride, C, 0,
                               ATTN_BALANCED | ATTN_PROGRAMMATIC)
        rt.check_status(work)
        out, left = np.zeros((B, Hq, D), dt), np.zeros_like(mark)
        rt.safe_memcpy_device_to_host(out, out_at, "direct entry output")
        rt.safe_memcpy_device_to_host(left, po, "direct entry output")
    finally:
        for p in bufs:
            rt.safe_free(p, "direct entry cleanup")
    assert np.array_equal(left, mark)
    orc.kv_cache_append(kn, vn, k, v, off)
    ref = orc.decode_attention(q, k, v, off)
    assert np.linalg.norm(out - ref) <= (2e-5 if f32 else 5e-4) * np.linalg.norm(ref)


@pytest.mark.gpu
@pytest.mark.parametrize("heads,B,S,clusters", [((28, 4, 128), 32, 4096, True), ((12, 2, 128), 8, 2048, True), ((12, 2, 128), 32, 32768, False),
                                                ((8, 2, 256), 16, 16384, False)])
def test_balanced_calls_that_a_long_sequence_could_slow_keep_the_equal_shares(cuda_runtime, heads, B, S, clusters):
    """The entry point sees no lengths.  Launches are captured and counted, not run: one of clusters, or split and combine,
    which a caller gets in any case who names the number of CTAs."""
    from vte_b200.bridge.cuda_runtime import ATTN_BALANCED, ATTN_PROGRAMMATIC
    rt, (Hq, Hkv, D) = cuda_runtime, heads
    p = rt.safe_malloc(4096, "direct entry output")
    try:
        for n_ctas, nodes in ((0, 1 if clusters else 2), (rt.get_num_cus(), 2)):
            rt.stream_begin_capture()
            rt.split_kv_decode(p, p, p, p, p, True, p, p, p, p, B, Hq, Hkv, D, 1 / math.sqrt(D), S * Hkv * D, 8, 0,
                               ATTN_BALANCED | ATTN_PROGRAMMATIC, n_ctas)
            graph = rt.stream_end_capture()
            assert rt.graph_node_count(graph) == nodes
            rt.graph_destroy(graph)
    finally:
        rt.safe_free(p, "direct entry cleanup")
