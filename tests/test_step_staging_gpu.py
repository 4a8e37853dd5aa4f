"""An end-to-end step's staging copies as launches."""
import numpy as np
import pytest

from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 3, 5], ids=lambda b: f"{b}_sequences")
def test_staging_by_launch_and_by_copy_node_give_the_same_step(cuda_runtime, codegen, batch, monkeypatch):
    """4, 12 and 20 bytes of offsets: the last 16-byte word of the copy is a part of one, one, and more than one.
    Both routes run the same attention launches on the same bytes, so the outputs are the same bits."""
    from vte_b200.core import decode_executor as de
    meta = {"attention.head_count": 12, "attention.head_count_kv": 2, "attention.key_length": 128}
    rng = np.random.default_rng(batch)
    f16 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(np.float16)
    S, L = 300, 2
    k, v = f16(batch, S, 2, 128), f16(batch, S, 2, 128)
    steps = [(f16(L, batch, 12, 128), rng.integers(0, S, size=batch).astype(np.int32)) for _ in range(3)]
    got = []
    for limit in (de.STAGE_COPY_MAX_BYTES, 0):
        monkeypatch.setattr(de, "STAGE_COPY_MAX_BYTES", limit)
        ex = de.DecodeAttentionExecutor(cuda_runtime, codegen, meta, batch, S, L, n_kv_buffers=1)
        try:
            ex.upload_cache(0, k, v)
            got.append([ex.execute_decode_batch(off, q).copy() for q, off in steps])
        finally:
            ex.cleanup()
    for by_launch, by_node, (q, off) in zip(*got, steps):
        assert np.array_equal(by_launch, by_node)
        for l in range(L):
            assert np.max(np.abs(by_launch[l] - orc.decode_attention(q[l], k, v, off))) <= 1e-5


def test_queued_steps_keep_their_own_offsets(cuda_runtime, codegen):
    """More steps in flight than there are staging slots, each appending at its own position: every row is written."""
    from vte_b200.core import decode_executor as de
    n, S = 2 * de.OFFSET_SLOTS + 5, 256
    ex = de.DecodeAttentionExecutor(cuda_runtime, codegen, {"attention.head_count": 12, "attention.head_count_kv": 2,
                                                            "attention.key_length": 128}, 2, S, 3, n_kv_buffers=1, with_append=True)
    try:
        rng = np.random.default_rng(0)
        new = [rng.standard_normal((2, 2, 128), dtype=np.float32).astype(np.float16) for _ in range(2)]
        zero = np.zeros((2, S, 2, 128), np.float16)
        ex.upload_cache(0, zero, zero)
        for l in range(3):
            ex.upload_layer(l, np.zeros((2, 12, 128), np.float16))
            ex.upload_new_kv(l, *new)
        for i in range(n):
            ex.execute_decode_batch(np.array([i, S - 1 - i], dtype=np.int32), read_output=False)
        cuda_runtime.stream_synchronize()
        k, v = ex.download_cache_rows(0, 0, S)
        assert np.array_equal(k[:n], np.broadcast_to(new[0][0], (n, 2, 128))) and not k[n:].any()
        k, v = ex.download_cache_rows(0, 1, S)
        assert np.array_equal(v[S - n:], np.broadcast_to(new[1][1], (n, 2, 128))) and not v[:S - n].any()
        ex.dispatcher_check()
    finally:
        ex.cleanup()
