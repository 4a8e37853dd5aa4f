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
