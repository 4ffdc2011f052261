"""Portions appended to a long session: the long pass cuts the context into parts where its groups of positions leave SMs
idle. Against short passes of eight tokens over the same session, in values and in time."""
import time

import numpy as np
import pytest

import ctox_llm_b200 as ctox
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu

GEOMETRIES = {
    # six queries per KV head: groups of five positions on the tensor-core kernel
    "mma-6": dict(num_attention_heads=24, num_key_value_heads=4, head_dim=256, rotary_dim=64, kv_dtype=ctox.BF16),
    "mma-16": dict(num_attention_heads=16, num_key_value_heads=8, head_dim=256, rotary_dim=64, kv_dtype=ctox.BF16),
    "cores-f32": dict(num_attention_heads=8, num_key_value_heads=2, head_dim=128, rotary_dim=32, kv_dtype=ctox.F32),
    "cores-6": dict(num_attention_heads=24, num_key_value_heads=4, head_dim=256, rotary_dim=64, kv_dtype=ctox.F32),
    "cores-bf16": dict(num_attention_heads=12, num_key_value_heads=2, head_dim=64, rotary_dim=16, kv_dtype=ctox.BF16),
}


def executor(geometry, context, **kw):
    be = ctox.B200Backend(0)
    cfg = dict(vocab_size=2048, hidden_size=1024, intermediate_size=1024, num_hidden_layers=2, full_attention_interval=2,
               linear_num_key_heads=4, linear_num_value_heads=8, max_context_tokens=context + 1024, max_draft_tokens=0,
               mtp_num_hidden_layers=0, draft_vocab=0, **GEOMETRIES[geometry])
    ex = ctox.B200Executor(be, ctox.qwen38_27b_config(**{**cfg, **kw}))
    ex.fill_synthetic(5)
    ex.warmup()
    return be, ex


@pytest.mark.parametrize("geometry", GEOMETRIES)
@pytest.mark.parametrize("position", [1, 130, 5003])
def test_portion_on_a_long_session(geometry, position):
    """Every part of the context is a sum in 32 bits, merged in 32 bits: 1e-4 of the logits as for the whole pass; through a
    16-bit cache 1e-3 (keys of the portion that round the other way)."""
    be, ex = executor(geometry, position)
    bound = 1e-4 if GEOMETRIES[geometry]["kv_dtype"] == ctox.F32 else 1e-3
    try:
        for n in (17, 26, 40, 200, 513):
            tokens = [int(t) for t in np.random.default_rng(n).integers(0, 2048, n)]
            ex.prefill_synthetic(position, 3)
            before = be.kernel_launches()
            ex.extend(tokens)
            launches = be.kernel_launches() - before
            assert launches < 30 or (n < 26 and position > 2048 and geometry.startswith("cores")), "one long pass"
            ex.prefill_synthetic(position, 3)
            whole = ex.extend(tokens, list(range(n)))
            ex.prefill_synthetic(position, 3)
            short = [row for a in range(0, n, 8) for row in ex.extend(tokens[a:a + 8], list(range(min(8, n - a))))]
            assert max(rel_l2(a, b) for a, b in zip(whole, short)) <= bound
    finally:
        ex.unload()
        be.close()


@pytest.mark.parametrize("geometry", GEOMETRIES)
@pytest.mark.parametrize("n", [17, 26, 64])
def test_portion_on_a_long_session_takes_no_longer(geometry, n):
    """On 30000 tokens, attention in every layer: not slower than the short passes it replaces (a tenth for the clock).
    Without parts a CTA per KV head and group walked the whole context: 18 ms where short passes took 1.2."""
    be, ex = executor(geometry, 30000, full_attention_interval=1)
    try:
        ex.prefill_synthetic(30000, 3)
        tokens = [int(t) for t in np.random.default_rng(n).integers(0, 2048, n)]
        best = [1e9, 1e9]
        for _ in range(5):
            for i, step in enumerate((n, 8)):
                t0 = time.perf_counter()
                for a in range(0, n, step):
                    ex.extend(tokens[a:a + step])
                best[i] = min(best[i], time.perf_counter() - t0)
        assert best[0] <= 1.1 * best[1], best
    finally:
        ex.unload()
        be.close()
