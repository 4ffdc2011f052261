"""Cancellation while a long pass is on its way: read between its layers, not only between passes."""
import threading
import time

import numpy as np
import pytest

import ctox_llm_b200 as ctox

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["extend", "prefill"])
def test_long_pass_is_cancelled_on_its_way(call):
    """One pass of 1000 tokens through 48 layers, cancelled after a third of its time: it returns before three quarters of it, the
    session is unusable until it is reset, and the reset session gives the bits of one that was never cancelled."""
    be = ctox.B200Backend(0)
    ex = ctox.B200Executor(be, ctox.qwen38_27b_config(
        vocab_size=2048, hidden_size=2048, intermediate_size=8192, num_hidden_layers=48, full_attention_interval=4, num_attention_heads=16,
        num_key_value_heads=4, head_dim=256, rotary_dim=64, linear_num_key_heads=8, linear_num_value_heads=16, max_context_tokens=1100,
        max_draft_tokens=0, mtp_num_hidden_layers=0, draft_vocab=0, kv_dtype=ctox.BF16))
    try:
        ex.fill_synthetic(4)
        ex.warmup()
        tokens = [int(t) for t in np.random.default_rng(3).integers(0, 2048, 1001 if call == "prefill" else 1000)]
        run = getattr(ex, call)

        def timed():
            ex.reset_session()
            token = ctox.CancellationToken()
            t0 = time.perf_counter()
            run(tokens, cancellation=token)
            return time.perf_counter() - t0

        full = min(timed() for _ in range(4))
        want = ex.last_hidden()
        ex.reset_session()
        token = ctox.CancellationToken()
        timer = threading.Thread(target=lambda: (time.sleep(full / 3), token.cancel()))
        t0 = time.perf_counter()
        timer.start()
        with pytest.raises(ctox.CtoxError) as e:
            run(tokens, cancellation=token)
        took = time.perf_counter() - t0
        timer.join()
        assert e.value.kind == "Cancelled" and took < 0.75 * full, (took, full)
        assert ex.session_state()["poisoned"]
        with pytest.raises(ctox.CtoxError):
            ex.extend(tokens[:20])
        timed()
        assert np.array_equal(ex.last_hidden(), want)
    finally:
        ex.unload()
        be.close()
