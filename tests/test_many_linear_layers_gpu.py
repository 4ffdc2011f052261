"""More linear-attention layers than one commit launch takes (128): a partly accepted block re-scans each layer by itself."""
import numpy as np
import pytest

import ctox_llm_b200 as ctox

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [128, 132])
@pytest.mark.parametrize("accepted", [0, 1, 2])
def test_partly_accepted_block_leaves_the_state_of_a_short_pass(layers, accepted):
    """The state after a block of which some drafts were accepted is, bit for bit, that of a pass over just these tokens: the
    re-scan takes the pass's own sums."""
    be = ctox.B200Backend(0)
    ex = ctox.B200Executor(be, ctox.qwen38_27b_config(
        vocab_size=512, hidden_size=256, intermediate_size=256, num_hidden_layers=layers, full_attention_interval=1000, num_attention_heads=4,
        num_key_value_heads=2, head_dim=64, rotary_dim=16, linear_num_key_heads=2, linear_num_value_heads=4, max_context_tokens=256,
        max_draft_tokens=3, mtp_num_hidden_layers=1, draft_vocab=0, kv_dtype=ctox.F32))
    try:
        ex.fill_synthetic(7)
        ex.warmup()
        prompt = [int(t) for t in np.random.default_rng(layers).integers(0, 512, 16)]
        ex.extend(prompt[:8])
        block = ex.decode(prompt[8], mtp_enabled=True, force_accept=accepted)
        assert ex.position() == 9 + accepted
        got = ex.extend(prompt[9:13], [0, 1, 2, 3])
        ex.reset_session()
        ex.extend(prompt[:8])
        ex.extend([prompt[8]] + list(block.accepted_draft_tokens))
        want = ex.extend(prompt[9:13], [0, 1, 2, 3])
        assert np.isfinite(want).all() and np.array_equal(got, want)
    finally:
        ex.unload()
        be.close()
