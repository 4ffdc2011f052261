"""The buffers of long passes are spare: an allocation that does not fit beside them gets them back, and the model that had
them runs short passes."""
import numpy as np
import pytest
import torch

import ctox_llm_b200 as ctox
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu


def executor(be, **kw):
    cfg = dict(vocab_size=2048, hidden_size=1024, intermediate_size=1024, num_hidden_layers=2, full_attention_interval=2,
               num_attention_heads=8, num_key_value_heads=2, head_dim=128, rotary_dim=32, linear_num_key_heads=4, linear_num_value_heads=8,
               max_context_tokens=2048, max_draft_tokens=0, mtp_num_hidden_layers=0, draft_vocab=0, kv_dtype=ctox.F32)
    return ctox.B200Executor(be, ctox.qwen38_27b_config(**{**cfg, **kw}))


def fill(leave):
    """Takes the device's free memory but for about `leave` bytes."""
    held = []
    for chunk in (1 << 30, 64 << 20, 2 << 20):
        while torch.cuda.mem_get_info()[0] >= leave + chunk:
            n = (torch.cuda.mem_get_info()[0] - leave) // chunk * chunk
            if n < 10 << 20:  # torch takes 20 MB from the device for a request of 1 to 10 MB, and 2 MB for two of 1 MB
                held += [torch.empty(1 << 20, dtype=torch.uint8, device="cuda") for _ in range(n >> 20)]
            else:
                held.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
    return held


@pytest.mark.parametrize("second", [True, False])
def test_spare_buffers_are_given_back(second):
    """Beside 250 MB of buffers: a second executor whose caches take 200 MB, and the first one's logits (13 MB), with 64 and 4
    MB left on the device. The first executor's results stay (32-bit sums in another order: 1e-4)."""
    torch.zeros(1, device="cuda")
    be = ctox.B200Backend(0)
    first = executor(be, intermediate_size=17408, vocab_size=400000 if not second else 2048)
    other = executor(be, max_context_tokens=100000, num_hidden_layers=1, full_attention_interval=1) if second else None
    held = []
    try:
        first.fill_synthetic(1)
        if second:
            other.fill_synthetic(2)
        first.warmup()
        tokens = [int(t) for t in np.random.default_rng(1).integers(0, 2048, 100)]
        first.extend(tokens)
        want, before = first.last_hidden(), be.allocated_bytes()
        launches = be.kernel_launches()
        first.reset_session()
        first.extend(tokens)
        assert be.kernel_launches() - launches < 30, "one long pass"
        first.reset_session()
        held = fill((64 if second else 4) << 20)
        if second:
            other.warmup()
            assert other.extend(tokens, [99]).any()
            first.extend(tokens)
        else:
            assert first.extend(tokens, [0, 99]).any()
        assert be.allocated_bytes() < before + (220 << 20)
        assert rel_l2(first.last_hidden(), want) <= 1e-4
        held.clear()
        torch.cuda.empty_cache()
        first.warmup()  # and taken again
        launches = be.kernel_launches()
        first.extend(tokens)
        assert be.kernel_launches() - launches < 30, "one long pass"
        assert rel_l2(first.last_hidden(), want) <= 1e-6
    finally:
        held.clear()
        torch.cuda.empty_cache()
        first.unload()
        if other:
            other.unload()
        assert be.allocated_bytes() == 0
        be.close()
