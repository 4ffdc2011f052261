"""Groups of four tokens in the scan of a long pass, against the short passes' recurrence token by token."""
import numpy as np
import pytest

import ctox_llm_b200 as ctox
from gpu_util import rel_l2
from oracle_model import OracleModel, tiny_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,qk_heads", [(2, 2), (4, 2), (6, 2)])
@pytest.mark.parametrize("n", [17, 18, 19, 20, 32, 35, 49])
def test_groups_of_tokens(orc, n, heads, qk_heads):
    """n leaves every rest of a group of four and of a block of sixteen; the state left is what the next tokens' logits read.
    Sums of 128 products in 32 bits in another order: 1e-4, as for whole long passes."""
    be = ctox.B200Backend(0)
    cfg = tiny_config(max_context_tokens=128, kv_dtype=ctox.F32, linear_num_value_heads=heads, linear_num_key_heads=qk_heads)
    ex = ctox.B200Executor(be, cfg)
    try:
        OracleModel(orc, cfg, seed=8).load_into(ex)
        ex.warmup()
        tokens = [int(t) for t in np.random.default_rng(n).integers(0, cfg.vocab_size, n + 3)]
        runs = []
        for step in (n, 8):
            ex.reset_session()
            for a in range(0, n, step):
                ex.extend(tokens[a:min(a + step, n)])
            last = ex.last_hidden()
            runs.append([last, ex.extend(tokens[n:], [0, 1, 2])])
        for got, want in zip(*runs):
            assert rel_l2(got, want) <= 1e-4
    finally:
        ex.unload()
        be.close()
