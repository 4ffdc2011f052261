"""Long passes of the hybrid model (tensor-core products, row kernels, token scan) against short passes of
eight tokens over the same weights: logits, and what speculative blocks do with the state and caches left."""
import numpy as np
import pytest

import ctox_llm_b200 as ctox
from gpu_util import rel_l2
from oracle_model import OracleModel, tiny_config

pytestmark = pytest.mark.gpu


CONFIGS = {
    # widths that are not whole tiles of 128 rows or 256 columns; CUDA-core attention over both cache types
    "ragged-f32": dict(kv_dtype=ctox.F32, hidden_size=320, intermediate_size=704),
    "ragged-bf16": dict(kv_dtype=ctox.BF16, hidden_size=320, intermediate_size=704),
    # the tensor-core attention kernel; every second layer attention; groups of eight positions, and of five
    "head256": dict(num_attention_heads=4, num_key_value_heads=1, head_dim=256, rotary_dim=64, kv_dtype=ctox.BF16,
                    full_attention_interval=2),
    "head256-6": dict(num_attention_heads=6, num_key_value_heads=1, head_dim=256, rotary_dim=64, kv_dtype=ctox.BF16,
                      full_attention_interval=2),
}


@pytest.mark.parametrize("name", CONFIGS)
@pytest.mark.parametrize("n", [17, 18, 31, 63, 65, 129, 300, 1025 + 40])
def test_long_pass_equals_short_passes(orc, name, n):
    """n crosses the groups of 5 and 8 positions and of 16 tokens, and the 1024 positions of one pass; at these widths the
    products take tiles of 32 to 112 positions, one to ten of them (test_packed_pair_gpu.py has the wide ones). Both sides sum the same products in 32 bits in another order: 1e-4 of the logits for a 32-bit
    cache; rounding keys and values to 16 bits turns such differences into steps of 2^-9 (1e-3, the bound of the
    oracle's comparisons)."""
    be = ctox.B200Backend(0)
    cfg = tiny_config(max_draft_tokens=3, max_context_tokens=1200, **CONFIGS[name])
    model = OracleModel(orc, cfg, seed=4)
    ex = ctox.B200Executor(be, cfg)
    bound = 1e-4 if cfg.kv_dtype == ctox.F32 else 1e-3
    try:
        model.load_into(ex)
        ex.warmup()
        ex.keep_logits(True)
        prompt = [int(t) for t in np.random.default_rng(n).integers(0, cfg.vocab_size, n + 1)]
        want = sorted({0, 7, 8, n // 2, n - 2, n - 1})
        runs = []
        launches = {}
        for step in (n, 8):
            ex.reset_session()
            before = be.kernel_launches()
            for a in range(0, n, step):
                ex.extend(prompt[a:min(a + step, n)])
            launches[step] = be.kernel_launches() - before
            ex.reset_session()
            rows = []
            for a in range(0, n, step):
                b = min(a + step, n)
                here = [w - a for w in want if a <= w < b]
                if here:
                    rows += list(ex.extend(prompt[a:b], here))
                else:
                    ex.extend(prompt[a:b])
            assert ex.position() == n
            out = [np.stack(rows), ex.last_hidden()[None]]
            tok = prompt[n]
            for _ in range(2):  # the MTP cache and the recurrent state
                ex.decode(tok, mtp_enabled=True, force_accept=0)
                out += [ex.last_logits(0)[None], np.stack(ex.last_draft_logits()[:1]), np.stack(ex.last_mtp_hidden()[:1])]
            runs.append(out)
        assert launches[n] < 0.8 * launches[8], "a long pass where the other side has three short ones or more"
        for got, ref in zip(*runs):
            for g, r in zip(got, ref):
                assert rel_l2(g, r) <= bound
    finally:
        ex.unload()
        be.close()


def test_long_pass_on_top_of_a_session_matches_oracle(orc):
    """A long pass behind a short one and before another: positions, page offsets and carried state against the oracle."""
    be = ctox.B200Backend(0)
    cfg = tiny_config(max_draft_tokens=2)
    model = OracleModel(orc, cfg, seed=6)
    ex = ctox.B200Executor(be, cfg)
    try:
        model.load_into(ex)
        ex.warmup()
        prompt = [int(t) for t in np.random.default_rng(5).integers(0, cfg.vocab_size, 48)]
        _, exp_logits, _ = model.greedy(prompt, 1)
        ex.reset_session()
        ex.extend(prompt[:5])
        ex.extend(prompt[5:42])
        got = ex.extend(prompt[42:], [5])
        assert rel_l2(got[0], exp_logits[0]) <= 1e-3
    finally:
        ex.unload()
        be.close()


@pytest.mark.parametrize("kv", [ctox.F32, ctox.BF16])
@pytest.mark.parametrize("head_dim,heads,kv_heads", [(64, 4, 2), (64, 12, 2), (128, 4, 4), (128, 6, 1), (192, 4, 2)])
def test_attention_on_cuda_cores_matches_oracle(orc, head_dim, heads, kv_heads, kv):
    """Four, two and one groups of threads per head dimension; 8, 24 and 48 queries per CTA; a context that ends inside a tile
    of 32 tokens; long and short passes and single positions."""
    be = ctox.B200Backend(0)
    cfg = tiny_config(max_draft_tokens=2, num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=head_dim, rotary_dim=32,
                      kv_dtype=kv, full_attention_interval=2)
    model = OracleModel(orc, cfg, seed=8)
    ex = ctox.B200Executor(be, cfg)
    try:
        model.load_into(ex)
        ex.warmup()
        ex.keep_logits(True)
        prompt = [int(t) for t in np.random.default_rng(head_dim).integers(0, cfg.vocab_size, 75)]
        tokens, logits, _ = model.greedy(prompt, 2)
        for cuts in ((0, 75), (0, 8, 16, 60, 68, 75)):
            ex.reset_session()
            for a, b in zip(cuts, cuts[1:]):
                got = ex.extend(prompt[a:b], [b - a - 1])
            assert rel_l2(got[0], logits[0]) <= 1e-3
            ex.decode(tokens[0], mtp_enabled=True, force_accept=0)
            assert rel_l2(ex.last_logits(0), logits[1]) <= 1e-3
    finally:
        ex.unload()
        be.close()
