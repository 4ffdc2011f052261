"""Products of long passes in tiles shared by two CTAs: passes large enough to take them, with rows and columns that end
inside a tile, against the same prompt in portions too small for them."""
import numpy as np
import pytest

import ctox_llm_b200 as ctox
from ctox_llm_b200 import native as N
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,width,ff", [(1500, 2056, 8200), (1409, 1032, 16520), (1281, 2048, 8192)])
def test_large_pass_equals_portions(n, width, ff):
    """n = 1409, 1281: one row past a tile of 128, so that the second CTA of the last pair has one row or none. Every
    product sums in the same order whatever its tile; attention sees other tiles, rounded to bf16 (1e-2, as between the
    16-bit kernels and the plain implementation)."""
    be = ctox.B200Backend(0)
    spec = dict(rope_base=1e4, mixer=N.MIXER_LATENT_ATTENTION, heads=8, dim=64, rot_dim=32, vdim=64, q_rank=256, kv_rank=128,
                window=300, kv_from=-1, score_scale=96 ** -0.5, mlp=N.MLP_RELU2, ff=ff)
    ex = ctox.B200Executor(be, ctox.StackConfig(vocab_size=500, hidden_size=width, norm_eps=1e-6, logit_softcap=30.0,
                                                layers=[N.LayerConfig(**spec) for _ in range(2)], max_context_tokens=1600))
    try:
        ex.fill_synthetic(3)
        ex.warmup()
        tokens = [int(t) for t in np.random.default_rng(n).integers(0, 500, n)]
        want = [0, 127, 128, 700, n - 2, n - 1]
        whole = ex.extend(tokens, want)
        ex.reset_session()
        parts = []
        for a in range(0, n, 100):
            here = [w - a for w in want if a <= w < a + 100]
            rows = ex.extend(tokens[a:a + 100], here) if here else ex.extend(tokens[a:a + 100])
            if here:
                parts += list(rows)
        for got, ref in zip(whole, parts):
            assert rel_l2(got, ref) <= 1e-2
    finally:
        ex.unload()
        be.close()
