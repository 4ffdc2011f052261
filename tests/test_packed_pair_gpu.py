"""Products of long passes whose tiles are shared by two CTAs (more than 128 positions), Q2 and Q4, against 64 bits: one
layer whose mixer adds nothing, so that its two feed-forward products are nearly all that lies between the embedding
and the logits."""
import numpy as np
import pytest
import torch

import ctox_llm_b200 as ctox
from ctox_llm_b200 import native as N

pytestmark = pytest.mark.gpu

# 79 blocks of columns (not whole super-tiles of 256) and 39.5 tiles of 128 output rows; 71 tiles of rows and 71 blocks
HIDDEN, FF, VOCAB = 5056, 4544, 512


def packed(rng, dtype, rows, cols, gain, s_in=None, s_out=None):
    """Random canonical blocks [f16 scale][codes], and what they stand for without recovery scales."""
    out = torch.randint(0, 256, (rows, cols // 64, 34 if dtype == N.Q4B64 else 18), device="cuda", generator=rng, dtype=torch.uint8)
    scale = (torch.exp(torch.randn(rows, cols // 64, 1, device="cuda", generator=rng) * 0.5) * (gain * 1.4 / cols ** 0.5)).half()
    f16 = lambda n: (torch.rand(n, device="cuda", generator=rng) * 0.5 + 0.75).half()
    return dict(dtype=dtype, blocks=out, scale=scale, s_in=f16(cols) if s_in is None else s_in, s_out=f16(rows) if s_out is None else s_out)


def operation(m):
    m["blocks"][:, :, :2] = m["scale"].view(torch.uint8)
    host = lambda t: t.contiguous().view(torch.uint8).reshape(-1).cpu().numpy()
    return ctox.FusedMatVec(m["dtype"], host(m["blocks"]), m["s_out"].numel(), m["s_in"].numel(), None, s_in=host(m["s_in"]),
                            s_out=host(m["s_out"]))


def values(m):
    codes = m["blocks"][:, :, 2:]
    if m["dtype"] == N.Q4B64:
        q = (torch.stack([codes & 15, codes >> 4], -1).double() - 7.5) / 7.5
    else:
        q = (torch.stack([(codes >> s) & 3 for s in (0, 2, 4, 6)], -1).double() * 2 - 3) / 3
    q = q.reshape(*m["scale"].shape[:2], 64) * m["scale"].double()
    return q.reshape(m["s_out"].numel(), -1) * m["s_in"].double() * m["s_out"].double()[:, None]


def model(dtype, outlier):
    """outlier > 0: one column of either product's input is about 2^outlier times the others, and the weights of the 64
    columns around it are zero, so that the outputs are made of the others alone."""
    rng = torch.Generator(device="cuda").manual_seed(11)
    H, F = HIDDEN, FF
    m = dict(embed=packed(rng, N.Q4B64, VOCAB, H, 16.0), head=packed(rng, N.Q4B64, VOCAB, H, 3.0),
             qkv=packed(rng, N.Q4B64, 2 * 256 + 2 * 64, H, 1.0), o=packed(rng, N.Q4B64, H, 256, 1.0),
             gate_up=packed(rng, dtype, 2 * F, H, 1.0), down=packed(rng, dtype, H, F, 8.0), post=torch.zeros(H, device="cuda"))
    m["o"]["scale"].zero_()
    if outlier:
        m["post"][100] = 2.0 ** outlier
        m["gate_up"]["scale"][:, 1] = 0
        for row in (200, F + 200):  # gate and up of one column of the second product
            m["gate_up"]["s_out"][row] *= 2.0 ** min(outlier // 2, 15)
        m["down"]["scale"][:, 3] = 0
    return m


def load(ex, m):
    G = N.LAYER_GLOBAL
    for tensor, key in ((N.T_EMBED, "embed"), (N.T_LM_HEAD, "head")):
        ex.load_matrix(G, tensor, operation(m[key]))
    for tensor, key in ((N.T_ATTN_QKV, "qkv"), (N.T_ATTN_O, "o"), (N.T_MLP_GATE_UP, "gate_up"), (N.T_MLP_DOWN, "down")):
        ex.load_matrix(0, tensor, operation(m[key]))
    ex.load_vector(G, N.T_FINAL_NORM, np.zeros(HIDDEN, np.float32))
    for tensor, v in ((N.T_INPUT_NORM, np.zeros(HIDDEN)), (N.T_POST_NORM, m["post"].cpu().numpy()), (N.T_Q_NORM, np.zeros(64)),
                      (N.T_K_NORM, np.zeros(64))):
        ex.load_vector(0, tensor, v.astype(np.float32))


def exact(m, tokens):
    norm = lambda x: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6)
    h = values(m["embed"])[torch.as_tensor(tokens, device="cuda")]
    y = (norm(h) * (1 + m["post"].double())) @ values(m["gate_up"]).T
    g, u = y[:, :FF], y[:, FF:]
    h = h + (g * torch.sigmoid(g) * u) @ values(m["down"]).T
    return (norm(h) @ values(m["head"]).T).cpu().numpy()


@pytest.mark.parametrize("dtype", [ctox.Q4B64, ctox.Q2B64])
@pytest.mark.parametrize("outlier", [0, 14, 24, 40])
def test_pair_products_against_64_bits(dtype, outlier):
    """160, 200 and 256 positions: tiles of 160 to 256, the last one full or cut, over 71 row tiles and 39.5 of them. The sums
    of 79 and of 71 blocks are 32-bit: roundings of 2^-24 that add up at worst like their number, 9e-6 over both products
    (measured: 3e-6 for the worst position). The same call again gives the same bits."""
    be = ctox.B200Backend(0)
    cfg = ctox.qwen38_27b_config(
        vocab_size=VOCAB, hidden_size=HIDDEN, intermediate_size=FF, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=1,
        head_dim=64, rotary_dim=16, full_attention_interval=1, linear_num_key_heads=2, linear_num_value_heads=2, max_context_tokens=1100,
        max_draft_tokens=0, mtp_num_hidden_layers=0, draft_vocab=0, kv_dtype=N.F32)
    ex = ctox.B200Executor(be, cfg)
    try:
        m = model(dtype, outlier)
        load(ex, m)
        ex.warmup()
        for n in (160, 200, 256):
            tokens = [int(t) for t in np.random.default_rng(n).integers(0, VOCAB, n)]
            want = exact(m, tokens)
            runs = []
            for _ in range(4):
                ex.reset_session()
                before = be.kernel_launches()
                ex.extend(tokens)
                assert be.kernel_launches() - before < 30, "one long pass"
                ex.reset_session()
                runs.append(np.stack(ex.extend(tokens, list(range(n)))))
            assert all(np.array_equal(r, runs[0]) for r in runs[1:])
            error = np.linalg.norm(runs[0] - want, axis=1) / np.linalg.norm(want, axis=1)
            assert error.max() <= 1e-5, (n, error.max(), error.mean())
    finally:
        ex.unload()
        be.close()
