"""The gated-delta scan where its chunks of eight tokens end, over layers, in place, and with keys and queries that cannot be
read four at a time, against the recurrence in 64 bits."""
import numpy as np
import pytest
import torch

import ctox_llm_b200 as ctox

pytestmark = pytest.mark.gpu


def plain(q, k, v, g, beta, state):
    L, T, K, _ = q.shape
    H = v.shape[2]
    unit = lambda x: (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // K, 2)
    q, k, out = unit(q) * 128 ** -0.5, unit(k), []
    for t in range(T):
        state = state * torch.exp(g[:, t])[..., None, None]
        d = (v[:, t] - torch.einsum("lhk,lhkv->lhv", k[:, t], state)) * beta[:, t][..., None]
        state = state + k[:, t][..., None] * d[..., None, :]
        out.append(torch.einsum("lhk,lhkv->lhv", q[:, t], state))
    return torch.stack(out, 1), state


@pytest.mark.parametrize("tokens", [1, 7, 8, 9, 16, 17, 40])
@pytest.mark.parametrize("layers,heads,qk,offset", [(1, 4, 4, 0), (3, 6, 2, 1), (2, 12, 4, 3)])
def test_scan_at_chunk_edges(tokens, layers, heads, qk, offset):
    """32-bit sums of 128 terms per token, carried over 40 tokens: 1e-5 of the result."""
    be = ctox.B200Backend(0)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g, dtype=torch.float64).float()
    shape = (layers, tokens, qk, 128)
    n = layers * tokens * qk * 128
    qf, kf = rnd(n + 4), rnd(n + 4)
    q, k = qf[offset:offset + n], kf[offset:offset + n]
    v, state = rnd(layers, tokens, heads, 128), rnd(layers, heads, 128, 128) * 0.1
    decay, beta = torch.log(torch.sigmoid(rnd(layers, tokens, heads) + 2)), torch.sigmoid(rnd(layers, tokens, heads))
    want, want_state = plain(*(t.double() for t in (q.view(shape), k.view(shape), v, decay, beta, state)))
    out, moved = torch.zeros_like(v), state.clone()
    torch.cuda.synchronize()
    be.gated_delta_scan_layers(*(t.data_ptr() for t in (q, k, v, decay, beta, moved, moved, out)), layers, tokens, heads, qk)
    be.synchronize()
    for got, ref in ((out, want), (moved, want_state)):
        assert float((got.double() - ref).norm() / ref.norm()) <= 1e-5
    be.close()
