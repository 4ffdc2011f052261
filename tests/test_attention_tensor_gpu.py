"""Attention of short passes over a long bf16 cache on tcgen05 (k_attention_tensor): up to 32 query rows, contexts that end at and around
the edge of a 64-token tile, scores flat and steep enough for the softmax reference to move, against 64-bit attention and against long
passes over the same session, which take k_attention_mma."""
import os
import subprocess
import sys

import numpy as np
import pytest

import ctox_llm_b200 as ctox
from ctox_llm_b200 import _native as N
from gpu_util import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gain", [0.0, 6.0])
@pytest.mark.parametrize("page_tokens", [16, 256, 48])
def test_short_passes_on_a_long_session(page_tokens, gain):
    """Both sum the same products of 16-bit halves in 32 bits; keys and values of the portion may round the other way in the
    16-bit cache: 1e-3 of the logits as for the long passes (test_long_session_gpu.py). A gain of 1 + 6 on the queries makes
    scores of 7 to 10 powers of two and as much more of their error."""
    be = ctox.B200Backend(0)
    ex = ctox.B200Executor(be, ctox.qwen38_27b_config(
        vocab_size=2048, hidden_size=1024, intermediate_size=1024, num_hidden_layers=2, full_attention_interval=2, num_attention_heads=24,
        num_key_value_heads=4, head_dim=256, rotary_dim=64, linear_num_key_heads=4, linear_num_value_heads=8, max_context_tokens=11000,
        kv_page_tokens=page_tokens, max_draft_tokens=0, mtp_num_hidden_layers=0, draft_vocab=0, kv_dtype=ctox.BF16))
    try:
        ex.fill_synthetic(5)
        if gain:
            ex.load_vector(1, N.T_Q_NORM, np.full(256, gain, np.float32))
        ex.warmup()
        for position in (9472, 9533, 9599):  # 148 tiles and more: four per part of the context
            tokens = [int(t) for t in np.random.default_rng(position).integers(0, 2048, 20)]
            ex.prefill_synthetic(position, 3)
            whole = ex.extend(tokens, list(range(20)))
            for m in (1, 2, 3, 4, 5):
                assert ex.attention_kernel(position, m) == 2
                ex.prefill_synthetic(position, 3)
                short = [row for a in range(0, 20, m) for row in ex.extend(tokens[a:a + m], list(range(min(m, 20 - a))))]
                assert max(rel_l2(a, b) for a, b in zip(short, whole)) <= (1e-3 if not gain else 7e-3), (position, m)
    finally:
        ex.unload()
        be.close()


def test_a_key_that_is_nan_has_no_weight():
    """Keys that overflow (norm weights of 3e38: the turn of two infinities is NaN) are passed over by short passes as by long ones; the
    tokens ahead of the portion have other keys."""
    be = ctox.B200Backend(0)
    ex = ctox.B200Executor(be, ctox.qwen38_27b_config(
        vocab_size=2048, hidden_size=1024, intermediate_size=1024, num_hidden_layers=2, full_attention_interval=2, num_attention_heads=24,
        num_key_value_heads=4, head_dim=256, rotary_dim=64, linear_num_key_heads=4, linear_num_value_heads=8, max_context_tokens=11000,
        max_draft_tokens=0, mtp_num_hidden_layers=0, draft_vocab=0, kv_dtype=ctox.BF16))
    try:
        ex.fill_synthetic(5)
        ex.load_vector(1, N.T_K_NORM, np.full(256, 3e38, np.float32))
        ex.warmup()
        tokens = [int(t) for t in np.random.default_rng(1).integers(0, 2048, 20)]
        runs = []
        assert ex.attention_kernel(9600, 1) == ex.attention_kernel(9600, 4) == 2
        for step in (1, 4, 20):
            ex.prefill_synthetic(9600, 3)
            runs.append(np.concatenate([ex.extend(tokens[a:a + step], list(range(step))) for a in range(0, 20, step)]))
        assert np.isfinite(runs[-1]).all()
        for short in runs[:-1]:
            assert max(rel_l2(a, b) for a, b in zip(short, runs[-1])) <= 1e-3  # as above
    finally:
        ex.unload()
        be.close()


@pytest.mark.parametrize("gain", [0.0, 6.0])
@pytest.mark.parametrize("heads,kv_heads,passes", [(24, 4, (1, 2, 3, 4, 5, 5)), (16, 4, (1, 4, 5, 6, 7, 8)), (20, 4, (3, 4, 6, 6)), (4, 4, (1, 8, 8)),
                                                   (4, 1, (1, 8, 8)), (32, 8, (4, 5, 8))])
def test_against_64_bits(heads, kv_heads, passes, gain):
    """Passes behind 12000 tokens (38400 with one KV head) of one layer against plain 64-bit attention over keys and values rounded to the cache's 16 bits, at every
    form's largest number of query rows (16, 24, 32) among others, and with more merging CTAs (positions x heads) than SMs.
    Bound: keys of 32-bit projections (1e-6 off) round the other way in the cache in one value of 2000, by 2^-8 of it; a score of standard
    deviation 1 + gain moves by 9e-5 (1 + gain). Flat scores spread over thousands of tokens, whose moves cancel (3e-5); steep ones lie
    on a few, three deviations of which are allowed.
    The long pass over the same tokens reads the same cache, so that only the two bf16 parts of queries and weights are left (2^-17
    of a value, and of a score of up to 4 (1 + gain))."""
    import torch
    from perf import cases
    n0 = 12000 if kv_heads > 1 else 38400  # 148 parts of four tiles
    c = dict(kind="hybrid", width=1024, layers=1, interval=1, ff=1024, vocab=2048, heads=heads, kv_heads=kv_heads, head_dim=256, linear_heads=4,
             linear_qk=2, prompt=n0, blocks=64, drafts=0, kv="bf16")
    t = cases.hybrid_tensors(c, heads)
    a = t["layers"][0]
    a["qn"] += gain
    tokens = cases.tokens_of(2048, n0 + sum(passes), 3)
    be = ctox.B200Backend(0)
    ex = ctox.B200Executor(be, cases.hybrid_config(c))
    try:
        cases.load_hybrid(ex, t)
        ex.warmup()
        ex.extend(tokens[:n0])
        got, at = [], n0
        for m in passes:
            assert ex.attention_kernel(at, m) == 2
            got.append(ex.extend(tokens[at:at + m], list(range(m))))
            at += m
        ex.reset_session()
        ex.extend(tokens[:n0])
        whole = ex.extend(tokens[n0:], list(range(sum(passes))))
    finally:
        ex.unload()
        be.close()
    F64, n, r = torch.float64, len(tokens), sum(passes)
    w = lambda v: 1.0 + v.to(F64)
    x = cases.values64(dict(t["embed"], rows=n, blocks=t["embed"]["blocks"][tokens], s_out=t["embed"]["s_out"][tokens]))
    h = cases.rms(x) * w(a["in_ln"])
    q, k, v = (h @ cases.values64(m).T for m in a["qkv"])
    q = q.view(n, heads, 2, 256)
    gate = q[-r:, :, 1].reshape(r, -1)
    q = cases.rotate_halves(cases.rms(q[:, :, 0]) * w(a["qn"]), 64, 1e7)[-r:]
    k = cases.rotate_halves(cases.rms(k.view(n, kv_heads, 256)) * w(a["kn"]), 64, 1e7).bfloat16().to(F64)
    v = v.view(n, kv_heads, 256).bfloat16().to(F64)
    seen = torch.arange(n, device="cuda")[None, :] <= torch.arange(n - r, n, device="cuda")[:, None]
    y = torch.cat([torch.softmax((q[:, i] @ k[:, i * kv_heads // heads].T / 16.0).masked_fill(~seen, -np.inf), -1) @ v[:, i * kv_heads // heads]
                   for i in range(heads)], -1) * torch.sigmoid(gate)
    x = x[-r:] + y @ cases.values64(a["o"]).T
    h = cases.rms(x) * w(a["post_ln"])
    x = x + (cases.silu(h @ cases.values64(a["gate_up"][0]).T) * (h @ cases.values64(a["gate_up"][1]).T)) @ cases.values64(a["down"]).T
    want = (cases.rms(x) * w(t["final"])) @ cases.values64(t["head"]).T
    got = np.concatenate(got)
    off, apart = (max(rel_l2(x, y) for x, y in zip(got, other)) for other in (want.cpu().numpy(), whole))
    assert off <= (2.8e-4 * (1 + gain) if gain else 3e-5)
    assert apart <= 3e-5 * (1 + gain)


@pytest.mark.parametrize("session", ["12000", "stack"])
def test_overlap_changes_no_bit(tmp_path, session):
    """As test_dependent_launch_overlap_changes_no_bit, where cache rows of earlier passes are copied ahead of the wait: by this kernel
    (12000 tokens: 187 tiles in 37 parts) and by the attention of layer stacks."""
    here = os.path.dirname(os.path.abspath(__file__))
    outs = []
    for pdl in ("1", "0"):
        env = dict(os.environ, CTOX_PDL=pdl, PYTHONPATH=os.path.dirname(here) + os.pathsep + os.environ.get("PYTHONPATH", ""))
        path = str(tmp_path / (pdl + ".npz"))
        r = subprocess.run([sys.executable, os.path.join(here, "pdl_worker.py"), path, session], env=env, capture_output=True, text=True, timeout=900)
        assert r.returncode == 0, r.stderr[-2000:]
        outs.append(np.load(path))
    for name in outs[0]:
        assert np.array_equal(outs[0][name], outs[1][name]), name
