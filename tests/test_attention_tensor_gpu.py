"""Attention of short passes over a long bf16 cache on tcgen05 (k_attention_tensor): 16, 24 and 32 query rows, contexts that end at
and around the edge of a 64-token tile, scores flat and steep enough for the softmax reference to move, against long passes over the
same session, which take k_attention_mma."""
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
        for step in (1, 4, 20):
            ex.prefill_synthetic(9600, 3)
            runs.append(np.concatenate([ex.extend(tokens[a:a + step], list(range(step))) for a in range(0, 20, step)]))
        assert np.isfinite(runs[-1]).all()
        for short in runs[:-1]:
            assert max(rel_l2(a, b) for a, b in zip(short, runs[-1])) <= 1e-3  # as above
    finally:
        ex.unload()
        be.close()


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
