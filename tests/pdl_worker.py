"""Helper of test_exec_gpu.py: speculative blocks of an 8-layer synthetic model of the full widths,
results written to the .npz named on the command line (run once with programmatic dependent launch
and once with CTOX_PDL=0). A second argument gives the length of the session, or "stack" for short
passes of layer-stack models in its place."""
import sys

import numpy as np

import ctox_llm_b200 as ctox


def main(path, session=2000):
    be = ctox.B200Backend(0)
    cfg = ctox.qwen38_27b_config(max_context_tokens=session + 2096, num_hidden_layers=8, max_draft_tokens=3)
    ex = ctox.B200Executor(be, cfg)
    ex.fill_synthetic(seed=0)
    ex.warmup()
    ex.keep_logits(True)
    ex.prefill([int(t) for t in np.random.default_rng(3).integers(0, cfg.vocab_size, 21)])
    ex.prefill_synthetic(session, seed=1)
    tok, tokens, logits, hidden = 1, [], [], []
    for i in range(15):
        blk = ex.decode(tok, mtp_enabled=i % 4 != 3, force_accept=[-1, 0, 1, 2, 3][i % 5])
        tokens.append(list(blk.emitted) + [-1] * (5 - len(blk.emitted)) + list(blk.draft_tokens) +
                      [-1] * (4 - len(blk.draft_tokens)))
        logits.append(ex.last_logits(0).copy())
        hidden.append(ex.last_hidden().copy())
        tok = blk.token_id
    ex.unload()
    be.close()
    np.savez(path, tokens=np.array(tokens), logits=np.stack(logits), hidden=np.stack(hidden))


def stack(path):
    """Portions of one to eight positions: caches and states of earlier passes are read ahead of waits."""
    import tempfile

    import lomelorn_util as lomelorn
    import vasanex_util as vasanex
    models = (lomelorn.model([lomelorn.layer(heads=8, dim=128, rot_dim=64, vdim=128, q_rank=192, kv_rank=512, window=256, ff=1024)] * 2,
                             vocab=1000, width=2048),
              vasanex.model([vasanex.attention(heads=16, kv_heads=4, dim=128, vdim=128, window=200, ff=1024), vasanex.mlstm(heads=4, dim=128, vdim=256, ff=1024)] * 2,
                            vocab=1000, width=2048))
    out = {}
    for i, (config, tensors) in enumerate(models):
        be = ctox.B200Backend(0)
        with tempfile.TemporaryDirectory() as d:
            ex = ctox.open_model(lomelorn.write_model(d + "/m", config, tensors), backend=be, dtype="bfloat16", max_context_tokens=512)
        tokens = [int(t) for t in np.random.default_rng(i).integers(0, 1000, 400)]
        ex.extend(tokens[:300])
        at, logits = 300, []
        for m in [1, 1, 1, 3, 1, 8, 1, 1, 5, 1, 2, 1, 1, 1] * 3:
            logits.append(ex.extend(tokens[at:at + m], list(range(m))))
            at += m
        out[f"logits{i}"] = np.concatenate(logits)
        ex.unload()
        be.close()
    np.savez(path, **out)


if __name__ == "__main__":
    if sys.argv[2:] == ["stack"]:
        stack(sys.argv[1])
    else:
        main(sys.argv[1], *map(int, sys.argv[2:]))
