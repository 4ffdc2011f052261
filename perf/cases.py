"""The work that users of this package have it do, as measurable cases.

Every case goes through the public interface (`ctox_llm_b200`): prepared packed matrices
(`prepare_fused_matvec`, `dispatch_device`, `fanout_dispatch_device`, `lmhead_verify`), the gated-delta
scan, and `B200Executor` for the three model families (the hybrid model in packed weights, Lomelorn and
Vasanex layer stacks in bf16). Weights and inputs are random, in the distributions of the benchmark.
`exact` restates each path in plain 64-bit torch where the weights are made here; the two largest
models are filled by the executor itself (`fill_synthetic`) and have no such value.
"""
import math

import torch

import ctox_llm_b200 as ctox
from ctox_llm_b200 import native as N

DEV = "cuda"
BLOCK_BYTES = {"q4": 34, "q2": 18}
CODE = {"q4": N.Q4B64, "q2": N.Q2B64}
F64 = torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one small projection for one position: launch latency (a router, an adapter, a draft model's layer)
        dict(name="matvec-small", kind="matvec", dtype="q4", rows=1024, cols=1024, positions=1, x="bf16"),
        # the headline matrix of the benchmark: gate or up projection in Q4, plain decode
        dict(name="matvec-q4", kind="matvec", dtype="q4", rows=17408, cols=5120, positions=1, x="f32"),
        # the down projection in Q2 for a verify pass of three drafts and the current token
        dict(name="matvec-q2-verify", kind="matvec", dtype="q2", rows=5120, cols=17408, positions=4, x="bf16"),
        # query, key and value projections of one layer for a draft tree of 16 nodes
        dict(name="fanout-tree", kind="fanout", dtype="q4", rows=12288, kv_rows=1024, cols=5120, positions=16, x="bf16"),
        # lm_head, softmax statistics and acceptance over a chain of 8 positions, the real vocabulary
        dict(name="head-verify", kind="head", rows=248320, cols=5120, nodes=8, temperature=0.7),
        # the recurrence of a verify pass over all 48 linear-attention layers
        dict(name="delta-layers", kind="delta", layers=48, heads=48, qk_heads=16, tokens=4),
        # a small hybrid model, a short prompt and a few speculative blocks: latency throughout
        dict(name="hybrid-small", kind="hybrid", width=1024, layers=4, interval=4, ff=2816, vocab=16384, heads=8, kv_heads=2,
             head_dim=128, linear_heads=16, linear_qk=8, prompt=37, blocks=8, drafts=3, kv="bf16"),
        # the flagship: 64 layers, 32768 tokens of context, speculative decode with three drafts
        dict(name="hybrid-decode-32k", kind="flagship", layers=64, context=32768, blocks=2, drafts=3),
        # a prompt of a thousand tokens through eight layers of the flagship's width, then the first block
        dict(name="hybrid-prompt", kind="hybrid", width=5120, layers=8, interval=4, ff=17408, vocab=32768, heads=24, kv_heads=4,
             head_dim=256, linear_heads=48, linear_qk=16, prompt=1000, blocks=1, drafts=3, kv="bf16"),
        # a long prompt through a wide latent-attention model
        dict(name="latent-prompt", kind="stack", design="latent", width=5120, layers=8, ff=17408, vocab=32768, heads=40,
             window=4096, prompt=4096, tokens=0, kv="bf16", weights="synthetic"),
        # plain decode of the same model with 8192 tokens of context
        dict(name="latent-decode-8k", kind="stack", design="latent", width=5120, layers=8, ff=17408, vocab=32768, heads=40,
             window=4096, context=8192, tokens=16, kv="bf16", weights="synthetic"),
        # a whole request on a grouped-attention and matrix-memory model: ragged prompt, then an answer
        dict(name="vasanex-request", kind="stack", design="vasanex", width=2048, layers=8, ff=8192, vocab=32768, heads=16,
             kv_heads=4, memory_heads=4, window=1024, prompt=1500, tokens=32, kv="bf16", weights="seeded"),
    ]


def log_int(rng, low, high, step=1):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high))) / step)) * step))


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "fanout", "head", "delta", "hybrid", "hybrid", "latent", "vasanex"])
    if kind == "matvec":
        return dict(kind=kind, dtype=rng.choice(["q4", "q2"]), rows=log_int(rng, 300, 40000), cols=log_int(rng, 512, 18432, 64),
                    positions=rng.choice([1, 1, 2, 3, 4, 4, 5, 8, 11, 16]), x=rng.choice(["f32", "bf16"]))
    if kind == "fanout":
        return dict(kind=kind, dtype=rng.choice(["q4", "q2"]), rows=log_int(rng, 1024, 20000), kv_rows=log_int(rng, 128, 2048),
                    cols=log_int(rng, 1024, 8192, 64), positions=rng.randint(1, 16), x=rng.choice(["f32", "bf16"]))
    if kind == "head":
        return dict(kind=kind, rows=log_int(rng, 30000, 248320), cols=log_int(rng, 1024, 5120, 64), nodes=rng.randint(1, 16),
                    temperature=rng.choice([0.0, 0.7, 1.0]))
    if kind == "delta":
        qk = rng.choice([4, 8, 16])
        return dict(kind=kind, layers=rng.randint(1, 48), heads=qk * rng.choice([1, 2, 3]), qk_heads=qk,
                    tokens=rng.randint(1, 8))
    if kind == "hybrid":
        heads, kv = rng.choice([(8, 2), (16, 4), (24, 4)])
        qk = rng.choice([8, 16])
        return dict(kind=kind, width=rng.choice([1024, 2048, 2560, 4096]), layers=rng.choice([2, 4, 6]), interval=rng.choice([1, 2, 4]),
                    ff=log_int(rng, 2048, 11264, 64), vocab=16384, heads=heads, kv_heads=kv, head_dim=rng.choice([128, 256, 256]),
                    linear_heads=qk * rng.choice([1, 2, 3]), linear_qk=qk, prompt=log_int(rng, 5, 1200), blocks=rng.randint(1, 12),
                    drafts=rng.choice([0, 1, 3, 4]), kv=rng.choice(["bf16", "bf16", "bf16", "f32"]))
    kv = rng.choice(["bf16", "bf16", "bf16", "f32"])
    case = dict(kind="stack", design=kind, width=rng.choice([1024, 2048, 2560]), layers=rng.choice([2, 4, 6]),
                ff=log_int(rng, 2048, 8192, 64), vocab=16384, heads=rng.choice([8, 16, 24]), window=rng.choice([256, 1024, 4096]),
                prompt=log_int(rng, 5, 300 if kv == "f32" else 2500), tokens=rng.randint(1, 40), kv=kv, weights="seeded")
    if kind == "vasanex":
        case.update(kv_heads=rng.choice([4, 8]), memory_heads=rng.choice([2, 4, 8]))
    return case


# ------------------------------------------------------------------ random tensors, made on the GPU from the seed alone
class Rng:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(1000003 * seed + 7)

    def normal(self, *shape, std=1.0, mean=0.0):
        return torch.randn(*shape, device=DEV, generator=self.g) * std + mean

    def scales(self, n):
        """Recovery scales: f16 values in [0.75, 1.25)."""
        return (torch.rand(n, device=DEV, generator=self.g) * 0.5 + 0.75).half()

    def packed(self, dtype, rows, cols, scale):
        """Canonical blocks [f16 scale][codes]: uniform codes, log-normal block scales around `scale`."""
        bb = BLOCK_BYTES[dtype]
        out = torch.randint(0, 256, (rows, cols // 64, bb), device=DEV, generator=self.g, dtype=torch.uint8)
        sc = (torch.exp(self.normal(rows, cols // 64, 1, std=0.5)) * scale).half()
        out[:, :, :2] = sc.view(torch.uint8)
        return out

    def matrix(self, dtype, rows, cols, s_in=None, gain=1.0):
        """A packed matrix whose products keep the size of their input, times `gain`."""
        return dict(dtype=dtype, rows=rows, cols=cols, blocks=self.packed(dtype, rows, cols, gain * 1.4 / math.sqrt(cols)),
                    s_in=self.scales(cols) if s_in is None else s_in, s_out=self.scales(rows))

    def bf16(self, rows, cols, gain=1.0):
        return (torch.randn(rows, cols, device=DEV, generator=self.g) * (gain / math.sqrt(cols))).bfloat16()


def host(t):
    return t.contiguous().view(torch.uint8).reshape(-1).cpu().numpy()


def operation(mats):
    """The rows of one or several packed matrices (one s_in) as one operation."""
    m = mats[0]
    import numpy as np
    return ctox.FusedMatVec(CODE[m["dtype"]], np.concatenate([host(x["blocks"]) for x in mats]), sum(x["rows"] for x in mats), m["cols"],
                            None, s_in=host(m["s_in"]), s_out=np.concatenate([host(x["s_out"]) for x in mats]))


def values64(m):
    """What a packed matrix stands for, recovery scales included: [rows, cols] in 64 bits."""
    b = m["blocks"]
    scale = b[:, :, :2].contiguous().view(torch.float16).to(F64)
    codes = b[:, :, 2:]
    if m["dtype"] == "q4":
        q = torch.stack([codes & 15, codes >> 4], -1).to(F64).sub_(7.5).div_(7.5)
    else:
        q = torch.stack([(codes >> s) & 3 for s in (0, 2, 4, 6)], -1).to(F64).mul_(2).sub_(3).div_(3)
    q = q.reshape(m["rows"], m["cols"] // 64, 64).mul_(scale).reshape(m["rows"], m["cols"])
    return q.mul_(m["s_in"].to(F64)).mul_(m["s_out"].to(F64)[:, None])


def backend():
    stream = torch.cuda.Stream()
    return ctox.B200Backend(torch.cuda.current_device(), stream=stream.cuda_stream), stream


X_TYPE = {"f32": (torch.float32, N.F32), "bf16": (torch.bfloat16, N.BF16)}


def op_inputs(case, seed):
    r = Rng(seed)
    x = r.normal(case["positions"], case["cols"]).to(X_TYPE[case["x"]][0])
    s_in = r.scales(case["cols"])
    rows = [case["rows"]] if case["kind"] == "matvec" else [case["rows"], case["kv_rows"], case["kv_rows"]]
    mats = []
    for n in rows:  # block scales as in the benchmark: exp(N(-4, 0.5))
        mats.append(dict(dtype=case["dtype"], rows=n, cols=case["cols"], blocks=r.packed(case["dtype"], n, case["cols"], math.exp(-4.0)),
                         s_in=s_in, s_out=r.scales(n)))
    return x, mats


def head_inputs(case, seed):
    r = Rng(seed)
    m = r.matrix("q4", case["rows"], case["cols"], gain=3.0)
    hidden = r.normal(case["nodes"], case["cols"])
    tokens = torch.randint(0, case["rows"], (case["nodes"],), device=DEV, generator=r.g)
    return m, hidden, tokens


def delta_inputs(case, seed):
    r = Rng(seed)
    L, T, H, K = case["layers"], case["tokens"], case["heads"], case["qk_heads"]
    unit = lambda *s: torch.nn.functional.normalize(r.normal(*s), dim=-1)
    return dict(q=unit(L, T, K, 128), k=unit(L, T, K, 128), v=r.normal(L, T, H, 128),
                g=torch.log(torch.sigmoid(r.normal(L, T, H, mean=2.0))), beta=torch.sigmoid(r.normal(L, T, H)),
                state=r.normal(L, H, 128, 128, std=0.02))


# ------------------------------------------------------------------ models
def hybrid_config(c):
    return ctox.qwen38_27b_config(
        vocab_size=c["vocab"], hidden_size=c["width"], intermediate_size=c["ff"], num_hidden_layers=c["layers"],
        num_attention_heads=c["heads"], num_key_value_heads=c["kv_heads"], head_dim=c["head_dim"], rotary_dim=c["head_dim"] // 4,
        full_attention_interval=c["interval"], linear_num_key_heads=c["linear_qk"], linear_num_value_heads=c["linear_heads"],
        max_context_tokens=c["prompt"] + c["blocks"] + 64, max_draft_tokens=c["drafts"], mtp_num_hidden_layers=1 if c["drafts"] else 0,
        draft_vocab=0, kv_dtype=N.BF16 if c["kv"] == "bf16" else N.F32)


def hybrid_tensors(c, seed):
    r, H = Rng(seed), c["width"]
    norm = lambda n, mean=0.0: r.normal(n, std=0.05, mean=mean)
    qw, kvw = c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"]
    kw, vw = c["linear_qk"] * 128, c["linear_heads"] * 128
    t = dict(embed=r.matrix("q4", c["vocab"], H, gain=16.0), head=r.matrix("q4", c["vocab"], H, gain=3.0), final=norm(H), layers=[])
    for l in range(c["layers"] + (1 if c["drafts"] else 0)):
        full = l >= c["layers"] or (l + 1) % c["interval"] == 0
        a = dict(full=full, in_ln=norm(H), post_ln=norm(H))
        s = r.scales(H)
        if full:
            a.update(qkv=[r.matrix("q4", n, H, s) for n in (2 * qw, kvw, kvw)], o=r.matrix("q4", H, qw), qn=norm(c["head_dim"]), kn=norm(c["head_dim"]))
        else:
            a.update(fan=[r.matrix("q4", n, H, s) for n in (2 * kw + vw, vw, c["linear_heads"], c["linear_heads"])], o=r.matrix("q4", H, vw),
                     conv=r.normal(2 * kw + vw, 4, std=0.4), a_log=r.normal(c["linear_heads"], std=0.5), dt=r.normal(c["linear_heads"], std=0.5),
                     ln=norm(128, 1.0))
        s = r.scales(H)
        a.update(gate_up=[r.matrix("q2", c["ff"], H, s) for _ in range(2)], down=r.matrix("q2", H, c["ff"]))
        t["layers"].append(a)
    if c["drafts"]:
        t.update(fc=r.matrix("q4", H, 2 * H), ne=norm(H), nh=norm(H), nm=norm(H))
    return t


def load_hybrid(ex, t):
    G = N.LAYER_GLOBAL
    vec = lambda l, k, v: ex.load_vector(l, k, v.reshape(-1).cpu().numpy())
    ex.load_matrix(G, N.T_EMBED, operation([t["embed"]]))
    ex.load_matrix(G, N.T_LM_HEAD, operation([t["head"]]))
    vec(G, N.T_FINAL_NORM, t["final"])
    for l, a in enumerate(t["layers"]):
        vec(l, N.T_INPUT_NORM, a["in_ln"])
        vec(l, N.T_POST_NORM, a["post_ln"])
        if a["full"]:
            ex.load_matrix(l, N.T_ATTN_QKV, operation(a["qkv"]))
            ex.load_matrix(l, N.T_ATTN_O, operation([a["o"]]))
            vec(l, N.T_Q_NORM, a["qn"])
            vec(l, N.T_K_NORM, a["kn"])
        else:
            ex.load_matrix(l, N.T_LIN_IN, operation(a["fan"]))
            ex.load_matrix(l, N.T_LIN_OUT, operation([a["o"]]))
            for k, name in ((N.T_CONV_W, "conv"), (N.T_A_LOG, "a_log"), (N.T_DT_BIAS, "dt"), (N.T_LIN_NORM, "ln")):
                vec(l, k, a[name])
        ex.load_matrix(l, N.T_MLP_GATE_UP, operation(a["gate_up"]))
        ex.load_matrix(l, N.T_MLP_DOWN, operation([a["down"]]))
    if "fc" in t:
        ex.load_matrix(G, N.T_MTP_FC, operation([t["fc"]]))
        for k, name in ((N.T_MTP_NORM_E, "ne"), (N.T_MTP_NORM_H, "nh"), (N.T_MTP_NORM, "nm")):
            vec(G, k, t[name])


def stack_config(c):
    common = dict(ff=c["ff"], window=c["window"], rope_base=10000.0, kv_from=-1)
    top = dict(vocab_size=c["vocab"], hidden_size=c["width"], norm_eps=1e-6,
               max_context_tokens=max(c.get("context", 0) + 1024, c.get("prompt", 0) + c["tokens"] + 64),
               kv_dtype=N.BF16 if c["kv"] == "bf16" else N.F32)
    if c["design"] == "latent":
        layer = dict(common, mixer=N.MIXER_LATENT_ATTENTION, heads=c["heads"], dim=128, rot_dim=64, vdim=128, q_rank=c["width"] * 3 // 10 // 64 * 64,
                     kv_rank=512, score_scale=192 ** -0.5, mlp=N.MLP_RELU2)
        return ctox.StackConfig(layers=[N.LayerConfig(**layer) for _ in range(c["layers"])], logit_softcap=30.0, **top)
    mlp = dict(common, mlp=N.MLP_CLAMPED_GLU, mlp_limit=7.0, mlp_slope=1.702)
    grouped = dict(mlp, mixer=N.MIXER_GROUPED_ATTENTION, heads=c["heads"], kv_heads=c["kv_heads"], dim=128, vdim=128, rot_dim=64,
                   score_scale=128 ** -0.5, attn=15)
    memory = dict(mlp, mixer=N.MIXER_MATRIX_MEMORY, heads=c["memory_heads"], dim=256, vdim=512, gate_cap=15.0)
    return ctox.StackConfig(layers=[N.LayerConfig(**(memory if i % 2 else grouped)) for i in range(c["layers"])], logit_softcap=0.0,
                            norm=N.NORM_RMS, out_norms=False, tied_head=True, **top)


def stack_tensors(c, seed):
    """{(layer, tensor): bf16 matrix or f32 vector} in the executor's own tensor names."""
    r, W, G, t = Rng(seed), c["width"], N.LAYER_GLOBAL, {}
    norm = lambda n: r.normal(n, std=0.1, mean=1.0)
    latent = c["design"] == "latent"
    t[G, N.T_EMBED] = r.bf16(c["vocab"], W, math.sqrt(W) if latent else 3.0)
    if latent:
        t[G, N.T_LM_HEAD] = r.bf16(c["vocab"], W, 3.0)
    t[G, N.T_FINAL_NORM] = norm(W)
    q_rank = W * 3 // 10 // 64 * 64
    for l in range(c["layers"]):
        t[l, N.T_INPUT_NORM] = norm(W)
        if latent:
            H = c["heads"]
            for name, rows, cols in ((N.T_Q_DOWN, q_rank, W), (N.T_Q_UP, H * 192, q_rank), (N.T_KV_DOWN, 576, W), (N.T_K_UP, H * 128, 512),
                                     (N.T_V_UP, H * 128, 512), (N.T_ATTN_O, W, H * 128), (N.T_MLP_UP, c["ff"], W), (N.T_MLP_DOWN, W, c["ff"])):
                t[l, name] = r.bf16(rows, cols)
            for name, n in ((N.T_Q_DOWN_NORM, q_rank), (N.T_KV_DOWN_NORM, 512), (N.T_MIX_OUT_NORM, W), (N.T_POST_NORM, W), (N.T_MLP_OUT_NORM, W)):
                t[l, name] = norm(n)
            continue
        if l % 2:
            H = c["memory_heads"]
            shapes = ((N.T_MIX_Q, H * 256, W), (N.T_MIX_K, H * 256, W), (N.T_MIX_V, H * 512, W), (N.T_MIX_GATE, H * 512, W), (N.T_ATTN_O, W, H * 512),
                      (N.T_MEM_IN, H, W), (N.T_MEM_FORGET, H, W))
            t[l, N.T_MIX_HEAD_NORM] = norm(H * 512)
            t[l, N.T_MEM_IN_BIAS], t[l, N.T_MEM_FORGET_BIAS] = r.normal(H, std=0.5, mean=-0.5), r.normal(H, std=0.5, mean=4.0)
        else:
            H, K = c["heads"] * 128, c["kv_heads"] * 128
            shapes = ((N.T_MIX_Q, H, W), (N.T_MIX_K, K, W), (N.T_MIX_V, K, W), (N.T_ATTN_O, W, H))
            for name, n in ((N.T_MIX_Q_BIAS, H), (N.T_MIX_K_BIAS, K), (N.T_MIX_V_BIAS, K), (N.T_MIX_O_BIAS, W)):
                t[l, name] = r.normal(n, std=0.1)
            t[l, N.T_Q_NORM], t[l, N.T_K_NORM], t[l, N.T_ATTN_SINK] = norm(H), norm(K), r.normal(c["heads"])
            t[l, N.T_V_MIX] = r.normal(1, std=0.1, mean=0.4)
        for name, rows, cols in shapes + ((N.T_MLP_GATE, c["ff"], W), (N.T_MLP_UP, c["ff"], W), (N.T_MLP_DOWN, W, c["ff"])):
            t[l, name] = r.bf16(rows, cols)
        t[l, N.T_POST_NORM] = norm(W)
    return t


def load_stack(ex, tensors):
    for (l, name), v in tensors.items():
        if v.dim() == 2:
            ex.load_matrix(l, name, ctox.FusedMatVec(N.BF16, host(v), v.shape[0], v.shape[1], None))
        else:
            ex.load_vector(l, name, v.cpu().numpy())


def tokens_of(vocab, n, seed):
    g = torch.Generator().manual_seed(seed + 11)
    return torch.randint(0, vocab, (n,), generator=g).tolist()


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    be, stream = backend()
    s = dict(case=case, be=be, stream=stream)
    kind = case["kind"]
    if kind in ("matvec", "fanout"):
        s["x"], mats = op_inputs(case, seed)
        s["mats"] = [be.prepare_fused_matvec(operation([m])) for m in mats]
        s["y"] = [torch.zeros(case["positions"], m["rows"], device=DEV) for m in mats]
    elif kind == "head":
        m, s["hidden"], tokens = head_inputs(case, seed)
        s["head"], s["tokens"] = be.prepare_fused_matvec(operation([m])), tokens.tolist()
        s["logits"] = torch.zeros(case["nodes"], case["rows"], device=DEV)
    elif kind == "delta":
        s["in"] = delta_inputs(case, seed)
        s["out"], s["state"] = torch.zeros_like(s["in"]["v"]), torch.zeros_like(s["in"]["state"])
    elif kind == "hybrid":
        s["ex"] = ctox.B200Executor(be, hybrid_config(case))
        load_hybrid(s["ex"], hybrid_tensors(case, seed))
        s["prompt"] = tokens_of(case["vocab"], case["prompt"] + case["blocks"], seed)
    elif kind == "flagship":
        s["ex"] = ctox.B200Executor(be, ctox.qwen38_27b_config(num_hidden_layers=case["layers"], max_draft_tokens=case["drafts"],
                                                               max_context_tokens=case["context"] + 1024))
        s["ex"].fill_synthetic(seed)
        s["prompt"] = tokens_of(248320, 64, seed)
    else:
        s["ex"] = ctox.B200Executor(be, stack_config(case))
        if case["weights"] == "seeded":
            load_stack(s["ex"], stack_tensors(case, seed))
        else:
            s["ex"].fill_synthetic(seed)
        s["prompt"] = tokens_of(case["vocab"], case.get("prompt", 0) + max(case["tokens"], 64), seed)
    if "ex" in s:
        s["ex"].warmup()
        s["ex"].keep_logits(True)
        if "context" in case:
            s["ex"].prefill_synthetic(case["context"], seed)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ run
def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind in ("matvec", "fanout"):
        x, C, M = s["x"], case["cols"], case["positions"]
        if kind == "matvec":
            s["mats"][0].dispatch_device(x.data_ptr(), X_TYPE[case["x"]][1], M, C, s["y"][0].data_ptr(), case["rows"])
        else:
            s["be"].fanout_dispatch_device(s["mats"], x.data_ptr(), X_TYPE[case["x"]][1], M, C, [y.data_ptr() for y in s["y"]],
                                           [y.shape[1] for y in s["y"]])
        return s["y"]
    if kind == "head":
        n = case["nodes"]
        rec = s["head"].lmhead_verify(s["hidden"].data_ptr(), N.F32, case["cols"], list(range(-1, n - 1)), s["tokens"], case["temperature"],
                                      seed=3, step=5, logits_out_ptr=s["logits"].data_ptr())
        return dict(logits=s["logits"], greedy=rec["node_argmax"])
    if kind == "delta":
        i = s["in"]
        s["be"].gated_delta_scan_layers(*(i[k].data_ptr() for k in ("q", "k", "v", "g", "beta", "state")), s["state"].data_ptr(),
                                        s["out"].data_ptr(), case["layers"], case["tokens"], case["heads"], case["qk_heads"])
        return dict(out=s["out"], state=s["state"])
    ex = s["ex"]
    if kind == "stack" and "context" not in case:
        # the prompt in one call, the answer token by token; the tokens are given, so that every pass does the same work
        ex.reset_session()
        n = case["prompt"]
        first = ex.extend(s["prompt"][:n], [n - 1])
        for token in s["prompt"][n:n + case["tokens"]]:
            ex.decode(token, mtp_enabled=False)
        return dict(first=first, hidden=ex.last_hidden(), **({"logits": ex.last_logits(0)} if case["tokens"] else {}))
    mtp = bool(case.get("drafts"))
    if kind == "hybrid":
        ex.prefill(s["prompt"][:case["prompt"]])  # all but the last token, which the first block takes
        todo = s["prompt"][case["prompt"] - 1:case["prompt"] - 1 + case["blocks"]]
    else:  # a session that goes on; a full context starts the next one
        n = case.get("blocks") or case["tokens"]
        if ex.position() + n + 32 > case["context"] + 1024:
            ex.prefill_synthetic(case["context"], 1)
        todo = s["prompt"][:n]
    for token in todo:  # no draft is accepted, whatever a random model would draft: one token a block
        ex.decode(token, mtp_enabled=mtp, force_accept=0 if mtp else -1)
    out = dict(hidden=ex.last_hidden(), logits=ex.last_logits(0))
    if mtp:  # of the first draft; what follows it hangs on the token chosen there
        out["draft"] = ex.last_draft_logits()[0]
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def packed_bytes(dtype, rows, cols):
    return rows * (cols // 64) * BLOCK_BYTES[dtype]


def hybrid_work(c, full, linear, width, ff, heads, kv_heads, head_dim, linear_heads, linear_qk):
    """(weight bytes, weights) of the layers, per full and per linear layer summed."""
    q, kv, kw, vw = heads * head_dim, kv_heads * head_dim, linear_qk * 128, linear_heads * 128
    mats = [("q4", 2 * q + 2 * kv, width, full), ("q4", width, q, full), ("q4", 2 * kw + 2 * vw + 2 * linear_heads, width, linear),
            ("q4", width, vw, linear), ("q2", 2 * ff, width, full + linear), ("q2", width, ff, full + linear)]
    return sum(n * packed_bytes(d, r, k) for d, r, k, n in mats), sum(n * r * k for d, r, k, n in mats)


def work(case):
    kind = case["kind"]
    if kind in ("matvec", "fanout"):
        rows, P, C = case["rows"] + 2 * case.get("kv_rows", 0), case["positions"], case["cols"]
        return dict(bytes=packed_bytes(case["dtype"], rows, C) + P * (C * (2 if case["x"] == "bf16" else 4) + rows * 4) + 4 * (rows + C),
                    flops=2.0 * rows * C * P)
    if kind == "head":
        rows, C, n = case["rows"], case["cols"], case["nodes"]
        return dict(bytes=packed_bytes("q4", rows, C) + n * (C + rows) * 4 + 4 * (rows + C), flops=2.0 * rows * C * n)
    if kind == "delta":
        L, T, H, K = case["layers"], case["tokens"], case["heads"], case["qk_heads"]
        return dict(bytes=4.0 * L * (2 * H * 16384 + T * (2 * K * 128 + 2 * H * 128 + 2 * H)), flops=8.0 * L * T * H * 16384)
    if kind in ("hybrid", "flagship"):
        if kind == "hybrid":
            c = case
            dims = (c["width"], c["ff"], c["heads"], c["kv_heads"], c["head_dim"], c["linear_heads"], c["linear_qk"])
            interval, vocab, draft, prompt, start, kv = c["interval"], c["vocab"], c["vocab"], c["prompt"] - 1, c["prompt"], 2 if c["kv"] == "bf16" else 4
        else:
            c, dims = case, (5120, 17408, 24, 4, 256, 48, 16)
            interval, vocab, draft, prompt, start, kv = 4, 248320, 40000, 0, c["context"], 2
        full = c["layers"] // interval
        linear, mtp, blocks, m = c["layers"] - full, 1 if c["drafts"] else 0, c["blocks"], c["drafts"] + 1
        W, q, kvw = dims[0], dims[2] * dims[4], dims[3] * dims[4]
        wb, wn = hybrid_work(c, full, linear, *dims)
        mb, mn = hybrid_work(c, 1, 0, *dims)
        mb, mn = mb + packed_bytes("q4", W, 2 * W), mn + 2 * W * W
        state = linear * 2 * dims[5] * 16384 * 4.0
        cache = 2.0 * full * kvw * kv
        b = (1 if prompt else 0) * (wb + mtp * mb + state) + prompt * cache
        f = 2.0 * prompt * (wn + mtp * mn) + 4.0 * full * q * prompt * prompt / 2 + 8.0 * linear * dims[5] * 16384 * prompt
        b += blocks * (wb + packed_bytes("q4", vocab, W) + state + start * cache)
        b += blocks * mtp * c["drafts"] * (mb + packed_bytes("q4", draft, W) + start * 2.0 * kvw * kv)
        f += 2.0 * blocks * (m * (wn + vocab * W) + mtp * c["drafts"] * (mn + draft * W))
        f += blocks * (4.0 * m * full * q * start + 8.0 * m * linear * dims[5] * 16384)
        return dict(bytes=b, flops=f)
    c, W, L = case, case["width"], case["layers"]
    n, g, start = c.get("prompt", 0), c["tokens"], c.get("context", c.get("prompt", 0))
    vocab = c["vocab"] * W
    kv = 2 if c["kv"] == "bf16" else 4
    seen = min(start, c["window"])
    pairs = n * seen - seen * seen / 2 if n else 0  # (query, key) pairs of the prompt
    if c["design"] == "latent":
        q_rank, H = W * 3 // 10 // 64 * 64, c["heads"]
        weights = L * (q_rank * W + H * 192 * q_rank + 576 * W + 2 * H * 128 * 512 + W * H * 128 + 2 * W * c["ff"])
        row, per_pair, per_read = L * 576 * kv, L * 2.0 * H * 320, L * 2.0 * H * 1088
        state, memory_flops = 0, 0
    else:
        att, mem = (L + 1) // 2, L // 2
        H, K, M = c["heads"] * 128, c["kv_heads"] * 128, c["memory_heads"]
        weights = att * (2 * H + 2 * K) * W + mem * M * (512 + 3 * 512 + 2) * W + L * 3 * W * c["ff"]
        row, per_pair, per_read = att * 2 * K * kv, att * 4.0 * H, att * 4.0 * H
        state, memory_flops = mem * M * 256 * 512 * 4, mem * M * 256 * 512 * 6.0
    b = (2.0 * weights + n * row + 2 * state) * (1 if n else 0) + (2.0 * vocab if n else 0)
    f = 2.0 * n * weights + pairs * per_pair + n * memory_flops + (2.0 * vocab if n else 0)
    b += g * (2.0 * (weights + vocab) + seen * row + 2 * state)
    f += g * (2.0 * (weights + vocab) + seen * per_read + memory_flops)
    return dict(bytes=b, flops=f)


def tolerance(case):
    kind = case["kind"]
    if kind in ("matvec", "fanout", "head", "delta"):
        return dict(rel=1e-5, max=1e-4)  # 32-bit sums: up to 2.5e-6 from the 64-bit values
    if kind == "stack" and case["kv"] == "bf16":
        # bf16 activations between the kernels of a long pass: 0.4 % to 2.3 % from the 64-bit values, rows with nearly
        # cancelling matrix-memory sums most
        return dict(rel=3e-2, max=0.5)
    if case.get("kv") == "f32":
        return dict(rel=1e-4, max=1e-3)
    # keys and values in bf16, all else in 32 bits: 6e-5 to 1.4e-4 from the 64-bit values
    return dict(rel=1e-3, max=2e-2)


# ------------------------------------------------------------------ 64-bit restatements
def rms(x, eps=1e-6):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def rotate_halves(x, dims, base):
    """x [tokens, heads, width]: dimension i < dims / 2 is turned with i + dims / 2."""
    h = dims // 2
    angle = torch.arange(x.shape[0], device=DEV, dtype=F64)[:, None, None] * base ** (-2.0 * torch.arange(h, device=DEV, dtype=F64) / dims)
    u, v = x[..., :h], x[..., h:dims]
    return torch.cat([u * angle.cos() - v * angle.sin(), v * angle.cos() + u * angle.sin(), x[..., dims:]], -1)


def attend(q, k, v, scale, window=None, sink=None):
    """q [n, H, d], k [n, K, d], v [n, K, e] -> [n, H * e], causal."""
    n, H, K = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(n, device=DEV)
    see = i[None, :] <= i[:, None]
    if window:
        see &= i[:, None] - i[None, :] < window
    out = []
    for h in range(H):
        score = (q[:, h] @ k[:, h * K // H].T * scale).masked_fill_(~see, -math.inf)
        if sink is not None:
            score = torch.cat([score, sink[h].expand(n, 1)], -1)
        out.append(torch.softmax(score, -1)[:, :n] @ v[:, h * K // H])
    return torch.cat(out, -1)


def silu(x):
    return x * torch.sigmoid(x)


def exact_hybrid(c, seed):
    t = hybrid_tensors(c, seed)
    ids = torch.tensor(tokens_of(c["vocab"], c["prompt"] + c["blocks"], seed)[:c["prompt"] - 1 + c["blocks"]], device=DEV)
    n = len(ids)
    w = lambda v: 1.0 + v.to(F64)
    e = t["embed"]
    x = values64(dict(e, rows=n, blocks=e["blocks"][ids], s_out=e["s_out"][ids]))
    for a in t["layers"][:c["layers"]]:
        h = rms(x) * w(a["in_ln"])
        if a["full"]:
            H, K, d = c["heads"], c["kv_heads"], c["head_dim"]
            q, k, v = (h @ values64(m).T for m in a["qkv"])
            q = q.view(n, H, 2, d)
            q, gate = q[:, :, 0], q[:, :, 1].reshape(n, -1)
            q = rotate_halves(rms(q) * w(a["qn"]), d // 4, 1e7)
            k = rotate_halves(rms(k.view(n, K, d)) * w(a["kn"]), d // 4, 1e7)
            y = attend(q, k, v.view(n, K, d), d ** -0.5) * torch.sigmoid(gate)
        else:
            K, H = c["linear_qk"], c["linear_heads"]
            mixed, z, alpha, b = (h @ values64(m).T for m in a["fan"])
            past = torch.cat([mixed.new_zeros(3, mixed.shape[1]), mixed])
            conv = silu(sum(past[j:j + n] * a["conv"][:, j].to(F64) for j in range(4)))
            unit = lambda v: v * torch.rsqrt((v * v).sum(-1, keepdim=True) + 1e-6)
            q = unit(conv[:, :K * 128].view(n, K, 128)).repeat_interleave(H // K, 1) * 128 ** -0.5
            k = unit(conv[:, K * 128:2 * K * 128].view(n, K, 128)).repeat_interleave(H // K, 1)
            v = conv[:, 2 * K * 128:].view(n, H, 128)
            decay = torch.exp(-torch.exp(a["a_log"].to(F64)) * torch.nn.functional.softplus(alpha + a["dt"].to(F64)))
            y, _ = delta64(q, k, v, decay, torch.sigmoid(b), x.new_zeros(H, 128, 128))
            y = (rms(y) * a["ln"].to(F64) * silu(z.view(n, H, 128))).reshape(n, -1)
        x = x + y @ values64(a["o"]).T
        h = rms(x) * w(a["post_ln"])
        x = x + (silu(h @ values64(a["gate_up"][0]).T) * (h @ values64(a["gate_up"][1]).T)) @ values64(a["down"]).T
    hidden = rms(x[-1]) * w(t["final"])
    out = dict(hidden=hidden, logits=values64(t["head"]) @ hidden)
    if c["drafts"]:
        out["draft"] = None
    return out


def delta64(q, k, v, decay, beta, state):
    """q (scaled), k [T, H, 128] of unit length; state [H, 128 keys, 128 values]."""
    out = []
    for i in range(len(q)):
        state = state * decay[i][:, None, None]
        d = (v[i] - torch.bmm(k[i][:, None], state)[:, 0]) * beta[i][:, None]
        state = torch.baddbmm(state, k[i][:, :, None], d[:, None])
        out.append(torch.bmm(q[i][:, None], state)[:, 0])
    return torch.stack(out), state


def exact_stack(c, seed):
    t = stack_tensors(c, seed)
    g64 = lambda l, name: t[l, name].to(F64)
    G, n = N.LAYER_GLOBAL, c["prompt"] + c["tokens"]
    ids = torch.tensor(tokens_of(c["vocab"], c["prompt"] + max(c["tokens"], 64), seed)[:n], device=DEV)
    x = t[G, N.T_EMBED][ids].to(F64)
    latent = c["design"] == "latent"
    ln = lambda v, wt: torch.nn.functional.layer_norm(v, v.shape[-1:], eps=1e-6) * wt
    norm = ln if latent else (lambda v, wt: rms(v) * wt)
    first = None
    for l in range(c["layers"]):
        m = lambda name: g64(l, name)
        h = norm(x, m(N.T_INPUT_NORM))
        if latent:
            H = c["heads"]
            q = (rms(h @ m(N.T_Q_DOWN).T) * m(N.T_Q_DOWN_NORM) @ m(N.T_Q_UP).T).view(n, H, 192)
            down = h @ m(N.T_KV_DOWN).T
            lat = rms(down[:, :512]) * m(N.T_KV_DOWN_NORM)
            pairs = lambda v: rotate_pairs(v, 10000.0)
            q = torch.cat([q[..., :128], pairs(q[..., 128:])], -1)
            k = torch.cat([(lat @ m(N.T_K_UP).T).view(n, H, 128), pairs(down[:, None, 512:]).expand(n, H, 64)], -1)
            y = attend(q, k, (lat @ m(N.T_V_UP).T).view(n, H, 128), 192 ** -0.5, c["window"]) @ m(N.T_ATTN_O).T
            x = x + norm(y, m(N.T_MIX_OUT_NORM))
            y = torch.relu(norm(x, m(N.T_POST_NORM)) @ m(N.T_MLP_UP).T) ** 2 @ m(N.T_MLP_DOWN).T
            x = x + norm(y, m(N.T_MLP_OUT_NORM))
            continue
        if l % 2:
            x = x + memory64(h, m, c["memory_heads"]) @ m(N.T_ATTN_O).T
        else:
            H, K = c["heads"], c["kv_heads"]
            q = (rms(h @ m(N.T_MIX_Q).T + m(N.T_MIX_Q_BIAS)) * m(N.T_Q_NORM)).view(n, H, 128)
            k = (rms(h @ m(N.T_MIX_K).T + m(N.T_MIX_K_BIAS)) * m(N.T_K_NORM)).view(n, K, 128)
            v = (h @ m(N.T_MIX_V).T + m(N.T_MIX_V_BIAS)).view(n, K, 128)
            mix = m(N.T_V_MIX)
            first, v = (v, v) if first is None else (first, (1 - mix) * v + mix * first)
            y = attend(rotate_halves(q, 64, 10000.0), rotate_halves(k, 64, 10000.0), v, 128 ** -0.5, c["window"], m(N.T_ATTN_SINK))
            x = x + y @ m(N.T_ATTN_O).T + m(N.T_MIX_O_BIAS)
        h = norm(x, m(N.T_POST_NORM))
        gate, up = (h @ m(N.T_MLP_GATE).T).clamp(max=7.0), (h @ m(N.T_MLP_UP).T).clamp(-7.0, 7.0)
        x = x + (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ m(N.T_MLP_DOWN).T
    last = norm(x, g64(G, N.T_FINAL_NORM))
    logits = last[[c["prompt"] - 1, n - 1]] @ g64(G, N.T_LM_HEAD if latent else N.T_EMBED).T
    if latent:
        logits = 30.0 * torch.tanh(logits / 30.0)
    return dict(first=logits[:1], hidden=last[-1], **({"logits": logits[1]} if c["tokens"] else {}))


def rotate_pairs(x, base):
    """x [tokens, heads, dims]: dimension 2i is turned with 2i + 1."""
    d = x.shape[-1]
    angle = torch.arange(x.shape[0], device=DEV, dtype=F64)[:, None, None] * base ** (-torch.arange(0, d, 2, device=DEV, dtype=F64) / d)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * angle.cos() - v * angle.sin(), v * angle.cos() + u * angle.sin()], -1).flatten(-2)


def memory64(h, m, H):
    n = len(h)
    q = (h @ m(N.T_MIX_Q).T * 256 ** -0.5).view(n, H, 256)
    k, v = (h @ m(N.T_MIX_K).T).view(n, H, 256), (h @ m(N.T_MIX_V).T).view(n, H, 512)
    cap = lambda z: 15.0 * torch.tanh(z / 15.0)
    i = cap(h @ m(N.T_MEM_IN).T + m(N.T_MEM_IN_BIAS))
    f = torch.nn.functional.logsigmoid(cap(h @ m(N.T_MEM_FORGET).T + m(N.T_MEM_FORGET_BIAS)))
    S, s, top, out = h.new_zeros(H, 256, 512), h.new_zeros(H, 256), h.new_zeros(H), []
    for t in range(n):
        new = torch.maximum(f[t] + top, i[t])
        keep, take = torch.exp(f[t] + top - new), torch.exp(i[t] - new)
        kt = k[t] * take[:, None]
        S = torch.baddbmm(S * keep[:, None, None], kt[:, :, None], v[t][:, None])
        s = s * keep[:, None] + kt
        top = new
        den = torch.maximum((s * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        out.append(torch.bmm(q[t][:, None], S)[:, 0] / den[:, None])
    return rms(torch.stack(out)).reshape(n, -1) * m(N.T_MIX_HEAD_NORM) * torch.sigmoid(h @ m(N.T_MIX_GATE).T)


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind in ("matvec", "fanout"):
        x, mats = op_inputs(case, seed)
        return [x.to(F64) @ values64(m).T for m in mats]
    if kind == "head":
        m, hidden, _ = head_inputs(case, seed)
        part = -(-m["rows"] // 8)
        rows = [values64(dict(m, rows=b.shape[0], blocks=b, s_out=so)) for b, so in zip(m["blocks"].split(part), m["s_out"].split(part))]
        return dict(logits=torch.cat([hidden.to(F64) @ r.T for r in rows], -1), greedy=None)
    if kind == "delta":
        i = {k: v.to(F64) for k, v in delta_inputs(case, seed).items()}
        L, T, H = case["layers"], case["tokens"], case["heads"]
        unit = lambda v: (v * torch.rsqrt((v * v).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // case["qk_heads"], 2).transpose(0, 1).reshape(T, L * H, 128)
        line = lambda v: v.transpose(0, 1).reshape(T, L * H, *v.shape[3:])
        out, state = delta64(unit(i["q"]) * 128 ** -0.5, unit(i["k"]), line(i["v"]), line(torch.exp(i["g"])), line(i["beta"]), i["state"].reshape(L * H, 128, 128))
        return dict(out=out.view(T, L, H, 128).transpose(0, 1), state=state.view(L, H, 128, 128))
    if kind == "hybrid":
        return exact_hybrid(case, seed)
    if kind == "stack" and case["weights"] == "seeded":
        return exact_stack(case, seed)
    return None
