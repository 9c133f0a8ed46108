"""The work that users of the framework have it do, as timed cases: decoding layers, sampling, prefill, attention, training
blocks, convolution blocks and the optimizer, each through the entry points that a program calls.

Layer dimensions are those of the configurations of ``models/sciagent.py`` (350m, 12-layer benchmark model, 7b, llama3_8b)
and of ``models/cnn.py``; all weights and inputs are random."""
import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from scirust_b200 import ops
from scirust_b200.generate import SamplingParams
from scirust_b200.models.cnn import BasicBlock
from scirust_b200.models.infer import InferenceEngine
from scirust_b200.models.sciagent import GQADecoder, SciAgentConfig
from scirust_b200.ops import attention as att, conv as conv_ops, decode as D
from scirust_b200.ops.sampling import DeviceSampler

BF = torch.bfloat16
F64 = torch.float64
DEV = "cuda"
EPS = 1e-5
PAGE = 64
# d_model, heads, kv heads, d_ff, vocabulary, RoPE base of the repository's configurations
DIMS = {"350m": (1024, 16, 4, 2816, 32768, 1e6), "gqa_12l": (1024, 16, 4, 2816, 32000, 1e4),
        "7b": (4096, 32, 8, 11008, 32768, 1e6), "llama3_8b": (4096, 32, 8, 14336, 128256, 5e5)}


def listed():
    return [
        # one decoder layer of a small model, one user, short context: the smallest call, bound by latency
        dict(name="decode_350m_1", kind="decode", dims="350m", rows=1, ctx=128, quant=False, graph=False),
        # one decoder layer of an 8B model for one user at the benchmark's context; captured once and replayed, as the
        # inference engine does with its decode step
        dict(name="decode_8b_1", kind="decode", dims="llama3_8b", rows=1, ctx=2048, quant=False, graph=True),
        # the same for a batch of 16 with int8 weights
        dict(name="decode_8b_16_int8", kind="decode", dims="llama3_8b", rows=16, ctx=2304, quant=True, graph=True),
        # and for the benchmark's largest batch, bf16
        dict(name="decode_8b_64", kind="decode", dims="llama3_8b", rows=64, ctx=2048, quant=False, graph=True),
        # sampled decoding: one token per sequence from the logits of a 128k vocabulary
        dict(name="sample_16", kind="sample", rows=16, vocab=128256, top_k=50, top_p=0.95, temperature=0.8, penalty=1.0),
        # a whole prefill call of the inference engine: int8 weights, one prompt of the benchmark's length
        dict(name="prefill_8b_int8", kind="prefill", dims="llama3_8b", layers=2, batch=1, seq=2048, quant=True),
        # causal attention of a long prompt of ragged length, head dimension 128
        dict(name="attention_prefill", kind="attention", dims="llama3_8b", batch=1, seq=5000, backward=False),
        # training attention at head dimension 128, forward and backward
        dict(name="attention_train", kind="attention", dims="7b", batch=2, seq=2048, backward=True),
        # forward and backward of two layers, embedding, head and loss of the benchmark's model at the benchmark's batch
        dict(name="train_12l", kind="train", dims="gqa_12l", layers=2, batch=8, seq=2048),
        # a short ragged fine-tuning batch through one layer
        dict(name="train_ragged", kind="train", dims="350m", layers=1, batch=3, seq=333),
        # a residual block of the CIFAR ResNet, forward and backward
        dict(name="conv_block", kind="conv", batch=128, size=32, c_in=64, c_out=64, stride=1),
        # gradient norm and AdamW update of a flat parameter buffer
        dict(name="optimizer", kind="optimizer", n=60_000_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "sample", "prefill", "attention", "train", "conv", "optimizer"])
    if kind == "decode":
        rows = _log_int(rng, 1, 64)
        return dict(kind=kind, dims=rng.choice(["350m", "7b", "llama3_8b"]), rows=rows, ctx=_log_int(rng, 16, 2048),
                    quant=rng.random() < 0.4, graph=rng.random() < 0.7)
    if kind == "sample":
        return dict(kind=kind, rows=_log_int(rng, 1, 64), vocab=rng.choice([256, 32000, 32768, 128256]),
                    top_k=rng.choice([0, 20, 50]), top_p=rng.choice([1.0, 0.9, 0.95]),
                    temperature=rng.choice([0.7, 0.8, 1.0]), penalty=rng.choice([1.0, 1.1]))
    if kind == "prefill":
        return dict(kind=kind, dims=rng.choice(["350m", "7b"]), layers=1, batch=rng.randint(1, 4),
                    seq=_log_int(rng, 33, 2048), quant=rng.random() < 0.5)
    if kind == "attention":
        backward = rng.random() < 0.5
        return dict(kind=kind, dims=rng.choice(["350m", "7b"]), batch=rng.randint(1, 3),
                    seq=_log_int(rng, 100, 2048 if backward else 4096), backward=backward)
    if kind == "train":
        return dict(kind=kind, dims=rng.choice(["350m", "gqa_12l"]), layers=rng.randint(1, 2), batch=rng.randint(1, 4),
                    seq=_log_int(rng, 64, 2048))
    if kind == "conv":
        size, c = rng.choice([(32, 64), (16, 128), (8, 256)])
        down = rng.random() < 0.4
        return dict(kind=kind, batch=_log_int(rng, 16, 128), size=size, c_in=c, c_out=2 * c if down else c,
                    stride=2 if down else 1)
    return dict(kind=kind, n=_log_int(rng, 100_000, 60_000_000))


# ---------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape, std=1.0, dtype=BF):
    return (torch.randn(shape, generator=g, device=DEV) * std).to(dtype)


def _layer_weights(g, dims):
    d, H, Hkv, ff, _, _ = DIMS[dims]
    dh = d // H
    return {"rms1": _randn(g, d, std=0.1) + 1, "wqkv": _randn(g, d, (H + 2 * Hkv) * dh, std=0.02),
            "wo": _randn(g, d, d, std=0.02), "rms2": _randn(g, d, std=0.1) + 1,
            "wgu": _randn(g, d, 2 * ff, std=0.02), "wd": _randn(g, ff, d, std=0.02)}


def _decode_inputs(case, seed):
    g = _gen(seed)
    d, H, Hkv, ff, _, theta = DIMS[case["dims"]]
    dh, B, ctx = d // H, case["rows"], case["ctx"]
    w = _layer_weights(g, case["dims"])
    blocks = (ctx + PAGE - 1) // PAGE
    # tokens already in the cache of each sequence: at least three quarters of the longest
    past = torch.randint(ctx * 3 // 4, ctx, (B,), generator=g, device=DEV).int()
    past[0] = ctx - 1
    table = torch.randperm(B * blocks, generator=g, device=DEV).int().reshape(B, blocks)
    pool = _randn(g, B * blocks, 2, Hkv, PAGE, dh)
    return w, _randn(g, B, d), past, table, pool


def _model_inputs(case, seed):
    g = _gen(seed)
    d, H, Hkv, ff, V, theta = DIMS[case["dims"]]
    layers = [_layer_weights(g, case["dims"]) for _ in range(case["layers"])]
    embed = _randn(g, V, d, std=0.02)
    head = _randn(g, V, d, std=0.02) if case["dims"] == "llama3_8b" else None
    rms = _randn(g, d, std=0.1) + 1
    tokens = torch.randint(0, V, (case["batch"], case["seq"] + 1), generator=g, device=DEV)
    return layers, embed, head, rms, tokens[:, :-1].contiguous(), tokens[:, 1:].contiguous()


def _model(case, seed):
    d, H, Hkv, ff, V, theta = DIMS[case["dims"]]
    layers, embed, head, rms, tokens, targets = _model_inputs(case, seed)
    cfg = SciAgentConfig(V, d, case["layers"], H, Hkv, ff, 4096, theta, tie_embeddings=head is None)
    model = GQADecoder(cfg, device=DEV)
    with torch.no_grad():
        model.embed.copy_(embed)
        model.rms_final.copy_(rms)
        if head is not None:
            model.lm_head.copy_(head)
        for l, w in zip(model.layers, layers):
            for to, name in ((l.rms_attn, "rms1"), (l.wqkv, "wqkv"), (l.wo, "wo"), (l.rms_ffn, "rms2"), (l.wgu, "wgu"),
                             (l.wd, "wd")):
                to.copy_(w[name])
    return model, tokens, targets


def _sample_inputs(case, seed):
    g = _gen(seed)
    logits = _randn(g, case["rows"], case["vocab"], std=2.5, dtype=torch.float32)
    prompt = torch.randint(0, case["vocab"], (case["rows"], 32), generator=g, device=DEV)
    return logits, prompt


def _attention_inputs(case, seed):
    g = _gen(seed)
    d, H, Hkv, _, _, _ = DIMS[case["dims"]]
    dh, n = d // H, case["batch"] * case["seq"]
    return _randn(g, n, (H + 2 * Hkv) * dh), _randn(g, n, d)


def _conv_block(case, seed):
    block = BasicBlock(case["c_in"], case["c_out"], case["stride"], torch.Generator().manual_seed(int(seed))).to(DEV)
    return block, conv_ops.ConvGeom(case["batch"], case["size"], case["size"], case["c_in"])


def _conv_inputs(case, seed):
    g = _gen(seed)
    out = case["size"] // case["stride"]
    x = torch.relu(_randn(g, case["batch"] * case["size"] ** 2, case["c_in"]))
    return x, _randn(g, case["batch"] * out * out, case["c_out"], std=0.1)


def _optimizer_inputs(case, seed):
    g = _gen(seed)
    n = case["n"]
    p = _randn(g, n, std=0.02, dtype=torch.float32)
    m = _randn(g, n, std=1e-4, dtype=torch.float32)
    v = _randn(g, n, std=1e-4, dtype=torch.float32).square()
    return p, m, v, _randn(g, n, std=1e-3)


ADAMW = dict(lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, max_grad_norm=1.0)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "decode":
        d, H, Hkv, ff, _, theta = DIMS[case["dims"]]
        w, x, past, table, pool = _decode_inputs(case, seed)
        if case["quant"]:
            for k in ("wqkv", "wo", "wgu", "wd"):
                w[k] = D.quantize_per_channel(w[k])
                if case["rows"] > 8:
                    w[k].transposed()
        cos, sin = ops.rope_table(8192, d // H, theta, torch.device(DEV))
        s.update(w=w, x=x, past=past, length=past + 1, table=table, pool=pool, cos=cos, sin=sin,
                 seq_of=torch.arange(case["rows"], dtype=torch.int32, device=DEV))
        if case["graph"]:
            graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream(device=DEV)
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                _run_decode(s)                   # allocates the workspaces before the capture
                with torch.cuda.graph(graph, stream=stream):
                    out = _run_decode(s)
            torch.cuda.current_stream().wait_stream(stream)
            s["replay"] = (graph, out)
    elif kind == "sample":
        logits, prompt = _sample_inputs(case, seed)
        params = SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"],
                                repetition_penalty=case["penalty"])
        sampler = DeviceSampler(params, case["rows"], case["vocab"], [seed + b for b in range(case["rows"])], DEV,
                                history_len=64)
        sampler.set_history(prompt)
        s.update(logits=logits, sampler=sampler)
    elif kind == "prefill":
        model, tokens, _ = _model(case, seed)
        s.update(engine=InferenceEngine(model, quant="int8" if case["quant"] else None, max_batch=case["batch"],
                                        max_seq=case["seq"] + 64), tokens=tokens)
    elif kind == "attention":
        s["qkv"], s["do"] = _attention_inputs(case, seed)
    elif kind == "train":
        s["model"], s["tokens"], s["targets"] = _model(case, seed)
    elif kind == "conv":
        s["block"], s["geom"] = _conv_block(case, seed)
        s["x"], s["dy"] = _conv_inputs(case, seed)
        s["x"].requires_grad_(True)
    else:
        s["p"], s["m"], s["v"], s["grad"] = _optimizer_inputs(case, seed)
        s["p_bf16"] = s["p"].to(BF)
        s["step"] = 10
    return s


# ---------------------------------------------------------------------------------------------- passes
def _linear(x, w, residual=None):
    if D.skinny_ok(x, w):
        return D.matmul_skinny(x, w, residual=residual)
    if isinstance(w, D.QuantWeight):
        return D.matmul_int8(x, w, residual=residual)
    return ops.matmul_nn(x, w, residual=residual)


def _run_decode(s):
    d, H, Hkv, ff, _, _ = DIMS[s["dims"]]
    dh, w, x = d // H, s["w"], s["x"]
    few = x.shape[0] <= D.gemv_max_rows(w["wqkv"])
    if few:
        qkv = D.gemv(x, w["wqkv"], rms_weight=w["rms1"], eps=EPS)
    else:
        qkv = _linear(ops.rmsnorm_fwd(x, w["rms1"], EPS, want_inv=False)[0], w["wqkv"])
    D.rope_kv_append(qkv, H, Hkv, dh, s["cos"], s["sin"], s["pool"], s["table"], PAGE, s["seq_of"], s["past"])
    a = D.decode_attention(qkv, s["pool"], s["table"], PAGE, s["length"], H, Hkv, dh, max_len=s["ctx"])
    if few:
        x = D.gemv(a, w["wo"], residual=x)
        gu = D.gemv(x, w["wgu"], rms_weight=w["rms2"], eps=EPS)
        y = D.gemv(gu, w["wd"], residual=x, swiglu=True)
    else:
        x = _linear(a, w["wo"], residual=x)
        gu = _linear(ops.rmsnorm_fwd(x, w["rms2"], EPS, want_inv=False)[0], w["wgu"])
        y = _linear(ops.swiglu_fwd(gu), w["wd"], residual=x)
    return {"qkv": qkv, "attention": a, "y": y, "pool": s["pool"]}


def run(state):
    s = state
    kind = s["kind"]
    if kind == "decode":
        if not s["graph"]:
            return _run_decode(s)
        graph, out = s["replay"]
        graph.replay()
        return out
    if kind == "sample":
        tokens = s["sampler"].sample(s["logits"])
        return {"tokens": tokens, "rng": s["sampler"].state}
    if kind == "prefill":
        with torch.no_grad():
            return {"logits": s["engine"].prefill(s["tokens"]), "pools": s["engine"].cache.pools}
    if kind == "attention":
        d, H, Hkv, _, _, _ = DIMS[s["dims"]]
        shape = (s["batch"], s["seq"], H, Hkv, d // H)
        o, lse = att.attention_fwd(s["qkv"], *shape, causal=True, want_lse=s["backward"])
        if not s["backward"]:
            return {"o": o}
        return {"o": o, "lse": lse, "dqkv": att.attention_bwd(s["qkv"], o, lse, s["do"], *shape, causal=True)}
    if kind == "train":
        model = s["model"]
        model.zero_grad_flags()
        loss = model(s["tokens"], s["targets"])
        loss.backward()
        return {"loss": loss.detach(), "grads": [p.main_grad for _, p, _ in model.ordered_params()]}
    if kind == "conv":
        y, _ = s["block"](s["x"], s["geom"])
        grads = torch.autograd.grad(y, [s["x"], *s["block"].parameters()], s["dy"])
        return {"y": y.detach(), "grads": list(grads), "running": [b.detach() for b in s["block"].buffers()]}
    sq = ops.sumsq(s["grad"])
    ops.optim_step(s["p"], s["m"], s["v"], s["grad"], s["p_bf16"], step=s["step"], grad_sumsq=sq, **ADAMW)
    s["step"] += 1
    return {"p": s["p"], "m": s["m"], "v": s["v"], "p_bf16": s["p_bf16"], "sumsq": sq}


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": case["rows"] * case["vocab"] * 4, "flops": case["rows"] * case["vocab"] * 4}
    if kind == "optimizer":
        return {"bytes": case["n"] * 28, "flops": case["n"] * 20}
    if kind == "conv":
        b, hw, ci, co = case["batch"], case["size"] ** 2, case["c_in"], case["c_out"]
        ohw = hw // case["stride"] ** 2
        macs = b * ohw * co * (9 * ci + 9 * co + (ci if ci != co else 0))
        # x, dy read; y, dx written
        return {"bytes": 2 * b * (2 * hw * ci + 2 * ohw * co), "flops": 6 * macs}
    d, H, Hkv, ff, V, _ = DIMS[case["dims"]]
    dh = d // H
    qkv = (H + 2 * Hkv) * dh
    weights = d * qkv + d * d + 3 * d * ff
    if kind == "decode":
        kv = case["rows"] * (case["ctx"] * 7 // 8) * 2 * Hkv * dh
        return {"bytes": weights * (1 if case["quant"] else 2) + kv * 2 + case["rows"] * d * 4,
                "flops": 2 * case["rows"] * weights + 2 * kv * (H // Hkv)}
    n = case["batch"] * case["seq"]
    scores = 2 * n * (case["seq"] + 1) * d          # two products over the lower triangle, multiply and add
    if kind == "attention":
        passes = 1 if not case["backward"] else 3.5
        return {"bytes": 2 * n * (qkv + d) * (1 if not case["backward"] else 3), "flops": passes * scores}
    if kind == "prefill":
        return {"bytes": case["layers"] * weights * (1 if case["quant"] else 2) + V * d * (1 if case["quant"] else 2)
                + n * d * 2 + case["layers"] * n * 4 * Hkv * dh,
                "flops": case["layers"] * (2 * n * weights + scores) + 2 * case["batch"] * V * d}
    total = case["layers"] * weights + V * d
    return {"bytes": 4 * total + 2 * n * d, "flops": 6 * n * total + 3.5 * case["layers"] * scores}


def tolerance(case):
    # int8 activations: a rounding that differs moves a code, 1/254 of the row's largest value; the convolution block has
    # ReLU masks in its gradients, which a rounding near zero flips
    if case.get("quant"):
        return {"rel": 3e-2, "max": 0.6}
    return {"decode": {"rel": 1e-2, "max": 0.2}, "sample": "exact", "prefill": {"rel": 1.5e-2, "max": 0.2},
            "attention": {"rel": 1e-2, "max": 0.3}, "train": {"rel": 2e-2, "max": 0.5},
            "conv": {"rel": 3e-2, "max": 0.9}, "optimizer": {"rel": 1e-4, "max": 1e-2}}[case["kind"]]


# ---------------------------------------------------------------------------------------------- 64-bit statements
def _rms64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w.to(F64)


def _codes(w, axis):
    mx = w.float().abs().amax(axis, keepdim=True)
    scale = torch.where(mx == 0, torch.ones_like(mx), mx / 127.0)
    v = w.float() / scale
    q = torch.where(v >= 0, torch.floor(v + 0.5), torch.ceil(v - 0.5)).clamp(-128, 127)
    return q.to(F64) * scale.to(F64)


def _dense64(x, w, quant, rows):
    """x . w; int8 weights are per output column, and between 9 and 1023 rows the activations are int8 per row too."""
    if not quant:
        return x @ w.to(F64)
    if 8 < rows < 1024:
        x = _codes(x, 1)
    return x @ _codes(w, 0)


def _rope64(x, heads, dh, pos, theta):
    """Interleaved pairs of the first ``heads`` heads of x [n, *] at the positions pos [n]."""
    freq = theta ** (-2.0 * torch.arange(dh // 2, device=x.device, dtype=F64) / dh)
    ang = pos.to(F64)[:, None] * freq
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    v = x[:, :heads * dh].reshape(x.shape[0], heads, dh // 2, 2)
    r = torch.stack((v[..., 0] * c - v[..., 1] * s, v[..., 0] * s + v[..., 1] * c), -1)
    return torch.cat((r.reshape(x.shape[0], heads * dh), x[:, heads * dh:]), 1)


def _attention64(qkv, B, S, H, Hkv, dh):
    """Causal attention, one sequence and key/value head at a time: (o [B*S, H*dh], lse [B, H, S])."""
    G = H // Hkv
    mask = torch.ones(S, S, dtype=torch.bool, device=qkv.device).triu(1)
    x = qkv.reshape(B, S, H + 2 * Hkv, dh)
    o, lse = [], []
    for b in range(B):
        for h in range(Hkv):
            q = x[b, :, h * G:(h + 1) * G].transpose(0, 1)
            s = (q @ x[b, :, H + h].T / math.sqrt(dh)).masked_fill(mask, float("-inf"))
            l = torch.logsumexp(s, -1)
            o.append(torch.exp(s - l[..., None]) @ x[b, :, H + Hkv + h])
            lse.append(l)
    o = torch.stack(o).reshape(B, H, S, dh).transpose(1, 2).reshape(B * S, H * dh)
    return o, torch.stack(lse).reshape(B, H, S)


def _block64(x, w, case):
    d, H, Hkv, ff, _, theta = DIMS[case["dims"]]
    dh, B, S, rows, quant = d // H, case["batch"], case["seq"], x.shape[0], case.get("quant", False)
    qkv = _dense64(_rms64(x, w["rms1"]), w["wqkv"], quant, rows)
    qkv = _rope64(qkv, H + Hkv, dh, torch.arange(S, device=x.device).repeat(B), theta)
    x = x + _dense64(_attention64(qkv, B, S, H, Hkv, dh)[0], w["wo"], quant, rows)
    gu = _dense64(_rms64(x, w["rms2"]), w["wgu"], quant, rows)
    return x + _dense64(F.silu(gu[:, :ff]) * gu[:, ff:], w["wd"], quant, rows)


def _exact_decode(case, seed):
    d, H, Hkv, ff, _, theta = DIMS[case["dims"]]
    dh, G, B, quant = d // H, H // Hkv, case["rows"], case["quant"]
    w, x, past, table, pool = _decode_inputs(case, seed)
    x = x.to(F64)
    qkv = _rope64(_dense64(_rms64(x, w["rms1"]), w["wqkv"], quant, B), H + Hkv, dh, past, theta)
    pool64 = pool.to(F64)
    kv = qkv[:, H * dh:].reshape(B, 2, Hkv, dh)
    a = torch.zeros(B, H * dh, dtype=F64, device=DEV)
    for b in range(B):
        n = int(past[b]) + 1
        pool64[table[b, (n - 1) // PAGE].long(), :, :, (n - 1) % PAGE] = kv[b]
        got = pool64[table[b].long()].permute(1, 2, 0, 3, 4).reshape(2, Hkv, -1, dh)[:, :, :n]
        q = qkv[b, :H * dh].reshape(Hkv, G, dh)
        a[b] = (torch.softmax(q @ got[0].transpose(-1, -2) / math.sqrt(dh), -1) @ got[1]).reshape(-1)
    x = x + _dense64(a, w["wo"], quant, B)
    gu = _dense64(_rms64(x, w["rms2"]), w["wgu"], quant, B)
    y = x + _dense64(F.silu(gu[:, :ff]) * gu[:, ff:], w["wd"], quant, B)
    return {"qkv": qkv, "attention": a, "y": y, "pool": pool64}


def _exact_train(case, seed):
    layers, embed, _, rms, tokens, targets = _model_inputs(case, seed)

    def leaf(t):
        return t.to(F64).requires_grad_(True)

    embed, rms = leaf(embed), leaf(rms)
    layers = [{k: leaf(v) for k, v in w.items()} for w in layers]
    with torch.enable_grad():
        x = embed[tokens.reshape(-1)]
        for w in layers:
            x = _block64(x, w, case)
        hidden = _rms64(x, rms)
        loss = 0.0
        for r in range(0, hidden.shape[0], 4096):
            part = checkpoint(
                lambda h, t: F.cross_entropy(h @ embed.T, t, reduction="sum"), hidden[r:r + 4096],
                targets.reshape(-1)[r:r + 4096], use_reentrant=False)
            loss = loss + part
        loss = loss / hidden.shape[0]
        order = [embed] + [w[k] for w in layers for k in ("wqkv", "wo", "wgu", "wd")]
        order += [w[k] for w in layers for k in ("rms1", "rms2")] + [rms]
        grads = torch.autograd.grad(loss, order)
    return {"loss": loss.detach(), "grads": list(grads)}


def _exact_conv(case, seed):
    block, _ = _conv_block(case, seed)
    x, dy = _conv_inputs(case, seed)
    n, hw, stride = case["batch"], case["size"], case["stride"]
    params = [p.detach().to(BF if p.dim() == 2 else F64).to(F64).requires_grad_(True) for p in block.parameters()]
    x = x.to(F64).requires_grad_(True)
    buffers = [b.to(F64) for b in block.buffers()]

    def conv_bn(t, i, k, stride):
        w, gamma, beta = params[3 * i:3 * i + 3]
        c = t.shape[1]
        t = F.conv2d(t, w[:, :k * k * c].reshape(-1, k, k, c).permute(0, 3, 1, 2), stride=stride, padding=k // 2)
        return F.batch_norm(t, buffers[2 * i], buffers[2 * i + 1], gamma, beta, True, 0.1, 1e-5)

    with torch.enable_grad():
        x4 = x.reshape(n, hw, hw, -1).permute(0, 3, 1, 2)
        y = conv_bn(torch.relu(conv_bn(x4, 0, 3, stride)), 1, 3, 1)
        y = torch.relu(y + (conv_bn(x4, 2, 1, stride) if len(params) > 6 else x4))
        y = y.permute(0, 2, 3, 1).reshape(-1, case["c_out"])
        grads = torch.autograd.grad(y, [x, *params], dy.to(F64))
    return {"y": y.detach(), "grads": list(grads), "running": buffers}


def _exact_optimizer(case, seed):
    p, m, v, grad = (t.to(F64) for t in _optimizer_inputs(case, seed))
    sq = grad.square().sum()
    g = grad * min(1.0, ADAMW["max_grad_norm"] / math.sqrt(float(sq)))
    b1, b2, step = ADAMW["beta1"], ADAMW["beta2"], 10
    m = b1 * m + (1 - b1) * g
    v = b2 * v + (1 - b2) * g * g
    update = (m / (1 - b1 ** step)) / (torch.sqrt(v / (1 - b2 ** step)) + ADAMW["eps"]) + ADAMW["weight_decay"] * p
    p = p - ADAMW["lr"] * update
    return {"p": p, "m": m, "v": v, "p_bf16": p, "sumsq": sq.reshape(1)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return None
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "conv":
        return _exact_conv(case, seed)
    with torch.no_grad():
        if kind == "decode":
            return _exact_decode(case, seed)
        if kind == "optimizer":
            return _exact_optimizer(case, seed)
        if kind == "prefill":
            layers, embed, head, rms, tokens, _ = _model_inputs(case, seed)
            x = embed[tokens.reshape(-1)].to(F64)
            for w in layers:
                x = _block64(x, w, case)
            last = _rms64(x.reshape(case["batch"], case["seq"], -1)[:, -1], rms)
            head = (embed if head is None else head).t().contiguous()
            return {"logits": _dense64(last, head, case["quant"], case["batch"]), "pools": [None] * case["layers"]}
    d, H, Hkv, _, _, _ = DIMS[case["dims"]]
    shape = (case["batch"], case["seq"], H, Hkv, d // H)
    qkv, do = _attention_inputs(case, seed)
    qkv = qkv.to(F64).requires_grad_(case["backward"])
    with torch.set_grad_enabled(case["backward"]):
        o, lse = _attention64(qkv, *shape)
        if not case["backward"]:
            return {"o": o}
        return {"o": o.detach(), "lse": lse.detach(), "dqkv": torch.autograd.grad(o, qkv, do.to(F64))[0]}
