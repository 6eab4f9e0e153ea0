"""The work that a user of this library has it do, as cases that can be timed: the calls of the public Python face
(``nntrainer_b200.backend``, ``nntrainer_b200.decoder``) on the shapes of the benchmark's and the tests' configurations,
over the whole range of each call.

kind "host"     the drop-in for the reference's gemm_*: activations and results in host memory, the weight resident
kind "gemm"     a projection on device tensors; M = 1 is a decode step, a few rows are concurrent streams, many a prefill
kind "moe"      one mixture-of-experts layer, Qwen form (Q4_K experts) or GPT-OSS form (Q4_0 experts, biases)
kind "attn"     one token's attention over an fp16 cache
kind "replay"   greedy decoding of a dense decoder at a given context from a captured CUDA graph
kind "generate" the same decoder fed a prompt and asked for new tokens
"""
import math
import os
import tempfile
import weakref

import torch

from nntrainer_b200 import backend as be
from nntrainer_b200.decoder import DecoderConfig, Qwen3Decoder, tensor_list

BYTES_PER_WEIGHT = {"q4_K": 144 / 256, "q4_0": 18 / 32, "q6_K": 210 / 256}
MOE_SHAPES = {  # hidden, expert width, experts, experts per token
    "qwen": ("q4_K", 2048, 768, 128, 8),
    "gpt_oss": ("q4_0", 2880, 2880, 32, 4),
}
MOST_FLOPS = 2 * 1024 * 24576 * 4096


def listed():
    return [
        # one projection of one token called from the host framework: A and C in host memory, the weight uploaded once
        dict(name="host q4_K 1x4096x4096", kind="host", qtype="q4_K", M=1, N=4096, K=4096),
        # the smallest device call: one projection of one token, a width that is no multiple of 128
        dict(name="gemm q4_0 1x2880x2880", kind="gemm", qtype="q4_0", M=1, N=2880, K=2880),
        # the q|k|v projection of eight concurrent decode streams
        dict(name="gemm q4_K 8x6144x2560", kind="gemm", qtype="q4_K", M=8, N=6144, K=2560),
        # the lm_head of eight concurrent decode streams
        dict(name="gemm q6_K 8x151936x2560", kind="gemm", qtype="q6_K", M=8, N=151936, K=2560),
        # prefill of a prompt of odd length through a square projection whose width is no multiple of 128
        dict(name="gemm q4_0 509x2880x2880", kind="gemm", qtype="q4_0", M=509, N=2880, K=2880),
        # prefill of 1024 tokens through a fused gate+up projection: the largest product of the configurations
        dict(name="gemm q4_K 1024x24576x4096", kind="gemm", qtype="q4_K", M=1024, N=24576, K=4096),
        # one decode token through a 128-expert layer
        dict(name="moe qwen 1", kind="moe", form="qwen", tokens=1),
        # prefill of 256 tokens through the same layer
        dict(name="moe qwen 256", kind="moe", form="qwen", tokens=256),
        # eight concurrent decode streams through a 32-expert layer with biases
        dict(name="moe gpt_oss 8", kind="moe", form="gpt_oss", tokens=8),
        # attention of one token at context 4096, 64 / 8 heads of 64 with sinks
        dict(name="attn 64/8x64 4096", kind="attn", heads=64, kv_heads=8, head_dim=64, rows=4096, window=0, sink=True,
             qk_norm=False),
        # greedy decoding at context 512: four layers with the layer dimensions of the 4B shape, 16 tokens
        dict(name="replay 4 layers 512+16", kind="replay", layers=4, context=512, new=16, vocab=32768),
        # the whole call a user makes: a prompt of 64 tokens, then 32 new ones
        dict(name="generate 4 layers 64+32", kind="generate", layers=4, context=64, new=32, vocab=32768),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(x, of):
    return max(of, x // of * of)


def draw(rng):
    kind = rng.choice(["host", "gemm", "gemm", "gemm", "gemm", "moe", "moe", "attn", "replay", "generate"])
    if kind in ("host", "gemm"):
        qtype = rng.choice(["q4_K", "q4_0", "q6_K"])
        m_max = 32 if kind == "host" else 1024
        M = 1 if rng.random() < (0.6 if kind == "host" else 0.25) else _log_uniform(rng, 2, m_max)
        # most widths are multiples of 128, some only of the format's row group
        N = _log_uniform(rng, 512, 24576)
        N = _multiple(N, 128) if rng.random() < 0.7 else N if qtype == "q6_K" else _multiple(N, 8)
        K = _multiple(_log_uniform(rng, 512, 12288), 32 if qtype == "q4_0" and rng.random() < 0.5 else 256)
        if qtype == "q6_K" and kind == "gemm" and rng.random() < 0.4:  # an lm_head
            N, K = rng.choice([32768, 151936]), rng.choice([2048, 2560, 4096])
        M = max(1, min(M, MOST_FLOPS // (2 * N * K)))
        return dict(kind=kind, qtype=qtype, M=M, N=N, K=K)
    if kind == "moe":
        return dict(kind=kind, form=rng.choice(["qwen", "gpt_oss"]), tokens=_log_uniform(rng, 1, 400))
    if kind == "attn":
        heads, kv_heads, head_dim = rng.choice([(32, 8, 128), (32, 4, 128), (64, 8, 64)])
        gpt_oss = head_dim == 64
        return dict(kind=kind, heads=heads, kv_heads=kv_heads, head_dim=head_dim, rows=_log_uniform(rng, 16, 6000),
                    window=128 if gpt_oss and rng.random() < 0.5 else 0, sink=gpt_oss, qk_norm=not gpt_oss)
    layers = rng.randint(1, 4)
    if kind == "replay":
        return dict(kind=kind, layers=layers, context=_log_uniform(rng, 16, 1500), new=rng.randint(2, 16),
                    vocab=rng.choice([8192, 32768]))
    return dict(kind=kind, layers=layers, context=_log_uniform(rng, 4, 64), new=rng.randint(2, 32),
                vocab=rng.choice([8192, 32768]))


# ------------------------------------------------------------------------------------------------------------- weights
def _normal(gen, shape, scale=1.0):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).mul_(scale)


def _bytes_of(t):
    return t.contiguous().view(torch.uint8).reshape(*t.shape[:-1], -1)


def _quantize_q4_0(w):
    """[N, K] fp32 -> block_q4_0x8 bytes (8-row interleave, nibbles XOR 8)."""
    N, K = w.shape
    b = w.view(N // 8, 8, K // 32, 32)
    at = b.abs().argmax(-1, keepdim=True)
    d = (b.gather(-1, at) / -8).half()
    inv = torch.where(d != 0, 1 / d.float(), torch.zeros_like(d, dtype=torch.float32))
    q = (b * inv + 8.5).floor().clamp_(0, 15).to(torch.uint8) ^ 8
    qs = q[..., :16] | (q[..., 16:] << 4)                      # byte i: elements i and 16 + i
    qs = qs.view(N // 8, 8, K // 32, 2, 8).permute(0, 2, 3, 1, 4).reshape(N // 8, K // 32, 128)
    d = _bytes_of(d.squeeze(-1).permute(0, 2, 1))
    return torch.cat([d, qs], -1).reshape(-1)


def _quantize_q4_K(w):
    """[N, K] fp32 -> block_q4_Kx8 bytes (8-row interleave)."""
    N, K = w.shape
    b = w.view(N // 8, 8, K // 256, 8, 32)                      # group, row, super-block, sub-block, element
    lo = b.amin(-1).clamp_(max=0)
    scale, mins = (b.amax(-1) - lo) / 15, -lo
    d, dmin = (scale.amax(-1) / 63).half(), (mins.amax(-1) / 63).half()
    df, mf = d.float().clamp_(min=1e-8).unsqueeze(-1), dmin.float().clamp_(min=1e-8).unsqueeze(-1)
    sc, mn = (scale / df).round_().clamp_(1, 63), (mins / mf).round_().clamp_(0, 63)
    q = ((b + (mf * mn).unsqueeze(-1)) / (df * sc).unsqueeze(-1)).round_().clamp_(0, 15).to(torch.uint8)
    q = q.view(N // 8, 8, K // 256, 4, 2, 32)
    qs = (q[..., 0, :] | (q[..., 1, :] << 4)).view(N // 8, 8, K // 256, 16, 8)
    qs = qs.permute(0, 2, 3, 1, 4).reshape(N // 8, K // 256, 1024)
    sc, mn = (t.to(torch.uint8).permute(0, 2, 3, 1) for t in (sc, mn))  # group, super-block, sub-block, row
    s0, s1, m0, m1 = sc[..., :4], sc[..., 4:], mn[..., :4], mn[..., 4:]
    packed = torch.cat([s0 | ((s1 >> 4) << 6), m0 | ((m1 >> 4) << 6), (s1 & 15) | ((m1 & 15) << 4)], -1)
    head = [_bytes_of(t.permute(0, 2, 1)) for t in (d, dmin)]
    return torch.cat(head + [packed.reshape(N // 8, K // 256, 96), qs], -1).reshape(-1)


def _quantize_q6_K(w):
    """[N, K] fp32 -> plain block_q6_K rows."""
    N, K = w.shape
    b = w.view(N, K // 256, 16, 16)
    at = b.abs().argmax(-1, keepdim=True)
    s = b.gather(-1, at).squeeze(-1) / -32
    big = s.gather(-1, s.abs().argmax(-1, keepdim=True))
    d = (big / -128).half()
    df = d.float()
    df = torch.where(df != 0, df, torch.full_like(df, 1e-8))
    sc = (s / df).round_().clamp_(-128, 127)
    ds = df * sc
    ds = torch.where(ds != 0, ds, torch.full_like(ds, 1e-8)).unsqueeze(-1)
    q = ((b / ds).round_().clamp_(-32, 31) + 32).to(torch.uint8).view(N, K // 256, 2, 4, 32)
    ql = torch.cat([(q[..., 0, :] & 15) | ((q[..., 2, :] & 15) << 4), (q[..., 1, :] & 15) | ((q[..., 3, :] & 15) << 4)], -1)
    qh = (q[..., 0, :] >> 4) | ((q[..., 1, :] >> 4) << 2) | ((q[..., 2, :] >> 4) << 4) | ((q[..., 3, :] >> 4) << 6)
    parts = [ql.reshape(N, K // 256, 128), qh.reshape(N, K // 256, 64), _bytes_of(sc.to(torch.int8)), _bytes_of(d)]
    return torch.cat(parts, -1).reshape(-1)


_QUANTIZE = {"q4_0": _quantize_q4_0, "q4_K": _quantize_q4_K, "q6_K": _quantize_q6_K}


def _weight(gen, qtype, N, K):
    """A weight tensor's bytes: N(0, 0.02^2) quantized in slices of rows, which bounds the temporaries."""
    step = max(8, (1 << 26) // K // 8 * 8)
    return torch.cat([_QUANTIZE[qtype](_normal(gen, (min(step, N - i), K), 0.02)) for i in range(0, N, step)])


# --------------------------------------------------------------------------------------------------------------- states
def _decoder(case, gen):
    cfg = DecoderConfig(n_layers=case["layers"], hidden=2560, n_heads=32, n_kv_heads=8, head_dim=128, inter=9728,
                        vocab=case["vocab"], max_seq=case["context"] + case["new"] + 16)
    with tempfile.TemporaryDirectory() as td:  # the decoder reads its weights from a .bin file
        path = os.path.join(td, "model.bin")
        with open(path, "wb") as f:
            for _, dtype, N, K in tensor_list(cfg):
                if dtype == "f32":
                    f.write((1 + _normal(gen, (N, K), 0.1)).cpu().numpy().tobytes())
                else:
                    if dtype == "q4_K":
                        f.write(b"\0\0")  # the quantization-scheme word in front of the data
                    f.write(_weight(gen, dtype, N, K).cpu().numpy().tobytes())
        dec = Qwen3Decoder(cfg, path, pdl=True)
    weakref.finalize(dec, dec.w.close)
    return cfg, dec


def prepare(case, seed):
    be.init(0)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("host", "gemm"):
        qtype, M, N, K = (case[k] for k in ("qtype", "M", "N", "K"))
        W, A = _weight(gen, qtype, N, K), _normal(gen, (M, K))
        if kind == "host":  # activations and results live in the memory the plug-in's allocator hands out
            B = W.cpu().numpy()
            be.register_weight(qtype, B, N, K)
            a, c = be.host_alloc((M, K)), be.host_alloc((M, N))
            a[...] = A.cpu().numpy()
            c[...] = 0
            weakref.finalize(c, _give_back, B, a, c.view())  # the view shares the memory but does not keep c itself alive
            s.update(call=be.bind_gemm(qtype, M, N, K, a, K, B, N, c, N))
        else:
            ws = torch.empty(max(16, be.gemm_workspace_bytes(qtype, M, N, K)), dtype=torch.uint8, device="cuda")
            s.update(fn=getattr(be, "gemm_" + qtype), args=(M, N, K, A, K, W, N, torch.zeros(M, N, device="cuda"), N, ws))
    elif kind == "moe":
        qtype, H, I, E, top_k = MOE_SHAPES[case["form"]]
        experts = lambda N, K: list(_weight(gen, qtype, E * N, K).chunk(E))  # noqa: E731
        bias = lambda *n: _normal(gen, n, 0.02)  # noqa: E731
        more = {}
        if case["form"] == "gpt_oss":
            more = dict(kind=1, router_bias=bias(E), gate_b=list(bias(E, I)), up_b=list(bias(E, I)),
                        down_b=list(bias(E, H)), alpha=1.702)
        s.update(layer=be.MoeLayer(_normal(gen, (H, E), 0.02), experts(I, H), experts(I, H), experts(H, I), top_k,
                                   qtype=qtype, **more), x=_normal(gen, (case["tokens"], H)))
    elif kind == "attn":
        hq, hkv, hd, rows = case["heads"], case["kv_heads"], case["head_dim"], case["rows"]
        sink = _normal(gen, (hq,)) if case["sink"] else None
        attn = be.Attention(hq, hkv, hd, rows, window=case["window"] or None, sink=sink)
        attn.kcache.copy_(_normal(gen, attn.kcache.shape))
        attn.vcache.copy_(_normal(gen, attn.vcache.shape))
        s.update(attn=attn, pos=rows - 1, q=_normal(gen, (hq * hd,)), k=_normal(gen, (hkv * hd,)),
                 v=_normal(gen, (hkv * hd,)), q_step=torch.empty(hq * hd, device="cuda"), qk_norm=None)
        if case["qk_norm"]:
            s["qk_norm"] = (1 + _normal(gen, (hd,), 0.1), 1 + _normal(gen, (hd,), 0.1), 1e-6)
    else:
        cfg, dec = _decoder(case, gen)
        ids = torch.randint(0, cfg.vocab, (case["context"],), generator=gen, device="cuda").tolist()
        s.update(dec=dec, new=case["new"], prompt=ids)
        if kind == "replay":  # a context of random cache rows stands in for the prompt
            for a in dec.attn:
                a.kcache.copy_(_normal(gen, a.kcache.shape))
                a.vcache.copy_(_normal(gen, a.vcache.shape))
            s.update(graph=dec.capture(case["context"]), pos=torch.tensor([case["context"], 0], dtype=torch.int32, device="cuda"),
                     tok=torch.tensor([float(ids[-1])], device="cuda"),
                     out=torch.zeros(case["new"], dtype=torch.int32, device="cuda"))
    return s


def _give_back(B, a, c):
    """The device copy of a host weight and the page-locked buffers of its calls."""
    be.unregister_weight(B)
    be.host_free(a)
    be.host_free(c)


def run(state):
    kind = state["kind"]
    if kind == "host":
        return state["call"]()
    if kind == "gemm":
        return state["fn"](*state["args"])
    if kind == "moe":
        return state["layer"].forward(state["x"])
    if kind == "attn":
        attn = state["attn"]
        state["q_step"].copy_(state["q"])  # the projection's output: the step may rotate it in place
        out = attn.step(state["q_step"], state["k"], state["v"], state["pos"], qk_norm=state["qk_norm"])
        return {"out": out, "kcache": attn.kcache, "vcache": attn.vcache}
    dec = state["dec"]
    if kind == "replay":
        dec.pos_dev.copy_(state["pos"])
        dec.tok_f.copy_(state["tok"])
        for i in range(state["new"]):
            state["graph"].replay()
            state["out"][i:i + 1].copy_(dec.tok)
        tokens = state["out"]
    else:
        tokens = dec.generate(state["prompt"], state["new"])
    caches = [c for a in dec.attn for c in (a.kcache, a.vcache)]
    return {"tokens": tokens, "logits": dec.b["logits"], "caches": caches}


# ---------------------------------------------------------------------------------------------------- what a pass needs
def work(case):
    kind = case["kind"]
    if kind in ("host", "gemm"):
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": BYTES_PER_WEIGHT[case["qtype"]] * N * K + 4 * M * (K + N), "flops": 2 * M * N * K}
    if kind == "moe":
        qtype, H, I, E, top_k = MOE_SHAPES[case["form"]]
        T = case["tokens"]
        touched = E * (1 - (1 - top_k / E) ** T)  # experts that a batch of near-uniform routing reaches
        return {"bytes": touched * 3 * H * I * BYTES_PER_WEIGHT[qtype] + 4 * H * E + 8 * T * H,
                "flops": 2 * T * (top_k * 3 * H * I + H * E)}
    if kind == "attn":
        rows = min(case["rows"], case["window"] or case["rows"])
        hq, hkv, hd = case["heads"], case["kv_heads"], case["head_dim"]
        return {"bytes": 4 * rows * hkv * hd + 8 * hq * hd + 8 * hkv * hd, "flops": 4 * rows * hq * hd}
    L, ctx, new = case["layers"], case["context"], case["new"]
    layer = 2560 * (6144 + 4096 + 3 * 9728)
    head = case["vocab"] * 2560
    passes = new if kind == "replay" else new + 1  # the prompt's tokens can share one pass over the weights
    rows = sum(range(ctx, ctx + new)) if kind == "replay" else sum(range(1, ctx + new + 1))
    tokens = new if kind == "replay" else ctx + new
    return {"bytes": passes * (L * layer * BYTES_PER_WEIGHT["q4_K"] + head * BYTES_PER_WEIGHT["q6_K"]) + L * rows * 4 * 1024,
            "flops": 2 * tokens * L * layer + 2 * passes * head + L * rows * 4 * 4096}


def tolerance(case):
    kind = case["kind"]
    if kind in ("host", "gemm"):
        # from 32 rows up the operands may be rounded to fp16 (2^-11 each) where the widths suit the fp16 tensor path;
        # everything else is integer sums and a short fp32 chain
        fp16 = case["M"] >= 32 and case["K"] % 64 == 0 and (case["qtype"] == "q6_K" or case["N"] % 256 == 0)
        return {"rel": 1e-3} if fp16 else {"rel": 1e-5}
    if kind == "moe":
        return {"rel": 1e-4}  # the second product's activations are quantized again: an ulp may become a step of 1/127
    if kind == "attn":
        return {"rel": 1e-5}
    return "exact"  # greedy decoding: the token stream, and the logits and caches behind it, are reproducible to the bit
