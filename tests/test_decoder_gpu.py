"""Greedy decoding on the GPU against the CPU pipeline built from the checker (tests/cpu_decoder.py): a 2-layer decoder
with Qwen3-4B's layer dimensions (hidden 2560, 32 query / 8 key-value heads of 128, SwiGLU 9728; vocabulary cut to
32768 rows to keep the CPU side short), Q4_K projections, Q6_K embedding and lm_head, weights loaded from a .bin file.
Every operator is bit-exact against its checker, so the token streams must be IDENTICAL over 64 steps; the test also
logs the smallest top-2 logit margin seen, which says how much room an inexact path would have had."""
import os
import tempfile

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from nntrainer_b200.decoder import DecoderConfig, Qwen3Decoder, tensor_list  # noqa: E402
from oracle import oracle as O  # noqa: E402
from oracle.cpu_decoder import CpuDecoder, synthetic_weights, write_bin  # noqa: E402


@pytest.fixture(scope="module")
def be():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from nntrainer_b200 import backend, build
    build.build()
    backend.init(0)
    return backend


_CPU_RUNS = {}


def _run(be, cfg, prompt, n_new, seed, fuse=True):
    w = synthetic_weights(cfg, seed)
    with tempfile.TemporaryDirectory() as td:
        path = os.path.join(td, "model.bin")
        write_bin(path, cfg, w)
        gpu = Qwen3Decoder(cfg, path, fuse=fuse)
        got = gpu.generate(prompt, n_new)
        be.device_status()
        gpu_logits = gpu.b["logits"].cpu().numpy()
        gpu.close()
    key = (repr(cfg), tuple(prompt), n_new, seed)
    if key in _CPU_RUNS:  # the CPU pipeline of the same model and prompt ran for the other launch sequence already
        want, last_logits, margin = _CPU_RUNS[key]
        return got, want, gpu_logits, last_logits, margin
    cos, sin = be.rope_table(cfg.head_dim, cfg.max_seq, cfg.rope_theta)
    cpu = CpuDecoder(cfg, w, cos, sin, matmul=O.ref(fast=True) if O.ref_available() else None)
    want, pos, margin = [], 0, np.inf
    for t in prompt:
        nxt = cpu.step(t, pos)
        pos += 1
    for _ in range(n_new):
        want.append(nxt)
        top2 = np.partition(cpu.last_logits, -2)[-2:]
        margin = min(margin, float(top2[1] - top2[0]))
        nxt = cpu.step(nxt, pos)
        pos += 1
    _CPU_RUNS[key] = (want, cpu.last_logits, margin)
    return got, want, gpu_logits, cpu.last_logits, margin


@pytest.mark.parametrize("fuse", [True, False], ids=["five_launches_per_layer", "nine_launches_per_layer"])
def test_greedy_token_stream_identical_over_64_steps(be, fuse):
    """Both launch sequences: with the residual adds and norms folded into the projections' prologues, and with every
    operator in a launch of its own."""
    cfg = DecoderConfig(n_layers=2, hidden=2560, n_heads=32, n_kv_heads=8, head_dim=128, inter=9728, vocab=32768,
                        max_seq=80)
    got, want, gl, cl, margin = _run(be, cfg, prompt=[11, 4097, 32767, 5], n_new=64, seed=0, fuse=fuse)
    print(f"smallest top-2 logit margin over 64 steps: {margin:.3e}")
    assert got == want
    assert len(set(got)) > 4, "degenerate stream: the test would not notice a wrong operator"
    assert np.array_equal(gl.view(np.uint32), cl.view(np.uint32)), "final logits differ in the last bits"


def test_sliding_window_shorter_than_the_context(be):
    cfg = DecoderConfig(n_layers=1, hidden=512, n_heads=8, n_kv_heads=2, head_dim=64, inter=768, vocab=1024, max_seq=48,
                        sliding_window=16)
    got, want, gl, cl, _ = _run(be, cfg, prompt=[1, 2, 3], n_new=40, seed=1)
    assert got == want
    assert np.array_equal(gl.view(np.uint32), cl.view(np.uint32))


def test_a_replaced_cache_is_used_by_every_launch_sequence(be):
    """The launches of a step are prepared once per launch sequence: after a layer's caches, rotary tables or an activation
    buffer were replaced, every one of them works on the new tensors."""
    cfg = DecoderConfig(n_layers=2, hidden=512, n_heads=8, n_kv_heads=2, head_dim=64, inter=768, vocab=1024, max_seq=32)
    with tempfile.TemporaryDirectory() as td:
        path = os.path.join(td, "model.bin")
        write_bin(path, cfg, synthetic_weights(cfg, 5))
        dec, other = Qwen3Decoder(cfg, path), Qwen3Decoder(cfg, path)
    tok = torch.tensor([7.0], device="cuda")
    for pdl in (True, False):  # two lists of calls, made for the first tensors
        dec.pdl = pdl
        dec.step(tok, 0)
    old = [(t, t.clone()) for a in dec.attn for t in (a.kcache, a.vcache, a.ws)] + [(dec.b["h"], dec.b["h"].clone())]
    for a in dec.attn:
        for name in ("kcache", "vcache"):
            setattr(a, name, torch.zeros_like(getattr(a, name)))
        for name in ("cos", "sin", "ws"):
            setattr(a, name, getattr(a, name).clone())
    dec.b["h"] = torch.empty_like(dec.b["h"])
    for pos, pdl in enumerate((True, False, True, False)):
        dec.pdl = pdl
        t, tf = dec.step(tok, pos)
        w, _ = other.step(tok, pos)
        assert int(t) == int(w)
        assert torch.equal(dec.b["logits"].view(torch.int32), other.b["logits"].view(torch.int32))
        tok = tf
    be.device_status()
    for a, b in zip(dec.attn, other.attn):
        assert torch.equal(a.kcache, b.kcache) and torch.equal(a.vcache, b.vcache)
    for t, was in old:
        assert torch.equal(t, was), "a launch still used a tensor that was replaced"
    dec.close()
    other.close()


@pytest.mark.parametrize("hq,hkv,hd", [(32, 8, 128), (32, 4, 128), (64, 8, 64)])
def test_a_captured_step_has_the_form_for_its_context_however_long_the_caches_are(be, launches_in, monkeypatch, hq, hkv, hd):
    """Long contexts have an attention launch of their own, slower for short ones: a graph is given it by the positions that
    it is meant for, not by the rows that the caches could hold."""
    make = torch.cuda.CUDAGraph
    monkeypatch.setattr(torch.cuda, "CUDAGraph", lambda: make(keep_graph=True))

    def grids(start, max_seq, tokens=0):
        cfg = DecoderConfig(n_layers=1, hidden=256, n_heads=hq, n_kv_heads=hkv, head_dim=hd, inter=256, vocab=256, max_seq=max_seq)
        with tempfile.TemporaryDirectory() as td:
            path = os.path.join(td, "model.bin")
            write_bin(path, cfg, synthetic_weights(cfg, 3))
            dec = Qwen3Decoder(cfg, path, pdl=True)
        g = dec.capture(start, tokens)
        seen = [x.grid for x in launches_in(g)]
        dec.close()
        return seen

    short, long = grids(100, 128), grids(2000, 2032)
    assert len(short) == len(long) and short != long
    assert grids(100, 4096) == short
    assert grids(2000, 4096) == long
    assert grids(100, 4096, 4000) == long and grids(100, 4096, 100) == short


@pytest.mark.parametrize("window,fc,P,hd", [(None, "q4_K", 2, 64), (None, "q4_K", 9, 64), (16, "q4_K", 40, 64), (None, "q6_K", 33, 64),
                                            (None, "q4_K", 300, 64), (None, "q4_K", 258, 64), (None, "q4_K", 258, 128),
                                            (100, "q4_K", 131, 128), (None, "q4_K", 20, 96), (None, "q4_0", 20, 64)])
def test_batched_prompt_equals_token_by_token(be, window, fc, P, hd):
    """The prompt's batched pass against feeding the prompt through step(): tokens, final logits and both caches of every
    layer, equal bits -- a prompt too short to be batched, ragged tiles of eight rows, a window shorter than the prompt,
    separate q, k and v projections (Q6_K, Q4_0), more tokens than one pass takes, a last pass of one row, and heads of more
    than 64 dimensions, of which a CTA owns all when many tokens are at hand."""
    cfg = DecoderConfig(n_layers=3, hidden=512, n_heads=8, n_kv_heads=2, head_dim=hd, inter=768, vocab=1024, max_seq=P + 8,
                        sliding_window=window, fc_dtype=fc)
    w = synthetic_weights(cfg, 3)
    rng = np.random.default_rng(P)
    w.update({name: O.random_q4_0x8(rng, N, K) for name, d, N, K in tensor_list(cfg) if d == "q4_0"})
    prompt = [int(t) for t in rng.integers(0, cfg.vocab, P)]
    with tempfile.TemporaryDirectory() as td:
        path = os.path.join(td, "model.bin")
        write_bin(path, cfg, w)
        got, want = Qwen3Decoder(cfg, path), Qwen3Decoder(cfg, path)
    tokens = got.generate(prompt, 4)
    ref, tok = [], torch.empty(1, device="cuda")
    for pos in range(P + 4):
        tok.fill_(float(prompt[pos] if pos < P else ref[-1]))
        nxt, _ = want.step(tok, pos)
        if pos >= P - 1 and len(ref) < 4:
            ref.append(int(nxt.item()))
    be.device_status()
    assert tokens == ref
    assert torch.isfinite(want.b["logits"]).all()
    assert torch.equal(got.b["logits"].view(torch.int32), want.b["logits"].view(torch.int32))
    for a, b in zip(got.attn, want.attn):
        assert torch.equal(a.kcache.view(torch.int16), b.kcache.view(torch.int16))
        assert torch.equal(a.vcache.view(torch.int16), b.vcache.view(torch.int16))
    got.close()
    want.close()
