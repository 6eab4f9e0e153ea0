"""Host-side mirror of the reference's Qwen3 decoder graph for greedy decoding, built from the device entry points of
the C ABI only (every tensor stays in HBM between operators; PyTorch provides the buffers and the stream).

Graph (Applications/CausalLM/causal_lm.cpp:174-233 constructModel, :566-612 createTransformerDecoderBlock,
qwen3_causallm.cpp:33-110 createAttention with per-head q/k norms, causal_lm.cpp:671-706 createMlp):

    embedding -> L x [ rms_norm -> wv, wk, k_norm, wq, q_norm -> mha_core -> attention_out -> add
                       -> rms_norm -> ffn_up, ffn_gate -> swiglu(ffn_up, ffn_gate) -> ffn_down -> add ]
              -> rms_norm -> lm_head -> arg-max (causal_lm.cpp:530-533)

The swiglu layer's first input (the one that goes through the sigmoid) is the layer NAMED ffn_up, the second the one
named ffn_gate (createMlp lists the inputs in that order; swiglu.cpp:55). Weights are read from a .bin file in the
order the layers request them (``tensor_list``).
"""
from __future__ import annotations

from dataclasses import dataclass

from . import backend as be


@dataclass
class DecoderConfig:
    n_layers: int
    hidden: int
    n_heads: int
    n_kv_heads: int
    head_dim: int
    inter: int
    vocab: int
    max_seq: int
    rope_theta: float = 1e6
    norm_eps: float = 1e-6
    fc_dtype: str = "q4_K"
    embedding_dtype: str = "q6_K"
    lmhead_dtype: str = "q6_K"
    tie_word_embeddings: bool = False
    sliding_window: int | None = None
    rope_scaling_factor: float | None = None  # rope_scaling_type "yarn" with this factor (None: default rope)
    rope_scaling_max_position_embeddings: int = 4096


def tensor_list(c: DecoderConfig):
    """(name, dtype, N, K) of every weight in file order. Quantized tensors: N rows of K weights (N = output units)."""
    t = [("embedding0", c.embedding_dtype, c.vocab, c.hidden)]
    q_dim, kv_dim = c.n_heads * c.head_dim, c.n_kv_heads * c.head_dim
    for i in range(c.n_layers):
        p = f"layer{i}_"
        t += [(p + "attention_norm", "f32", 1, c.hidden),
              (p + "wv", c.fc_dtype, kv_dim, c.hidden),
              (p + "wk", c.fc_dtype, kv_dim, c.hidden),
              (p + "k_norm", "f32", 1, c.head_dim),
              (p + "wq", c.fc_dtype, q_dim, c.hidden),
              (p + "q_norm", "f32", 1, c.head_dim),
              (p + "attention_out", c.fc_dtype, c.hidden, q_dim),
              (p + "ffn_norm", "f32", 1, c.hidden),
              (p + "ffn_up", c.fc_dtype, c.inter, c.hidden),
              (p + "ffn_gate", c.fc_dtype, c.inter, c.hidden),
              (p + "ffn_down", c.fc_dtype, c.hidden, c.inter)]
    t.append(("output_norm", "f32", 1, c.hidden))
    if not c.tie_word_embeddings:
        t.append(("output_of_causallm", c.lmhead_dtype, c.vocab, c.hidden))
    return t


class Qwen3Decoder:
    """Greedy decoding of a Qwen3-shaped dense decoder from a .bin file, batch 1, one token per step."""

    def __init__(self, cfg: DecoderConfig, bin_path: str, device: str = "cuda", pdl: bool = False, fuse: bool = True):
        import torch
        self.torch, self.cfg, self.dev = torch, cfg, device
        self.fuse = fuse  # fold the residual adds and RMS norms into the prologues of the projections behind them
        self.tensors = tensor_list(cfg)
        self.w = be.BinWeights(bin_path, [(d, n, k) for _, d, n, k in self.tensors])
        self.ptr = {name: self.w.ptr[i] for i, (name, *_r) in enumerate(self.tensors)}
        self._shape = {name: (d, n, k) for name, d, n, k in self.tensors}
        self.pdl = pdl
        cos, sin = be.rope_table(cfg.head_dim, cfg.max_seq, cfg.rope_theta, yarn_factor=cfg.rope_scaling_factor,
                                 yarn_original_max_position_embeddings=cfg.rope_scaling_max_position_embeddings)
        tabs = (torch.from_numpy(cos).to(device), torch.from_numpy(sin).to(device))
        self.attn = [be.Attention(cfg.n_heads, cfg.n_kv_heads, cfg.head_dim, cfg.max_seq, window=cfg.sliding_window,
                                  device=device, tables=tabs) for _ in range(cfg.n_layers)]
        f = lambda n: torch.empty(n, dtype=torch.float32, device=device)
        q_dim, kv_dim = cfg.n_heads * cfg.head_dim, cfg.n_kv_heads * cfg.head_dim
        qkv, ug = f(q_dim + 2 * kv_dim), f(2 * cfg.inter)  # q | k | v and ffn_up | ffn_gate, each from one launch
        self.b = dict(x=f(cfg.hidden), h=f(cfg.hidden), n=f(cfg.hidden), qkv=qkv, q=qkv[:q_dim],
                      k=qkv[q_dim:q_dim + kv_dim], v=qkv[q_dim + kv_dim:], a=f(q_dim), o=f(cfg.hidden), ug=ug,
                      up=ug[:cfg.inter], gate=ug[cfg.inter:], act=f(cfg.inter), d=f(cfg.hidden), logits=f(cfg.vocab))
        self._tables()
        import ctypes as C
        self._calls, self._addressof = {}, C.addressof
        self._arg = dict(tok=C.c_void_p(), pos=C.c_uint(), pos_dev=C.c_void_p(), idx=C.c_void_p(), idx_f=C.c_void_p(),
                         stream=C.c_void_p())

    class _P:  # a raw device address with the data_ptr() face the backend helpers use
        def __init__(self, p):
            self.p = p

        def data_ptr(self):
            return self.p

    def _norm(self, x, name, out, width=None):
        be.rms_norm(x, self._P(self.ptr[name]), self.cfg.norm_eps, width=width, out=out, pdl=self.pdl)

    def _tables(self):
        """Device tables of weight addresses for the batched launches: per layer the q, k and v projections as row
        slices of equal height (one launch computes q | k | v into one buffer), and ffn_up | ffn_gate."""
        torch, c = self.torch, self.cfg
        kv_dim, q_dim = c.n_kv_heads * c.head_dim, c.n_heads * c.head_dim
        self._qkv_ok = c.fc_dtype == "q4_K" and q_dim % kv_dim == 0 and kv_dim % 8 == 0
        self._qkv_tab, self._ug_tab = [], []
        row_bytes = c.hidden // 256 * 144
        for i in range(c.n_layers):
            p = f"layer{i}_"
            if self._qkv_ok:
                ptrs = [self.ptr[p + "wq"] + j * kv_dim * row_bytes for j in range(q_dim // kv_dim)]
                ptrs += [self.ptr[p + "wk"], self.ptr[p + "wv"]]
                self._qkv_tab.append(torch.tensor(ptrs, dtype=torch.int64, device=self.dev))
                self._ug_tab.append(torch.tensor([self.ptr[p + "ffn_up"], self.ptr[p + "ffn_gate"]], dtype=torch.int64,
                                                 device=self.dev))
        # With ``fuse`` the q, k and v projections run as ONE 6144-row problem (its per-SM share fits in shared memory, so
        # it takes the resident-weights kernel): the file stores wv, wk, k_norm, wq, so the three tensors are packed
        # once into q | k | v order (8.8 MB per layer beside the loaded copy).
        self._qkv_packed = []
        if self.fuse and self._qkv_ok:
            for i in range(c.n_layers):
                p = f"layer{i}_"
                packed = torch.empty((q_dim + 2 * kv_dim) * row_bytes, dtype=torch.uint8, device=self.dev)
                off = 0
                for name, rows in ((p + "wq", q_dim), (p + "wk", kv_dim), (p + "wv", kv_dim)):
                    be.check(be.lib().nntr_cuda_memcpy(packed.data_ptr() + off, self.ptr[name], rows * row_bytes, 3))
                    off += rows * row_bytes
                self._qkv_packed.append(packed)

    def step(self, token_f, pos: int, pos_dev=None, out_idx=None, out_idx_f=None):
        """One decode step: ``token_f`` is a 1-element float device tensor holding the token id (the reference keeps
        ids as floats); returns (next id as int32 tensor, as float32 tensor). Logits stay in ``self.b['logits']``.
        With ``pos_dev`` (a device word) the position is read on the device, so the launches can be captured once into
        a CUDA graph and replayed for every later token; ``pos`` is then where the positions start, which chooses the form of the
        attention launch (same bits in both).

        Launches per layer without ``fuse``: (residual add +) RMS norm; q | k | v projections (one batched launch);
        attention with its per-head norms, rotary work and cache append; attention_out; residual add + RMS norm;
        ffn_up | ffn_gate (one batched launch); SwiGLU; ffn_down -- nine. With ``fuse`` the two norms run in the
        prologues of the projections behind them and the SwiGLU in the epilogue of the up | gate launch -- five (attention
        takes more launches beyond 16384 rows). Every fusion keeps the bits of the separate operators."""
        torch = self.torch
        if out_idx is None:
            out_idx = torch.empty(1, dtype=torch.int32, device=self.dev)
        if out_idx_f is None:
            out_idx_f = torch.empty(1, dtype=torch.float32, device=self.dev)
        # The launches of a step differ from the next step's in five values only: they are made into a list of calls once, whose
        # arguments are converted already and share those five. A call then costs its launch and little else. A list is made
        # again when an address in it is no longer that of the tensor it was taken from.
        key, held = (self.pdl, self.fuse), self._held()
        made_for, calls = self._calls.get(key, (None, None))
        if made_for != held:
            calls = self._make_calls()
            self._calls[key] = held, calls
        v = self._arg
        v["tok"].value, v["pos"].value = token_f.data_ptr(), pos
        v["pos_dev"].value = pos_dev.data_ptr() if pos_dev is not None else None
        v["idx"].value, v["idx_f"].value = out_idx.data_ptr(), out_idx_f.data_ptr()
        v["stream"].value = be._stream()
        for fn, args in calls:
            rc = fn(*args)
            if rc:
                be.check(rc)
        return out_idx, out_idx_f

    def _held(self):
        """The addresses (and the sizes beside them) that a list of calls holds, as they are now."""
        held = [t.data_ptr() for ts in (self.b.values(), self._qkv_packed, self._qkv_tab, self._ug_tab) for t in ts]
        held += self.ptr.values()
        for a in self.attn:
            held += (self._addressof(a.desc), a.max_seq, a.kcache.data_ptr(), a.vcache.data_ptr(), a.cos.data_ptr(),
                     a.sin.data_ptr(), a.ws.data_ptr(), a.ws.numel())
        return held

    def _make_calls(self):
        """The C calls of a decode step in order, as (function, converted arguments)."""
        import ctypes as C
        from .capi import GEMV_PDL, QTYPE
        c, b, L, v = self.cfg, self.b, be.lib(), self._arg
        flags = GEMV_PDL if self.pdl else 0
        q_dim, kv_dim = c.n_heads * c.head_dim, c.n_kv_heads * c.head_dim
        calls = []

        def call(name, *args):
            fn = getattr(L, "nntr_cuda_" + name)
            conv = [a if isinstance(a, (C._SimpleCData, C.Structure)) or type(a).__name__ == "CArgObject" else
                    t(a.data_ptr()) if hasattr(a, "data_ptr") else t(a) for t, a in zip(fn.argtypes, args)]
            calls.append((fn, tuple(conv)))

        w = lambda name: self._P(self.ptr[name])  # noqa: E731
        st, eps = v["stream"], c.norm_eps

        def gemv(name, x, y):
            dtype, N, K = self._shape[name]
            call("gemv_dev", QTYPE[dtype], N, K, x, w(name), y, flags, st)

        def norm(x, name, out):
            call("rms_norm_dev", x, w(name), out, 1, c.hidden, eps, flags, st)

        def add_norm(x, r, name, total, out):
            call("add_rms_norm_dev", x, r, total, w(name), out, 1, c.hidden, eps, flags, st)

        call("embedding_dev", QTYPE[c.embedding_dtype], w("embedding0"), v["tok"], b["x"], 1, c.vocab, c.hidden, flags, st)
        x = b["x"]
        fuse, qt = self.fuse and self._qkv_ok, QTYPE[c.fc_dtype]
        for i in range(c.n_layers):
            p = f"layer{i}_"
            at = self.attn[i]

            def attention():
                call("attention_step_dev", C.byref(at.desc), v["pos"], v["pos_dev"], at.max_seq, b["q"], b["k"], b["v"],
                     w(p + "q_norm"), w(p + "k_norm"), eps, at.kcache, at.vcache, at.cos, at.sin, None, b["a"], at.ws,
                     at.ws.numel(), flags, st)

            if fuse:
                # 5 launches: (add +) norm + q|k|v; attention; o; add + norm + up|gate + SwiGLU; down
                # (behind the first layer: the previous block's output x = h + ffn_down, and its norm)
                src = (x, None, None) if i == 0 else (b["h"], b["d"], x)
                call("gemv_add_norm_dev", qt, q_dim + 2 * kv_dim, c.hidden, *src, w(p + "attention_norm"), eps,
                     self._qkv_packed[i], b["qkv"], flags, st)
                attention()
                gemv(p + "attention_out", b["a"], b["o"])
                call("gated_ffn_in_dev", qt, c.inter, c.hidden, x, b["o"], b["h"], w(p + "ffn_norm"), eps, w(p + "ffn_up"),
                     w(p + "ffn_gate"), b["act"], flags, st)
                gemv(p + "ffn_down", b["act"], b["d"])
                continue
            if i == 0:
                norm(x, p + "attention_norm", b["n"])
            else:  # the previous block's output x = h + ffn_down, and its norm
                add_norm(b["h"], b["d"], p + "attention_norm", x, b["n"])
            if self._qkv_ok:
                call("gemv_batched_dev", qt, kv_dim, c.hidden, b["n"], self._qkv_tab[i], q_dim // kv_dim + 2, b["qkv"], flags,
                     st)
            else:
                gemv(p + "wv", b["n"], b["v"])
                gemv(p + "wk", b["n"], b["k"])
                gemv(p + "wq", b["n"], b["q"])
            attention()  # with k_norm and q_norm (per-head RMS norms)
            gemv(p + "attention_out", b["a"], b["o"])
            add_norm(x, b["o"], p + "ffn_norm", b["h"], b["n"])
            if self._qkv_ok:
                call("gemv_batched_dev", qt, c.inter, c.hidden, b["n"], self._ug_tab[i], 2, b["ug"], flags, st)
            else:
                gemv(p + "ffn_up", b["n"], b["up"])
                gemv(p + "ffn_gate", b["n"], b["gate"])
            call("swiglu_dev", b["act"], b["up"], b["gate"], c.inter, flags, st)
            gemv(p + "ffn_down", b["act"], b["d"])
        add_norm(b["h"], b["d"], "output_norm", x, b["n"])
        gemv("embedding0" if c.tie_word_embeddings else "output_of_causallm", b["n"], b["logits"])
        call("argmax_dev", b["logits"], 1, c.vocab, c.vocab, v["idx"], v["idx_f"], flags, st)
        return calls

    def capture(self, start_pos: int, tokens: int = 0):
        """Captures one decode step into a CUDA graph: the token id lives in ``self.tok_f`` (device float, rewritten by
        the step's own arg-max), the position in ``self.pos_dev`` (device word, advanced by the graph). Returns the
        graph; every ``replay()`` decodes one more token and leaves its id in ``self.tok`` / ``self.tok_f``. ``tokens``: how
        many it is meant for, if that is known; the attention launches take the form for the middle of its positions, and any
        position up to ``max_seq`` may be replayed."""
        torch = self.torch
        likely_pos = int(start_pos) + int(tokens) // 2
        self.pos_dev = torch.full((2,), 0, dtype=torch.int32, device=self.dev)  # 8 bytes: the bump kernel adds to a u64
        self.pos_dev[0] = start_pos
        self.tok = torch.zeros(1, dtype=torch.int32, device=self.dev)
        self.tok_f = torch.zeros(1, dtype=torch.float32, device=self.dev)
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            self.step(self.tok_f, likely_pos, pos_dev=self.pos_dev, out_idx=self.tok, out_idx_f=self.tok_f)  # warm-up, eager
            self.pos_dev[0] = start_pos
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                self.step(self.tok_f, likely_pos, pos_dev=self.pos_dev, out_idx=self.tok, out_idx_f=self.tok_f)
                be.check(be.lib().nntr_cuda_epoch_bump_dev(self.pos_dev.data_ptr(), be._stream()))
        torch.cuda.current_stream().wait_stream(s)
        return g

    # Prompt tokens per batched pass: enough rows for the matrix kernels to read every weight once or a few times, few enough
    # for buffers of a few tens of megabytes.
    PROMPT_ROWS = 256

    def _prompt(self, ids, pos: int):
        """Fills the caches with the rows of the tokens ``ids`` from position ``pos`` on, all of them through each layer
        together. Every row runs the decode kernels' float chains (gemv_rows, Attention.rows, row norms), so the caches equal
        those of decoding the tokens one by one bit for bit. The last layer needs its keys and values only."""
        torch, c, pdl = self.torch, self.cfg, self.pdl
        T, q_dim, kv_dim = len(ids), c.n_heads * c.head_dim, c.n_kv_heads * c.head_dim
        ld = q_dim + 2 * kv_dim
        f = lambda n: torch.empty((T, n), dtype=torch.float32, device=self.dev)  # noqa: E731
        x, h, n, qkv, a, o, d = (f(k) for k in (c.hidden, c.hidden, c.hidden, ld, q_dim, c.hidden, c.hidden))
        up, gate = f(c.inter), f(c.inter)
        need = max(be.gemm_workspace_bytes(c.fc_dtype, T, N, K) for N, K in (
            (ld, c.hidden), (q_dim, c.hidden), (kv_dim, c.hidden), (c.hidden, q_dim), (c.inter, c.hidden), (c.hidden, c.inter)))
        ws = torch.empty(max(need, 16), dtype=torch.uint8, device=self.dev)
        be.embedding(c.embedding_dtype, self._P(self.ptr["embedding0"]),
                     torch.tensor([float(t) for t in ids], dtype=torch.float32).to(self.dev), c.vocab, c.hidden, out=x, pdl=pdl)

        def rows(name, src, dst, ldc):
            dtype, N, K = self._shape[name]
            be.gemv_rows(dtype, T, N, K, src, self._P(self.ptr[name]), dst, ldc, ws)

        q, k, v = qkv, qkv[:, q_dim:], qkv[:, q_dim + kv_dim:]
        for i in range(c.n_layers):
            p = f"layer{i}_"
            qk_norm = (self._P(self.ptr[p + "q_norm"]), self._P(self.ptr[p + "k_norm"]), c.norm_eps)
            if i == 0:
                self._norm(x, p + "attention_norm", n)
            else:
                be.add_rms_norm(h, d, self._P(self.ptr[p + "attention_norm"]), c.norm_eps, sum_out=x, out=n, pdl=pdl)
            if self._qkv_packed:
                be.gemv_rows(c.fc_dtype, T, ld, c.hidden, n, self._qkv_packed[i], qkv, ld, ws)
            else:
                rows(p + "wq", n, q, ld)
                rows(p + "wk", n, k, ld)
                rows(p + "wv", n, v, ld)
            self.attn[i].rows(q, k, v, ld, pos, T, a, q_dim, qk_norm=qk_norm, pdl=pdl)
            if i + 1 == c.n_layers:
                return
            rows(p + "attention_out", a, o, c.hidden)
            be.add_rms_norm(x, o, self._P(self.ptr[p + "ffn_norm"]), c.norm_eps, sum_out=h, out=n, pdl=pdl)
            rows(p + "ffn_up", n, up, c.inter)
            rows(p + "ffn_gate", n, gate, c.inter)
            be.swiglu(up, gate, out=up, pdl=pdl)
            rows(p + "ffn_down", up, d, c.hidden)

    def generate(self, prompt_ids, n_new: int):
        """Feeds the prompt, then ``n_new`` greedy tokens; returns them as a Python list. All of the prompt but its last token
        goes through the layers in batched passes (where their kernels apply: heads of up to 128 dimensions, hidden rows of
        up to 11264, up to 16384 positions), with the results of feeding it token by token; the token ids stay on the device until
        the end. An empty prompt and one of more than ``max_seq`` tokens are ValueErrors; no new tokens (0 or
        less) only feed the prompt."""
        torch, c = self.torch, self.cfg
        prompt_ids = list(prompt_ids)
        if not prompt_ids and n_new > 0:
            raise ValueError("generate: an empty prompt leaves nothing to continue")
        if len(prompt_ids) > c.max_seq:  # nothing is fed then
            raise ValueError(f"a prompt of {len(prompt_ids)} tokens does not fit the {c.max_seq} rows of the caches")
        tok = torch.empty(1, dtype=torch.float32, device=self.dev)
        n_new = max(n_new, 0)
        out = torch.empty(n_new + 1, dtype=torch.int32, device=self.dev)
        pos = 0
        if len(prompt_ids) > 3 and c.head_dim <= 128 and c.hidden <= 11264 and c.max_seq <= 16384:
            while pos < len(prompt_ids) - 1:
                n = min(self.PROMPT_ROWS, len(prompt_ids) - 1 - pos)
                self._prompt(prompt_ids[pos:pos + n], pos)
                pos += n
        for t in prompt_ids[pos:]:
            tok.fill_(float(t))
            self.step(tok, pos, out_idx=out[:1], out_idx_f=tok)
            pos += 1
        for i in range(n_new):
            self.step(tok, pos, out_idx=out[i + 1:i + 2], out_idx_f=tok)
            pos += 1
        return out[:n_new].tolist()

    def close(self):
        self.w.close()
