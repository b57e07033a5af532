"""Greedy decode through the quantized model with the per-token work captured as one CUDA graph.

The reference decodes with HF `generate` (generate.py:150-190): every token is a fresh Python walk over the model,
about 230 kernel-launching calls for a 7B Llama, and the GPU waits for the host (decode-sized A16W4 GEMMs run ~10 us
each).  Here the decode step — embedding, all layers with the one-launch decode GEMM (lq_gemv.cu), KV-cache update,
logits, argmax — is captured once on a static KV cache and replayed per token; the token and position live in
device buffers that the captured step itself advances, so a replay needs no host work at all.
"""
from __future__ import annotations

import functools
import os

import torch
from torch.nn.attention import SDPBackend, sdpa_kernel

# the cuDNN attention backend rebuilds its plan for every new KV length (milliseconds of host time per layer and token)
_SDPA = [SDPBackend.FLASH_ATTENTION, SDPBackend.EFFICIENT_ATTENTION, SDPBackend.MATH]

_PROJECTIONS = (("self_attn", ("q_proj", "k_proj", "v_proj")), ("mlp", ("gate_proj", "up_proj")), ("self_attn", ("o_proj",)), ("mlp", ("down_proj",)))


@functools.cache
def _classes():
    """What a prompt's route is decided by (looked up once: an import statement in a function costs microseconds in every call)."""
    from torch.nn.modules import module as nn_module
    from transformers.activations import ACT2FN
    from transformers.models.llama import modeling_llama as hf
    from .quant import QLinearA16W4
    return hf, type(ACT2FN["silu"]), QLinearA16W4, (nn_module._global_forward_hooks, nn_module._global_forward_pre_hooks)


def _words(t):
    """A flat tensor in 8-byte words where it consists of them (copies of many tensors in one launch move one element per thread at a time)."""
    whole = t.numel() * t.element_size() % 8 == 0 and t.storage_offset() * t.element_size() % 8 == 0 and t.data_ptr() % 8 == 0
    return t.view(torch.int64) if whole else t


class GraphedGreedyDecoder:
    """`decoder = GraphedGreedyDecoder(model, batch, max_len)`; `tokens = decoder.generate(prompt, max_new_tokens)`.

    `prompt` is a LongTensor [batch, P] on the model's device with P + max_new_tokens <= max_len.  The first call
    captures the decode step; later calls (any prompt of the same batch size) only replay it."""

    def __init__(self, model, batch: int, max_len: int):
        from transformers import StaticCache
        self.model, self.batch, self.max_len = model, batch, max_len
        self.device = next(model.parameters()).device
        self.cache = StaticCache(config=model.config, max_cache_len=max_len)
        self.tok = torch.zeros((batch, 1), dtype=torch.long, device=self.device)
        self.pos = torch.zeros((1,), dtype=torch.long, device=self.device)
        self.graph = None

    def _step(self):
        from . import ops
        with ops.decode_chain():          # the decode-sized GEMMs may fetch their (constant) weights while their predecessor runs
            out = self.model(input_ids=self.tok, past_key_values=self.cache, cache_position=self.pos, use_cache=True)
        self.tok.copy_(out.logits[:, -1:].argmax(-1))
        self.pos.add_(1)

    @torch.no_grad()
    def _capture(self, tok, pos):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):                       # warm-up: lazy initialisations must not be captured
            self.tok.copy_(tok); self.pos.fill_(pos)
            self._step(); self._step()
        torch.cuda.current_stream().wait_stream(side)
        self.graph = torch.cuda.CUDAGraph()
        self.tok.copy_(tok); self.pos.fill_(pos)
        with torch.cuda.graph(self.graph):
            self._step()
        # cache rows written during warm-up and capture lie at positions >= pos: they are masked until overwritten

    @torch.no_grad()
    def generate(self, prompt: torch.Tensor, max_new_tokens: int, use_graph: bool = True) -> torch.Tensor:
        b, p = prompt.shape
        if b != self.batch or p + max_new_tokens > self.max_len:
            raise ValueError("prompt does not fit the decoder's batch size / cache length")
        self.model.eval()
        with sdpa_kernel(_SDPA):
            if use_graph and self.graph is None:
                # capture on a throw-away prefill: warm-up and capture advance whatever bookkeeping the cache keeps
                # besides its K/V tensors, so the real decode below starts again from a reset cache
                self.cache.reset()
                out = self.model(input_ids=prompt, past_key_values=self.cache,
                                 cache_position=torch.arange(p, device=self.device), use_cache=True)
                self._capture(out.logits[:, -1:].argmax(-1), p)
            self.cache.reset()
            out = self.model(input_ids=prompt, past_key_values=self.cache,
                             cache_position=torch.arange(p, device=self.device), use_cache=True)
            first = out.logits[:, -1:].argmax(-1)
            self.tok.copy_(first); self.pos.fill_(p)
            toks = [first.clone()]
            for _ in range(max_new_tokens - 1):
                if use_graph:
                    self.graph.replay()
                else:
                    self._step()
                toks.append(self.tok.clone())
        return torch.cat(toks, dim=1)


class FusedLlamaGreedyDecoder:
    """Greedy decode of a Llama-architecture model (RMSNorm / RoPE / SwiGLU, no biases) whose decoder linears are
    `QLinearA16W4`, with the decode step written as a chain of this library's kernels instead of the eager modules:

        per layer   residual add + RMSNorm -> fused q|k|v projection (one launch, N = (Hq + 2 Hkv) hd) -> RoPE on q, k
                    with k, v written into the KV cache -> single-query attention over the cache -> o projection ->
                    residual add + RMSNorm -> fused gate|up projection (N = 2 I) -> silu(gate) * up -> down projection
        then        residual add + final RMSNorm -> lm_head -> argmax -> embedding of the new token

    five launches per layer for one or two sequences at hidden size 4096 (both norms, RoPE with the cache write and silu * up inside the
    projections' launches), seven up to 16 sequences, nine otherwise (the reference's fusion list: PTQ/quant/fused_attn.py:164-204 fused QKV, :8-58 RoPE,
    PTQ/quant/fused_mlp.py:84-168 gate/up with the silu epilogue, PTQ/quant/triton_norm.py:7-39 RMSNorm), captured
    once as a CUDA graph and replayed per token.  The prompt goes through the same kernels at its own token count (fused
    q|k|v and gate|up GEMMs, SDPA for its attention) into the same static KV cache, and only its last tokens through the
    head; a model whose modules do anything else, or are watched by hooks, runs its prompt through them
    (`_kernels_serve_prompts`).  `hf_rounding=True` rounds the steps' intermediates like the eager modules' bf16 tensor ops; a prompt
    is always rounded so, whichever way it goes.

    The weights are the model's at the start of each `generate` call: the fused projections are copies, which every call brings
    up to date (75 MB read and written for a layer of 4096 x 11008)."""

    def __init__(self, model, batch: int, max_len: int, hf_rounding: bool = True):
        from transformers import StaticCache
        cfg = model.config
        self.model, self.batch, self.max_len, self.hf = model, batch, max_len, hf_rounding
        self.device = dev = next(model.parameters()).device
        self.Hq, self.Hkv = cfg.num_attention_heads, getattr(cfg, "num_key_value_heads", None) or cfg.num_attention_heads
        self.hd = getattr(cfg, "head_dim", None) or cfg.hidden_size // cfg.num_attention_heads
        self.D, self.I, self.eps = cfg.hidden_size, cfg.intermediate_size, cfg.rms_norm_eps
        self.inv_freq = model.model.rotary_emb.inv_freq.detach().to(dev, torch.float32, copy=True).contiguous()
        self.cache = StaticCache(config=cfg, max_cache_len=max_len)

        self.layers = []
        for layer in model.model.layers:
            now = self._tensors(layer)
            if now is None:
                raise TypeError("FusedLlamaGreedyDecoder needs bias-free QLinearA16W4 projections")
            L = self._flat(now)
            rows = []
            for name, i, j in (("qkv", 0, 9), ("gu", 9, 15)):
                parts = [L["src"][n:j:3] for n in range(i, i + 3)]                # codes, scales, zeros of the projections
                L[name] = tuple(torch.cat(p) for p in parts)
                rows += [r for of in zip(*(t.split([x.numel() for x in p]) for t, p in zip(L[name], parts))) for r in of]
            L["rows"] = [_words(r) for r in rows]
            self.layers.append(L)
        self.ends = self._live_ends()
        bf = dict(dtype=torch.bfloat16, device=dev)
        self.h = torch.zeros((batch, self.D), **bf)
        self.xn = torch.zeros((batch, self.D), **bf)
        self.qkv = torch.zeros((batch, (self.Hq + 2 * self.Hkv) * self.hd), **bf)
        self.att = torch.zeros((batch, self.Hq * self.hd), **bf)
        self.tmp = torch.zeros((batch, self.D), **bf)
        self.h2 = torch.zeros((batch, self.D), **bf)
        self.fuse_norm = batch <= 2 and not os.environ.get("LQ_DECODE_NO_FUSED_NORM")
        self.fuse_rope = batch <= 16 and not os.environ.get("LQ_DECODE_NO_FUSED_ROPE")
        self.gu = torch.zeros((batch, 2 * self.I), **bf)
        self.act = torch.zeros((batch, self.I), **bf)
        self.tok = torch.zeros((batch,), dtype=torch.long, device=dev)
        self.pos = torch.zeros((batch,), dtype=torch.long, device=dev)
        self.logits = None
        self.graph = None
        self.prompt_kernels = self._kernels_serve_prompts()

    @staticmethod
    def _tensors(layer):
        """Codes, scales and zeros of q, k, v, gate, up, o, down and the weights of the two norms, where the model has them now; None unless
        all seven projections are bias-free int4 linears."""
        QLinearA16W4 = _classes()[2]
        sub, out = layer._modules, []                     # (a module's __getattr__ costs several times as much, in every call)
        for part, names in _PROJECTIONS:
            own = sub[part]._modules
            for name in names:
                lin = own[name]
                if not isinstance(lin, QLinearA16W4) or lin._parameters.get("bias") is not None:
                    return None
                w = lin.weight
                scales, zeros, _ = w.qparam
                out += (w.data, scales, zeros)
        return out + [sub["input_layernorm"].weight, sub["post_attention_layernorm"].weight]

    @staticmethod
    def _flat(now):
        src = [t.detach().reshape(-1) for t in now]
        return dict(src=src, words=[_words(t) for t in src[:15]], at=[t.data_ptr() for t in src], sizes=[t.numel() for t in src],
                    o=tuple(src[15:18]), down=tuple(src[18:21]), ln1=src[21], ln2=src[22])

    def _live_ends(self):
        m = self.model
        return m.model.norm.weight.detach(), m.lm_head.weight.detach(), m.model.embed_tokens.weight.detach()

    @torch.no_grad()
    def _take_weights(self):
        """The weights as they are now, for the steps and for a prompt through the kernels: the rows of the fused projections are copied
        anew, in place, where the captured step reads them; a weight that it reads in the model and that has moved since drops it.  (No version or
        address shows that the library's optimizer wrote a weight in place.)  Layers whose projections were replaced by something else stay."""
        to, frm, moved, T = [], [], False, torch.Tensor

        def same(now, at, sizes):                         # (what lay there is held: no other tensor has its address)
            return list(map(T.data_ptr, now)) == at and list(map(T.numel, now)) == sizes and all(map(T.is_contiguous, now))

        for L, layer in zip(self.layers, self.model.model.layers):
            now = self._tensors(layer)
            if now is None:
                continue
            if not same(now, L["at"], L["sizes"]):
                if any(t.numel() != h.numel() or t.dtype != h.dtype for t, h in zip(now, L["src"])):
                    continue
                moved |= not same(now[15:], L["at"][15:], L["sizes"][15:])
                L.update(self._flat(now))
            to += L["rows"]; frm += L["words"]
        ends = self._live_ends()
        if any(t.data_ptr() != h.data_ptr() or t.shape != h.shape or t.stride() != h.stride() for t, h in zip(ends, self.ends)):
            moved, self.ends = True, ends
        if to and {t.dtype for t in to + frm} == {torch.int64}:
            torch._foreach_copy_(to, frm)                 # two layers of 4096 x 11008: 53 us, 168 in bytes and bf16, 149 as copies one by one
        else:
            for d, t in zip(to, frm):
                d.view(torch.uint8).copy_(t.view(torch.uint8))
        if moved:
            self.graph = None

    def _kernels_serve_prompts(self) -> bool:
        """What the step's kernels compute is what the modules compute for a prompt, to rounding, and nothing watches the modules: the
        Llama classes themselves with their forwards untouched, torch's attention, silu, bf16, no autocast, frequencies that do not depend
        on the length of a prompt and need no scaling of the attention, keys kept for the whole length."""
        hf, silu, QLinearA16W4, global_hooks = _classes()

        def own(mod, cls):                                # of the class itself, its forward neither replaced nor watched
            d = mod.__dict__
            return type(mod) is cls and not (d["_forward_hooks"] or d["_forward_pre_hooks"] or "forward" in d)

        def norm(mod):
            return own(mod, hf.LlamaRMSNorm) and mod.variance_epsilon == self.eps and mod.weight.dtype == bf

        bf, scaling = torch.bfloat16, self.hd ** -0.5
        model = self.model
        if not own(model, hf.LlamaForCausalLM) or not own(model.model, hf.LlamaModel):
            return False
        cfg, inner = model.config, model.model
        rope, emb, head = inner.rotary_emb, inner.embed_tokens, model.lm_head
        for layer in inner.layers:
            sub = layer._modules
            if not (own(layer, hf.LlamaDecoderLayer) and own(sub["self_attn"], hf.LlamaAttention) and own(sub["mlp"], hf.LlamaMLP) and sub["self_attn"].scaling == scaling
                    and own(sub["mlp"]._modules["act_fn"], silu) and norm(sub["input_layernorm"]) and norm(sub["post_attention_layernorm"])
                    and all(own(sub[part]._modules[name], QLinearA16W4) for part, names in _PROJECTIONS for name in names)):
                return False
        if any(global_hooks) or torch.is_autocast_enabled(self.device.type):
            return False
        return (own(emb, torch.nn.Embedding) and own(rope, hf.LlamaRotaryEmbedding) and own(head, torch.nn.Linear) and norm(inner.norm)
                and len(inner.layers) == cfg.num_hidden_layers == len(self.layers) and cfg._attn_implementation == "sdpa"
                and rope.rope_type in ("default", "linear", "llama3") and rope.attention_scaling == 1.0
                and rope.inv_freq.shape == self.inv_freq.shape and not any(l.is_sliding for l in self.cache.layers)
                and self.hd % 4 == 0 and 8 <= self.hd <= 512
                and emb.weight.dtype == bf and emb.max_norm is None and head.weight.dtype == bf and head.bias is None)

    def _step(self):
        from . import ops
        with ops.decode_chain():          # launches may start while their predecessor runs (weights are constant here)
            self._step_kernels(ops)

    def _qkv(self, ops, L, h, h_alt, delta, kc, vc) -> bool:
        """Residual add + RMSNorm + q|k|v projection + RoPE + cache write of one layer in as few launches as the batch
        allows: one (one or two sequences at hidden size 4096), two (up to 16 sequences: RoPE and the cache write are
        the projection's epilogue) or three.  True when the residual stream now lives in `h_alt`."""
        Hq, Hkv, hd, D = self.Hq, self.Hkv, self.hd, self.D
        N = (Hq + 2 * Hkv) * hd
        rope = (self.pos, self.inv_freq, kc, vc, Hq, Hkv, hd, D)
        kw = dict(out=self.qkv, hf_rounding=self.hf)
        norm = (h, delta, L["ln1"], self.eps, h_alt)
        if self.fuse_norm and self.fuse_rope and ops.gemm_a16w4_fwd_qkv_rope(None, *L["qkv"], *rope, norm=norm, **kw) is not None:
            return delta is not None
        if self.fuse_norm and ops.gemm_a16w4_fwd_rmsnorm(*norm, *L["qkv"], N, D, **kw) is not None:
            ops.rope_kv_store(self.qkv, self.pos, self.inv_freq, kc, vc, Hq, Hkv, hd, hf_rounding=self.hf)
            return delta is not None
        ops.add_rmsnorm(h, delta, L["ln1"], self.eps, out=self.xn, hf_rounding=self.hf)
        if not (self.fuse_rope and ops.gemm_a16w4_fwd_qkv_rope(self.xn, *L["qkv"], *rope, **kw) is not None):
            ops.gemm_a16w4_fwd(self.xn, *L["qkv"], None, N, D, out=self.qkv)
            ops.rope_kv_store(self.qkv, self.pos, self.inv_freq, kc, vc, Hq, Hkv, hd, hf_rounding=self.hf)
        return False

    def _step_kernels(self, ops):
        D, I, Hq, Hkv, hd = self.D, self.I, self.Hq, self.Hkv, self.hd
        delta = None                        # self.h holds the embedding row of self.tok (written by the previous step's end)
        h, h_alt = self.h, self.h2          # the residual stream alternates between two buffers where the norm is fused
        for li, L in enumerate(self.layers):
            kc, vc = self.cache.layers[li].keys, self.cache.layers[li].values
            if self._qkv(ops, L, h, h_alt, delta, kc, vc):
                h, h_alt = h_alt, h
            ops.decode_attention(self.qkv, self.pos, kc, vc, Hq, Hkv, hd, out=self.att)
            ops.gemm_a16w4_fwd(self.att, *L["o"], None, D, Hq * hd, out=self.tmp)
            fused = self.fuse_norm and ops.gemm_a16w4_fwd_rmsnorm(h, self.tmp, L["ln2"], self.eps, h_alt, *L["gu"], 2 * I, D,
                                                                 out=self.act, silu_pair=True, hf_rounding=self.hf)
            if fused is None or fused is False:
                ops.add_rmsnorm(h, self.tmp, L["ln2"], self.eps, out=self.xn, hf_rounding=self.hf)
                ops.gemm_a16w4_fwd_silu(self.xn, *L["gu"], I, D, out=self.act, gate_up=self.gu, hf_rounding=self.hf)
            else:
                h, h_alt = h_alt, h
            ops.gemm_a16w4_fwd(self.act, *L["down"], None, D, I, out=self.tmp)
            delta = self.tmp
        norm, head, embed = self.ends
        ops.add_rmsnorm(h, delta, norm, self.eps, out=self.xn, hf_rounding=self.hf)
        self.logits = ops.linear_rows(self.xn, head)
        # argmax, position += 1 and the next step's embedding row in one launch
        ops.argmax_embed(self.logits, self.tok, self.pos, embed, self.h)

    def _seed(self, first, p):
        self.tok.copy_(first); self.pos.fill_(p)
        self.h.copy_(torch.nn.functional.embedding(self.tok, self.ends[2]))

    def _prompt_step(self, prompt):
        """The layers over all tokens of the prompt; logits of the last token of every sequence."""
        from . import ops
        B, P = prompt.shape
        D, I, Hq, Hkv, hd = self.D, self.I, self.Hq, self.Hkv, self.hd
        norm, head, embed = self.ends
        if not self.cache.layers[0].is_initialized:       # the modules would allocate the cache at their first call
            self.cache.early_initialization(B, Hkv, hd, torch.bfloat16, self.device)
        pos = torch.arange(P, device=self.device).repeat(B)
        h = torch.nn.functional.embedding(prompt.reshape(-1), embed)
        delta = None
        for li, L in enumerate(self.layers):
            kc, vc = self.cache.layers[li].keys, self.cache.layers[li].values
            qkv = ops.gemm_a16w4_fwd(ops.add_rmsnorm(h, delta, L["ln1"], self.eps), *L["qkv"], None, (Hq + 2 * Hkv) * hd, D)
            ops.rope_kv_store(qkv, pos, self.inv_freq, kc, vc, Hq, Hkv, hd, tokens_per_seq=P)
            q = qkv.view(B, P, -1, hd)[:, :, :Hq].transpose(1, 2)
            att = torch.nn.functional.scaled_dot_product_attention(q, kc[:, :, :P], vc[:, :, :P], is_causal=True, enable_gqa=Hq != Hkv)
            o = ops.gemm_a16w4_fwd(att.transpose(1, 2).reshape(B * P, Hq * hd), *L["o"], None, D, Hq * hd)
            act = ops.gemm_a16w4_fwd_silu(ops.add_rmsnorm(h, o, L["ln2"], self.eps), *L["gu"], I, D)
            delta = ops.gemm_a16w4_fwd(act, *L["down"], None, D, I)
        last = [t.view(B, P, D)[:, -1].contiguous() for t in (h, delta)]
        return ops.linear_rows(ops.add_rmsnorm(*last, norm, self.eps), head)

    @torch.no_grad()
    def _prefill(self, prompt):
        p = prompt.shape[1]
        if self.prompt_kernels:
            with sdpa_kernel(_SDPA):
                return self._prompt_step(prompt).argmax(-1)
        self.cache.reset()
        with sdpa_kernel(_SDPA):
            out = self.model(input_ids=prompt, past_key_values=self.cache,
                             cache_position=torch.arange(p, device=self.device), use_cache=True)
        return out.logits[:, -1].argmax(-1)

    @torch.no_grad()
    def _capture(self, first, p):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):                       # warm-up: lazy initialisations must not be captured
            self._seed(first, p)
            self._step(); self._step()
        torch.cuda.current_stream().wait_stream(side)
        self.graph = torch.cuda.CUDAGraph()
        self._seed(first, p)
        with torch.cuda.graph(self.graph):
            self._step()

    @torch.no_grad()
    def generate(self, prompt: torch.Tensor, max_new_tokens: int, use_graph: bool = True) -> torch.Tensor:
        b, p = prompt.shape
        if b != self.batch or p + max_new_tokens > self.max_len:
            raise ValueError("prompt does not fit the decoder's batch size / cache length")
        self.model.eval()
        self._take_weights()                                # (its copies run while the host looks at the modules)
        self.prompt_kernels = self._kernels_serve_prompts()
        if self.prompt_kernels:                             # (else they may belong to the length of the last prompt)
            self.inv_freq.copy_(self.model.model.rotary_emb.inv_freq)
        if use_graph and self.graph is None:
            self._capture(self._prefill(prompt), p)         # throw-away prefill: capture needs an allocated cache and tokens to start from
        first = self._prefill(prompt)
        self._seed(first, p)
        toks = [first.clone()]
        for _ in range(max_new_tokens - 1):
            if use_graph:
                self.graph.replay()
            else:
                self._step()
            toks.append(self.tok.clone())
        return torch.stack(toks, dim=1)
