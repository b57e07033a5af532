"""Greedy decode with the decode step captured as a CUDA graph against the same loop run eagerly."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_graphed_greedy_decode_equals_eager_loop():
    from latentq_llm_b200 import finetune as ft
    from latentq_llm_b200.generate import GraphedGreedyDecoder
    model = ft.build_model("llama-tiny", "cuda", seed=3)
    ft.quantize_decoder(model, lbit=4, gbit=16)
    model.eval()
    dec = GraphedGreedyDecoder(model, batch=2, max_len=96)
    g = torch.Generator(device="cuda").manual_seed(1)
    for trial in range(2):                                   # the second prompt replays the graph captured for the first
        prompt = torch.randint(0, 1024, (2, 40 + 8 * trial), device="cuda", generator=g)
        eager = dec.generate(prompt, 12, use_graph=False)
        graphed = dec.generate(prompt, 12, use_graph=True)
        assert eager.shape == (2, 12) and torch.equal(eager, graphed), trial
    assert dec.graph is not None
    with pytest.raises(ValueError):
        dec.generate(torch.zeros((2, 90), dtype=torch.long, device="cuda"), 12)


@pytest.mark.parametrize("arch", ["llama-tiny", "llama-gqa-tiny"])
def test_fused_llama_decoder_against_the_eager_modules(arch):
    """The decode step as a chain of this library's kernels (fused q|k|v and gate|up projections, RMSNorm, RoPE with
    the KV-cache write, single-query attention, silu*up) against the model's own eager modules on the same prompt:
    logits of the first decode step agree closely, greedy tokens agree wherever the eager loop's choice was not a
    near-tie, and graph replay equals the eager chain of the same kernels bit for bit."""
    from latentq_llm_b200 import finetune as ft
    from latentq_llm_b200.generate import FusedLlamaGreedyDecoder, GraphedGreedyDecoder, _SDPA
    from torch.nn.attention import sdpa_kernel
    model = ft.build_model(arch, "cuda", seed=3)
    ft.quantize_decoder(model, lbit=4, gbit=16)
    model.eval()
    B, P, T = 2, 40, 10
    fused = FusedLlamaGreedyDecoder(model, batch=B, max_len=96)
    ref = GraphedGreedyDecoder(model, batch=B, max_len=96)
    g = torch.Generator(device="cuda").manual_seed(1)
    prompt = torch.randint(0, 1024, (B, P), device="cuda", generator=g)

    # logits of the first decode step through the eager modules
    ref.cache.reset()
    with torch.no_grad(), sdpa_kernel(_SDPA):
        out = model(input_ids=prompt, past_key_values=ref.cache, cache_position=torch.arange(P, device="cuda"), use_cache=True)
        first = out.logits[:, -1:].argmax(-1)
        out = model(input_ids=first, past_key_values=ref.cache, cache_position=torch.tensor([P], device="cuda"), use_cache=True)
    want_logits = out.logits[:, -1].float()

    toks_eager_chain = fused.generate(prompt, 2, use_graph=False)
    got_logits = fused.logits.float()
    assert torch.equal(toks_eager_chain[:, 0], first.view(-1))
    diff = (got_logits - want_logits).abs().max().item()
    spread = (want_logits.max() - want_logits.min()).item()
    assert diff <= 0.02 * spread, (diff, spread)

    want = ref.generate(prompt, T, use_graph=False)
    got = fused.generate(prompt, T, use_graph=False)
    graphed = fused.generate(prompt, T, use_graph=True)
    assert torch.equal(got, graphed), "graph replay must equal the eager chain of the same kernels"
    agree = (got == want).float().mean().item()
    assert torch.equal(got[:, :2], want[:, :2]) and agree >= 0.7, agree
    # a second prompt replays the captured graph
    prompt2 = torch.randint(0, 1024, (B, P + 8), device="cuda", generator=g)
    assert torch.equal(fused.generate(prompt2, T, use_graph=True), fused.generate(prompt2, T, use_graph=False))


@pytest.mark.parametrize("B", [1, 2])
def test_fused_decoder_with_the_norm_inside_the_projections_decodes_the_same_tokens(monkeypatch, B):
    """One or two sequences at hidden size 4096: the residual add and both RMSNorms of a layer run inside the q|k|v and
    gate|up launches, the residual stream alternating between two buffers.  Same bits as the chain with separate norm
    launches: logits and tokens identical, eager chain and graph replay alike."""
    from latentq_llm_b200 import finetune as ft, ops
    from latentq_llm_b200.generate import FusedLlamaGreedyDecoder
    model = ft.build_model("llama-wide-tiny", "cuda", seed=5)
    ft.quantize_decoder(model, lbit=4, gbit=16)
    model.eval()
    P, T = 24, 8
    g = torch.Generator(device="cuda").manual_seed(B)
    prompt = torch.randint(0, 1024, (B, P), device="cuda", generator=g)
    monkeypatch.setenv("LQ_DECODE_NO_FUSED_NORM", "1")
    plain = FusedLlamaGreedyDecoder(model, batch=B, max_len=64)
    assert not plain.fuse_norm
    want = plain.generate(prompt, T, use_graph=False)
    want_logits = plain.logits.clone()
    monkeypatch.delenv("LQ_DECODE_NO_FUSED_NORM")
    fused = FusedLlamaGreedyDecoder(model, batch=B, max_len=64)
    assert fused.fuse_norm
    calls = []
    real = ops.gemm_a16w4_fwd_rmsnorm
    monkeypatch.setattr(ops, "gemm_a16w4_fwd_rmsnorm", lambda *a, **k: (calls.append(1), real(*a, **k))[1])
    got = fused.generate(prompt, T, use_graph=False)
    assert calls and torch.equal(got, want) and torch.equal(fused.logits, want_logits)
    assert torch.equal(fused.generate(prompt, T, use_graph=True), want)
    assert torch.equal(fused.logits, want_logits)


@pytest.mark.parametrize("arch,use_graph", [("llama-gqa-tiny", False), ("llama-gqa-tiny", True), ("llama-wide-tiny", True)])
def test_fused_decoder_after_the_weights_changed_equals_a_new_decoder(arch, use_graph):
    """Codes and scales written in place (as an optimizer step does), codes set anew, a norm and the head elsewhere: prompt and steps of the next call
    have the new weights, whether the step was captured before or not."""
    from latentq_llm_b200 import finetune as ft
    from latentq_llm_b200.generate import FusedLlamaGreedyDecoder
    model = ft.build_model(arch, "cuda", seed=3)
    ft.quantize_decoder(model, lbit=0, gbit=16)
    model.eval()
    B, P, T = 2, 40, 6
    g = torch.Generator(device="cuda").manual_seed(1)
    prompt = torch.randint(0, 1024, (B, P), device="cuda", generator=g)
    dec = FusedLlamaGreedyDecoder(model, batch=B, max_len=64)
    dec.generate(prompt, T, use_graph=use_graph)
    before = dec.logits.clone()
    for change in range(3):
        layer = model.model.layers[change % 2]
        if change == 0:
            layer.self_attn.k_proj.weight.data.copy_(layer.self_attn.k_proj.weight.data.flip(0))
            layer.mlp.up_proj.scales.data.mul_(0.5)
        elif change == 1:
            w = layer.self_attn.q_proj.weight
            w.set_value(w.data.flip(0), w.qparam)
        else:
            layer.input_layernorm.weight.data = layer.input_layernorm.weight.data * 1.5
            model.lm_head.weight.data = model.lm_head.weight.data.flip(0)
            w = layer.mlp.down_proj.weight
            w.set_value(w.data.flip(0), w.qparam)
        got = dec.generate(prompt, T, use_graph=use_graph)
        new = FusedLlamaGreedyDecoder(model, batch=B, max_len=64)
        want = new.generate(prompt, T, use_graph=use_graph)
        assert torch.equal(got, want) and torch.equal(dec.logits, new.logits) and not torch.equal(dec.logits, before), change
        assert torch.equal(dec.generate(prompt, 1, use_graph=use_graph)[:, 0], want[:, 0])
        before = dec.logits.clone()


def _in_64_bits(model):
    """The model with its weights as the codes say, in 64 bits (norms and angles stay in 32, as the classes compute them)."""
    from transformers import LlamaForCausalLM
    from latentq_llm_b200.quant import QLinearA16W4
    with torch.device("cuda"):
        ref = LlamaForCausalLM(model.config).double().eval()
    ref.model.rotary_emb.inv_freq = model.model.rotary_emb.inv_freq.float()
    own = dict(model.named_modules())
    with torch.no_grad():
        for name, mod in ref.named_modules():
            src = own[name]
            if isinstance(src, QLinearA16W4):
                n, k = src.wshape
                b = src.weight.data.view(torch.uint8).view(n, -1)
                q = torch.stack([b >> 4, b & 15], 2).view(n, k // 128, 128).double()
                s, z = (t.double().view(n, k // 128, 1) for t in src.weight.qparam[:2])
                mod.weight.copy_(((q - z) * s).view(n, k))
            elif isinstance(getattr(mod, "weight", None), torch.nn.Parameter):
                mod.weight.copy_(src.weight)
    return ref


LLAMA3 = {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 32, "rope_theta": 10000.0}


@pytest.mark.parametrize("arch,P,rope", [("llama-tiny", 1, None), ("llama-tiny", 67, {"rope_type": "linear", "factor": 2.0, "rope_theta": 10000.0}),
                                         ("llama-gqa-tiny", 9, None), ("llama-gqa-tiny", 131, LLAMA3), ("llama-wide-tiny", 40, None)])
def test_prompt_through_the_kernels_and_through_the_modules(monkeypatch, arch, P, rope):
    """Logits of the last prompt token and the cache rows of every layer, against 64 bits: the kernels' route is no further off than the modules' (both round
    to bf16 in the same places, so their errors are samples of one distribution: half more is allowed).  One token, token counts of the decode kernels and of
    the GEMM, the RoPE kernels of few and of many heads, grouped key heads, frequencies of other rope types."""
    from latentq_llm_b200 import finetune as ft
    from latentq_llm_b200.generate import FusedLlamaGreedyDecoder
    monkeypatch.setitem(ft.ARCHS, "under test", dict(ft.ARCHS[arch], **({"rope_parameters": rope} if rope else {})))
    model = ft.build_model("under test", "cuda", seed=3)
    ft.quantize_decoder(model, lbit=0, gbit=16)
    model.eval()
    B = 2
    prompt = torch.randint(0, 1024, (B, P), device="cuda", generator=torch.Generator(device="cuda").manual_seed(P))
    with torch.no_grad():
        out = _in_64_bits(model)(input_ids=prompt, use_cache=True)
    want = [out.logits[:, -1]] + [t for l in out.past_key_values.layers for t in (l.keys, l.values)]

    def of(dec, logits):
        return [logits] + [t[:, :, :P] for l in dec.cache.layers for t in (l.keys, l.values)]

    dec, logits = FusedLlamaGreedyDecoder(model, batch=B, max_len=160), []
    real = dec._prompt_step
    monkeypatch.setattr(dec, "_prompt_step", lambda p: (logits.append(real(p)), logits[-1])[1])
    first = dec.generate(prompt, 1, use_graph=False)[:, 0]
    assert dec.prompt_kernels and len(logits) == 1 and torch.equal(first, logits[0].argmax(-1))
    assert not any(t[:, :, P:].any() for l in dec.cache.layers for t in (l.keys, l.values))
    kernels = of(dec, logits[0])

    seen = []
    hook = model.lm_head.register_forward_hook(lambda mod, args, output: seen.append(output[:, -1]))
    watched = FusedLlamaGreedyDecoder(model, batch=B, max_len=160)
    first = watched.generate(prompt, 1, use_graph=False)[:, 0]
    assert not watched.prompt_kernels and len(seen) == 1 and torch.equal(first, seen[0].argmax(-1))
    modules = of(watched, seen[0])
    hook.remove()

    for i, (k, m, w) in enumerate(zip(kernels, modules, want)):
        ek, em = (float((t.double() - w).norm() / w.norm()) for t in (k, m))
        assert ek <= 1.5 * em and em < 0.05, (i, ek, em)


@pytest.mark.parametrize("cfg", [{"rope_parameters": {"rope_type": "yarn", "factor": 4.0, "rope_theta": 10000.0}},
                                 {"rope_parameters": {"rope_type": "dynamic", "factor": 2.0, "rope_theta": 10000.0}}, {"attn_implementation": "eager"}], ids=str)
def test_prompts_that_stay_with_the_modules(monkeypatch, cfg):
    """The first token is the modules' own; graph replay equals the eager chain behind such a prompt too."""
    from latentq_llm_b200 import finetune as ft
    from latentq_llm_b200.generate import FusedLlamaGreedyDecoder
    monkeypatch.setitem(ft.ARCHS, "under test", dict(ft.ARCHS["llama-gqa-tiny"], **cfg))
    model = ft.build_model("under test", "cuda", seed=3)
    ft.quantize_decoder(model, lbit=0, gbit=16)
    model.eval()
    prompt = torch.randint(0, 1024, (2, 40), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    with torch.no_grad():
        logits = model(input_ids=prompt).logits[:, -1].float()
    dec = FusedLlamaGreedyDecoder(model, batch=2, max_len=64)
    got = dec.generate(prompt, 6)
    assert not dec.prompt_kernels and torch.equal(got, dec.generate(prompt, 6, use_graph=False))
    chosen = logits.gather(1, got[:, :1])[:, 0]
    assert bool((chosen >= logits.max(1).values - 0.01 * (logits.max() - logits.min())).all())        # (near-ties: another attention backend without a cache)
