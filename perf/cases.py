"""The work that programs built on this package spend their GPU time on, as cases that a timing program can run.

Six kinds of work, each through the entry points that a user's program calls:

  linear      `QLinearA16W4` forward without gradients: eager decode (1 token) to prefill (4096 tokens)
  train       `QLinearA16W4` forward + backward of one micro-batch, the weight gradient accumulated into its arena
  decode      a captured decode step of Llama-architecture layers, written with the `ops` launches of a decode chain
  generate    `FusedLlamaGreedyDecoder.generate`: prefill and greedy decode of a small model, end to end
  optimizer   `MyAdam.step` over one quantized weight (8-bit states) and the dense parameters beside it
  fold        `ops.a16w4_fold_delta`: an update folded into packed codes and residual words
  a8w8        per-token activation quantizer + int8 GEMM with scaled epilogue
  a8w8_train  `QLinearA8W8` forward + backward of two micro-batches with the 8-bit gradient accumulator

Layer sizes are those of the OPT-1.3B and Llama-2-7B architectures that the fine-tuning and decode code is configured for;
drawn cases add token counts between and beside the listed ones, odd ones among them, and other layer sizes of the same range.
"""
import math

import torch

from latentq_llm_b200 import finetune, ops, quant
from latentq_llm_b200.generate import FusedLlamaGreedyDecoder

GROUP = 128
EPS = 1e-5
ROPE_THETA = 10000.0

# (in, out) of the linears of the two architectures: attention, fused q|k|v, MLP up and down
OPT = [(2048, 2048), (2048, 8192), (8192, 2048)]
LLAMA = [(4096, 4096), (4096, 11008), (11008, 4096), (4096, 12288)]


def listed():
    return [
        # one token through one attention projection, eager: what a `generate` loop over the modules does 4 times a layer
        dict(name="linear_1_token", kind="linear", tokens=1, K=4096, N=4096, bias=False),
        # a short prompt (or a decode batch of that size): ragged token count, weight-bound
        dict(name="linear_100_tokens", kind="linear", tokens=100, K=4096, N=11008, bias=False),
        # prefill / evaluation of a full micro-batch
        dict(name="linear_4096_tokens", kind="linear", tokens=4096, K=11008, N=4096, bias=False),
        # OPT-1.3B fine-tuning: micro-batch 4 x 512, the MLP's first linear with its bias
        dict(name="train_opt_fc1", kind="train", tokens=2048, K=2048, N=8192, bias=True),
        # Llama-2-7B fine-tuning: micro-batch 4 x 1024, an MLP up projection
        dict(name="train_llama_up", kind="train", tokens=4096, K=4096, N=11008, bias=False),
        # interactive decode: one sequence with half a thousand tokens of context
        dict(name="decode_batch_1", kind="decode", batch=1, context=512, layers=2, D=4096, I=11008, heads=32, kv_heads=32),
        # served decode: sixteen sequences
        dict(name="decode_batch_16", kind="decode", batch=16, context=512, layers=2, D=4096, I=11008, heads=32, kv_heads=32),
        # a whole call: prompt in, tokens out
        dict(name="generate_batch_2", kind="generate", batch=2, prompt=200, new_tokens=32, layers=2),
        # the optimizer step of one MLP weight of Llama-2-7B, with the norms of its layer
        dict(name="optimizer_llama_mlp", kind="optimizer", K=4096, N=11008, wbit=4, dense=4),
        # requantize with counter-based dither: an update of 2^27 weights folded back into int4 codes + residual
        dict(name="fold_philox", kind="fold", K=8192, N=16384, dither="philox"),
        # A8W8 serving / evaluation on OPT-1.3B: micro-batch 4 x 512, outlier channels in the activations
        dict(name="a8w8_opt_fc1", kind="a8w8", tokens=2048, K=2048, N=8192, bias=True),
        # A8W8 fine-tuning with the 8-bit gradient accumulator
        dict(name="a8w8_train_opt_fc2", kind="a8w8_train", tokens=2048, K=8192, N=2048, bias=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _layer_size(rng, shapes):
    """Mostly a layer of the two architectures, else sizes of the same range."""
    if rng.random() < 0.7:
        return rng.choice(shapes)
    return 128 * _log_int(rng, 8, 86), 64 * _log_int(rng, 16, 172)


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "train", "train", "decode", "decode", "generate", "optimizer", "fold", "a8w8",
                       "a8w8_train"])
    if kind == "linear":
        K, N = _layer_size(rng, OPT + LLAMA)
        return dict(kind=kind, tokens=_log_int(rng, 1, 4096), K=K, N=N, bias=rng.random() < 0.5)
    if kind == "train":
        K, N = _layer_size(rng, OPT + LLAMA[:3])
        return dict(kind=kind, tokens=8 * _log_int(rng, 16, 512), K=K, N=N, bias=rng.random() < 0.5)
    if kind == "decode":
        D, I, heads, kv = rng.choice([(4096, 11008, 32, 32), (4096, 11008, 32, 32), (2048, 5632, 16, 16), (4096, 14336, 32, 8)])
        return dict(kind=kind, batch=_log_int(rng, 1, 64), context=_log_int(rng, 64, 1500), layers=2, D=D, I=I, heads=heads, kv_heads=kv)
    if kind == "generate":
        return dict(kind=kind, batch=rng.randint(1, 6), prompt=_log_int(rng, 30, 500), new_tokens=rng.randint(8, 40), layers=2)
    if kind == "optimizer":
        K, N = _layer_size(rng, OPT + LLAMA)
        return dict(kind=kind, K=K, N=N, wbit=rng.choice([4, 4, 4, 8]), dense=rng.randint(1, 12))
    if kind == "fold":
        return dict(kind=kind, K=128 * _log_int(rng, 8, 86), N=64 * _log_int(rng, 16, 190), dither=rng.choice(["hash", "philox"]))
    K, N = _layer_size(rng, OPT)
    if kind == "a8w8":
        return dict(kind=kind, tokens=_log_int(rng, 16, 8192), K=K, N=N, bias=rng.random() < 0.5)
    return dict(kind=kind, tokens=8 * _log_int(rng, 16, 512), K=K, N=N, bias=rng.random() < 0.5)


# ---- inputs (plain torch) --------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000 + seed)


def _randn(g, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device="cuda", generator=g) * std).to(dtype)


def _int4(g, N, K):
    """W ~ N(0, 0.02) as min/max int4 codes of groups of 128: packed codes [N*K/2], scales and zeros bf16 [N*K/128, 1]."""
    w = torch.randn(N * K // GROUP, GROUP, device="cuda", generator=g) * 0.02
    lo, hi = w.amin(1, keepdim=True), w.amax(1, keepdim=True)
    s = ((hi - lo) / 15).to(torch.bfloat16)
    z = torch.round(-lo / s.float()).clamp(0, 15)
    q = torch.round(w / s.float() + z).clamp(0, 15).to(torch.uint8).view(-1, 2)
    return ((q[:, 0] << 4) | q[:, 1]).view(torch.int8), s, z.to(torch.bfloat16)


def _w64(packed, s, z, N, K):
    """The weight matrix that codes and group parameters stand for, in 64 bits."""
    b = packed.view(torch.uint8)
    q = torch.stack([b >> 4, b & 15], 1).view(-1, GROUP).double()
    return ((q - z.double()) * s.double()).view(N, K)


def _int8(g, N, K):
    w = torch.randn(N, K, device="cuda", generator=g) * 0.02
    s = (w.abs().amax(1, keepdim=True) / 127).to(torch.bfloat16)
    return torch.round(w / s.float()).clamp(-128, 127).to(torch.int8), s


def _outlier_tokens(g, M, K):
    """N(0, 1) activations with 1 % of the channels 20 times as large."""
    x = torch.randn(M, K, device="cuda", generator=g)
    ch = torch.randperm(K, device="cuda", generator=g)[:max(1, K // 100)]
    x[:, ch] *= 20.0
    return x.to(torch.bfloat16)


def _linear_inputs(case, seed):
    g = _gen(seed)
    N, K = case["N"], case["K"]
    d = dict(w=_int4(g, N, K), x=_randn(g, case["tokens"], K), bias=_randn(g, N, std=0.1) if case["bias"] else None)
    if case["kind"] == "train":
        d["dy"] = _randn(g, case["tokens"], N, std=1e-3)
    return d


def _linear_module(d, N, K, gbit=16):
    m = quant.QLinearA16W4(K, N, bias=d["bias"] is not None, lbit=4, gbit=gbit)
    codes, s, z = d["w"]
    m.scales.data, m.zeros.data = s, z
    if d["bias"] is not None:
        m.bias.data = d["bias"]
        m.bias.requires_grad_(False)
    m.weight.set_value(codes, [m.scales, m.zeros, m.wshape])
    m.to("cuda")
    return m


def _layer_inputs(g, D, I, heads, kv_heads):
    hd = D // heads
    return dict(qkv=_int4(g, (heads + 2 * kv_heads) * hd, D), o=_int4(g, D, heads * hd), gu=_int4(g, 2 * I, D), down=_int4(g, D, I),
                ln1=(1 + 0.1 * torch.randn(D, device="cuda", generator=g)).to(torch.bfloat16),
                ln2=(1 + 0.1 * torch.randn(D, device="cuda", generator=g)).to(torch.bfloat16))


def _decode_inputs(case, seed):
    g = _gen(seed)
    B, D, heads, kv = case["batch"], case["D"], case["heads"], case["kv_heads"]
    hd, ctx = D // heads, case["context"]
    layers = [_layer_inputs(g, D, case["I"], heads, kv) for _ in range(case["layers"])]
    for L in layers:
        L["k"], L["v"] = (_randn(g, B, kv, ctx + 8, hd) for _ in range(2))
    pos = torch.randint(ctx // 2, ctx, (B,), device="cuda", generator=g)          # sequences of different lengths
    return dict(layers=layers, h=_randn(g, B, D), pos=pos)


def _inv_freq(hd):
    return 1.0 / (ROPE_THETA ** (torch.arange(0, hd, 2, dtype=torch.float32, device="cuda") / hd))


def _generate_inputs(case, seed):
    """Weights of a small Llama-architecture model and a prompt.  The embedding is large and the head's rows are a permutation
    of the embedding's, so that the next token is as clear as it is for a trained model."""
    g = _gen(seed)
    cfg = finetune.ARCHS["llama-2-7b"]
    D, I, H, V = cfg["hidden_size"], cfg["intermediate_size"], cfg["num_attention_heads"], cfg["vocab_size"]
    layers = [_layer_inputs(g, D, I, H, H) for _ in range(case["layers"])]
    embed = torch.randn(V, D, device="cuda", generator=g)
    perm = torch.randperm(V, device="cuda", generator=g)
    return dict(layers=layers, embed=(2 * embed).to(torch.bfloat16), head=(0.02 * embed[perm]).to(torch.bfloat16),
                norm=(1 + 0.1 * torch.randn(D, device="cuda", generator=g)).to(torch.bfloat16), perm=perm,
                prompt=torch.randint(0, V, (case["batch"], case["prompt"]), device="cuda", generator=g), D=D, I=I, H=H, V=V)


# ---- prepare / run ---------------------------------------------------------------------------------------------------
def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def _prepare_linear(case, seed):
    d = _linear_inputs(case, seed)
    return dict(kind="linear", m=_linear_module(d, case["N"], case["K"]), x=d["x"])


@torch.no_grad()
def _run_linear(s):
    return s["m"](s["x"])


def _prepare_train(case, seed):
    d = _linear_inputs(case, seed)
    m = _linear_module(d, case["N"], case["K"])
    m.add_hook(direct=True)
    m.weight.grad = torch.zeros(case["N"], case["K"], dtype=torch.bfloat16, device="cuda")      # its view of the gradient arena
    return dict(kind="train", m=m, x=d["x"].requires_grad_(True), dy=d["dy"])


def _run_train(s):
    s["x"].grad = None
    y = s["m"](s["x"])
    y.backward(s["dy"])
    return dict(y=y.detach(), dx=s["x"].grad, dw=s["m"].weight.grad)


def _prepare_decode(case, seed):
    d = _decode_inputs(case, seed)
    D, heads, kv = case["D"], case["heads"], case["kv_heads"]
    s = dict(kind="decode", Hq=heads, Hkv=kv, hd=D // heads, D=D, I=case["I"], pos=d["pos"], h0=d["h"], inv=_inv_freq(D // heads),
             layers=[dict(L, **{k: (L[k][0], L[k][1].view(-1), L[k][2].view(-1)) for k in ("qkv", "o", "gu", "down")}) for L in d["layers"]])
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), torch.no_grad():
        _decode_step(s)
    torch.cuda.current_stream().wait_stream(side)
    s["graph"] = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(s["graph"]):
        s["out"] = _decode_step(s)
    return s


def _decode_step(s):
    """One token per sequence through the layers: the launches that a decode loop captures once and replays per token."""
    Hq, Hkv, hd, D, I, pos = s["Hq"], s["Hkv"], s["hd"], s["D"], s["I"], s["pos"]
    h, delta = s["h0"].clone(), None
    with ops.decode_chain():
        for L in s["layers"]:
            kc, vc = L["k"], L["v"]
            rope = (pos, s["inv"], kc, vc, Hq, Hkv, hd, D)
            h2 = torch.empty_like(h)
            qkv = ops.gemm_a16w4_fwd_qkv_rope(None, *L["qkv"], *rope, norm=(h, delta, L["ln1"], EPS, h2)) if len(h) <= 2 else None
            if qkv is not None:
                h = h if delta is None else h2
            else:
                xn = ops.add_rmsnorm(h, delta, L["ln1"], EPS)
                qkv = ops.gemm_a16w4_fwd_qkv_rope(xn, *L["qkv"], *rope) if len(h) <= 16 else None
                if qkv is None:
                    qkv = ops.gemm_a16w4_fwd(xn, *L["qkv"], None, (Hq + 2 * Hkv) * hd, D)
                    ops.rope_kv_store(qkv, pos, s["inv"], kc, vc, Hq, Hkv, hd)
            att = ops.decode_attention(qkv, pos, kc, vc, Hq, Hkv, hd)
            o = ops.gemm_a16w4_fwd(att, *L["o"], None, D, Hq * hd)
            h2 = torch.empty_like(h)
            act = ops.gemm_a16w4_fwd_rmsnorm(h, o, L["ln2"], EPS, h2, *L["gu"], 2 * I, D, silu_pair=True) if len(h) <= 2 else None
            if act is not None:
                h = h2
            else:
                act = ops.gemm_a16w4_fwd_silu(ops.add_rmsnorm(h, o, L["ln2"], EPS), *L["gu"], I, D)
            delta = ops.gemm_a16w4_fwd(act, *L["down"], None, D, I)
    return h + delta


def _run_decode(s):
    s["graph"].replay()
    return dict(h=s["out"], cache=[(L["k"], L["v"]) for L in s["layers"]])


def _prepare_generate(case, seed):
    d = _generate_inputs(case, seed)
    D, I = d["D"], d["I"]
    model = finetune.build_model("llama-2-7b", layers=case["layers"])
    finetune.quantize_decoder(model)
    with torch.no_grad():
        model.model.embed_tokens.weight.copy_(d["embed"])
        model.lm_head.weight.copy_(d["head"])
        model.model.norm.weight.copy_(d["norm"])
        for layer, L in zip(model.model.layers, d["layers"]):
            layer.input_layernorm.weight.copy_(L["ln1"])
            layer.post_attention_layernorm.weight.copy_(L["ln2"])
            a, m = layer.self_attn, layer.mlp
            for mods, w in (((a.q_proj, a.k_proj, a.v_proj), L["qkv"]), ((a.o_proj,), L["o"]), ((m.gate_proj, m.up_proj), L["gu"]),
                            ((m.down_proj,), L["down"])):
                for mod, part in zip(mods, zip(*(t.chunk(len(mods)) for t in w))):
                    mod.scales.data, mod.zeros.data = part[1].contiguous(), part[2].contiguous()
                    mod.weight.set_value(part[0], [mod.scales, mod.zeros, mod.wshape])
    dec = FusedLlamaGreedyDecoder(model, case["batch"], case["prompt"] + case["new_tokens"])
    dec.generate(d["prompt"], 2)                                  # captures the decode step
    return dict(kind="generate", dec=dec, prompt=d["prompt"], n=case["new_tokens"])


def _run_generate(s):
    tokens = s["dec"].generate(s["prompt"], s["n"])
    return dict(tokens=tokens, logits=s["dec"].logits)


def _prepare_optimizer(case, seed):
    g = _gen(seed)
    N, K = case["N"], case["K"]
    p = quant.QuantTensor([N, K], wbit=case["wbit"], gbit=16, lbit=4)
    if case["wbit"] == 4:
        codes, sc, z = _int4(g, N, K)
        p.set_value(codes, [sc, z, [N, K]])
    else:
        codes, sc = _int8(g, N, K)
        p.set_value(codes, sc)
    dense = [torch.nn.Parameter(torch.ones(K, dtype=torch.bfloat16, device="cuda")) for _ in range(case["dense"])]
    opt = quant.MyAdam([{"params": [p], "weight_decay": 0.0}, {"params": dense, "weight_decay": 0.0}], lr=1e-4, betas=(0.9, 0.95))
    s = dict(kind="optimizer", opt=opt, p=p, dense=dense)
    rows = torch.exp(torch.randn(N, 1, device="cuda", generator=g))      # gradients of different rows differ in size
    for _ in range(2):                                                   # states as they are in the middle of a run
        s["grad"] = (torch.randn(N, K, device="cuda", generator=g) * rows * 1e-4).to(torch.bfloat16)
        s["dgrad"] = [_randn(g, K, std=1e-3) for _ in dense]
        _run_optimizer(s)
    return s


def _run_optimizer(s):
    s["p"].grad = s["grad"]
    for q, dg in zip(s["dense"], s["dgrad"]):
        q.grad = dg
    s["opt"].step()
    st = s["opt"].state[s["p"]]
    return dict(codes=s["p"].data, words=s["p"].residual.residual_int, **{k: st[k] for k in ("state1", "state2", "qmap1", "qmap2", "absmax1", "absmax2")},
                dense=[q.data for q in s["dense"]])


def _prepare_fold(case, seed):
    g = _gen(seed)
    N, K = case["N"], case["K"]
    codes, sc, z = _int4(g, N, K)
    words = torch.randint(-2 ** 31, 2 ** 31, (N * K // 8,), device="cuda", generator=g, dtype=torch.int64).to(torch.int32)
    opts = ops.make_opts(codec=ops.CODEC_THREEFOLD, dither=ops.DITHER_PHILOX if case["dither"] == "philox" else ops.DITHER_HASH, seed=seed, step=3)
    return dict(kind="fold", codes=codes, words=words, scales=sc.view(-1), zeros=z.view(-1), delta=_randn(g, N * K, std=1e-4), opts=opts)


def _run_fold(s):
    ops.a16w4_fold_delta(s["codes"], s["words"], s["delta"], s["scales"], s["zeros"], s["opts"])
    return s["codes"], s["words"]


def _a8w8_inputs(case, seed):
    g = _gen(seed)
    N, K = case["N"], case["K"]
    w8, sc = _int8(g, N, K)
    d = dict(w8=w8, scale=sc, x=_outlier_tokens(g, case["tokens"], K), bias=_randn(g, N, std=0.1) if case["bias"] else None)
    if case["kind"] == "a8w8_train":
        d["x"] = [_randn(g, case["tokens"], K), _randn(g, case["tokens"], K)]
        d["dy"] = [_randn(g, case["tokens"], N, std=1e-3) for _ in range(2)]
    return d


def _prepare_a8w8(case, seed):
    d = _a8w8_inputs(case, seed)
    return dict(kind="a8w8", x=d["x"], w8=d["w8"], cs=d["scale"].float().view(-1), bias=d["bias"])


def _run_a8w8(s):
    x8, row_scale = ops.act_quant_per_token(s["x"])
    return ops.gemm_a8w8(x8, s["w8"], row_scale, s["cs"], 1.0, s["bias"])


def _prepare_a8w8_train(case, seed):
    d = _a8w8_inputs(case, seed)
    m = quant.QLinearA8W8(case["K"], case["N"], bias=case["bias"], lbit=4, gbit=8)
    m.qscales.data = d["scale"]
    if case["bias"]:
        m.bias.data = d["bias"]
        m.bias.requires_grad_(False)
    m.weight.set_value(d["w8"], m.qscales)
    m.to("cuda")
    m.add_hook()
    return dict(kind="a8w8_train", m=m, x=[x.requires_grad_(True) for x in d["x"]], dy=d["dy"])


def _run_a8w8_train(s):
    m, out = s["m"], []
    m.weight.grad.zero()
    for x, dy in zip(s["x"], s["dy"]):
        x.grad = None
        y = m(x)
        y.backward(dy)
        out.append((y.detach(), x.grad))
    return dict(out=out, grad=m.weight.grad.qdata, grad_scale=m.weight.grad.scale)


_PREPARE = dict(linear=_prepare_linear, train=_prepare_train, decode=_prepare_decode, generate=_prepare_generate,
                optimizer=_prepare_optimizer, fold=_prepare_fold, a8w8=_prepare_a8w8, a8w8_train=_prepare_a8w8_train)
_RUN = dict(linear=_run_linear, train=_run_train, decode=_run_decode, generate=_run_generate, optimizer=_run_optimizer, fold=_run_fold,
            a8w8=_run_a8w8, a8w8_train=_run_a8w8_train)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _w4_bytes(N, K):
    return N * K // 2 + 4 * N * K // GROUP


def _layer_work(case, D, I, heads, kv_heads, tokens):
    hd = D // heads
    shapes = [((heads + 2 * kv_heads) * hd, D), (D, heads * hd), (2 * I, D), (D, I)]
    return sum(_w4_bytes(n, k) for n, k in shapes) + 4 * D, sum(2 * tokens * n * k for n, k in shapes)


def work(case):
    kind = case["kind"]
    if kind in ("linear", "train"):
        M, N, K = case["tokens"], case["N"], case["K"]
        if kind == "linear":
            return dict(bytes=_w4_bytes(N, K) + 2 * M * (K + N) + (2 * N if case["bias"] else 0), flops=2 * M * N * K)
        # x, dy and the weight read, y and dx written, the gradient accumulated (read and written)
        return dict(bytes=_w4_bytes(N, K) + 2 * M * (2 * K + 2 * N) + 4 * N * K, flops=6 * M * N * K)
    if kind == "decode":
        B, D, kv, hd = case["batch"], case["D"], case["kv_heads"], case["D"] // case["heads"]
        by, fl = _layer_work(case, D, case["I"], case["heads"], kv, B)
        keys = B * 3 * case["context"] // 4
        return dict(bytes=case["layers"] * (by + 4 * keys * kv * hd + 4 * B * kv * hd) + 4 * B * D,
                    flops=case["layers"] * (fl + 4 * keys * case["heads"] * hd))
    if kind == "generate":
        cfg = finetune.ARCHS["llama-2-7b"]
        D, I, H, V = cfg["hidden_size"], cfg["intermediate_size"], cfg["num_attention_heads"], cfg["vocab_size"]
        B, P, T, n = case["batch"], case["prompt"], case["new_tokens"], case["layers"]
        by, fl = _layer_work(case, D, I, H, H, 1)
        keys = B * sum(P + t for t in range(T))
        # the weights once for the prompt and once per further token, the cache once per token
        return dict(bytes=T * (n * by + 2 * V * D) + n * 4 * keys * D, flops=B * (P + T - 1) * n * fl + 2 * B * T * V * D + n * 4 * keys * D)
    if kind == "optimizer":
        n = case["N"] * case["K"]
        codes = n // 2 if case["wbit"] == 4 else n
        qp = 4 * n // GROUP if case["wbit"] == 4 else 2 * case["N"]
        blocks = n // (2048 if n % 2048 == 0 else 128)
        return dict(bytes=2 * codes + 2 * (n // 2) + 2 * n + 4 * n + qp + 32 * blocks + 14 * case["K"] * case["dense"], flops=20 * n)
    if kind == "fold":
        n = case["N"] * case["K"]
        return dict(bytes=n + n + 2 * n + 4 * n // GROUP, flops=10 * n)
    M, N, K = case["tokens"], case["N"], case["K"]
    if kind == "a8w8":
        return dict(bytes=2 * M * K + N * K + 2 * M * N + 4 * N + (2 * N if case["bias"] else 0), flops=2 * M * N * K)
    # two micro-batches: x, dy read, y, dx written, the int8 weight read, the int8 accumulator written, then read and written
    return dict(bytes=2 * (2 * M * (2 * K + 2 * N) + N * K) + 3 * N * K, flops=12 * M * N * K)


# ---- tolerances and 64-bit results -----------------------------------------------------------------------------------
def tolerance(case):
    return dict(_TOLERANCE[case["kind"]]) if _TOLERANCE[case["kind"]] != "exact" else "exact"


_TOLERANCE = dict(
    linear={"rel": 1e-2}, train={"rel": 1e-2}, decode={"rel": 2e-2}, generate={"rel": 2e-2},
    # codes, residual words, 8-bit states and their block parameters are bit-defined
    optimizer="exact", fold="exact",
    # integer accumulators, one rounding to bf16
    a8w8={"rel": 1e-2},
    # the 8-bit accumulator's codes round the bf16 gradient: another order of its sums moves a few of them by one
    a8w8_train={"rel": 1e-2, "differ": 1e-2},
)


def exact(case, seed):
    f = _EXACT.get(case["kind"])
    return None if f is None else f(case, seed)


def _exact_linear(case, seed):
    d = _linear_inputs(case, seed)
    w = _w64(*d["w"], case["N"], case["K"])
    y = d["x"].double() @ w.t()
    y = y + d["bias"].double() if d["bias"] is not None else y
    if case["kind"] == "linear":
        return y
    return dict(y=y, dx=d["dy"].double() @ w, dw=d["dy"].double().t() @ d["x"].double())


def _rms64(h, gamma):
    return h / torch.sqrt((h * h).mean(-1, keepdim=True) + EPS) * gamma.double()


def _rope64(x, pos):
    """x [..., tokens, hd], pos [..., tokens]"""
    f = pos.double().unsqueeze(-1) * _inv_freq(x.shape[-1]).double()
    c, s = torch.cat([f, f], -1).cos(), torch.cat([f, f], -1).sin()
    a, b = x.chunk(2, -1)
    return x * c + torch.cat([-b, a], -1) * s


def _heads64(xn, L, heads, kv, hd, D):
    n = (heads + 2 * kv) * hd
    qkv = (xn @ _w64(*L["qkv"], n, D).t()).view(*xn.shape[:-1], heads + 2 * kv, hd)
    return qkv[..., :heads, :], qkv[..., heads:heads + kv, :], qkv[..., heads + kv:, :]


def _mlp64(h, L, I, D):
    gu = _rms64(h, L["ln2"]) @ _w64(*L["gu"], 2 * I, D).t()
    return (torch.nn.functional.silu(gu[..., :I]) * gu[..., I:]) @ _w64(*L["down"], D, I).t()


def _exact_decode(case, seed):
    d = _decode_inputs(case, seed)
    D, I, heads, kv = case["D"], case["I"], case["heads"], case["kv_heads"]
    hd, pos, h, cache = D // heads, d["pos"], d["h"].double(), []
    rows = torch.arange(case["batch"], device="cuda")
    valid = (torch.arange(case["context"] + 8, device="cuda") <= pos[:, None])[:, None]
    for L in d["layers"]:
        q, k, v = _heads64(_rms64(h, L["ln1"]), L, heads, kv, hd, D)
        q, k = _rope64(q, pos[:, None].expand(-1, heads)), _rope64(k, pos[:, None].expand(-1, kv))
        kc, vc = L["k"].double(), L["v"].double()
        kc[rows, :, pos], vc[rows, :, pos] = k, v
        cache.append((kc, vc))
        qg = q.view(-1, kv, heads // kv, hd)
        p = torch.einsum("bgrd,bgtd->bgrt", qg, kc) / math.sqrt(hd)
        p = torch.softmax(p.masked_fill(~valid[:, :, None], -math.inf), -1)
        att = torch.einsum("bgrt,bgtd->bgrd", p, vc).reshape(-1, heads * hd)
        h = h + att @ _w64(*L["o"], D, heads * hd).t()
        h = h + _mlp64(h, L, I, D)
    return dict(h=h, cache=cache)


def _exact_generate(case, seed):
    d = _generate_inputs(case, seed)
    D, I, H, hd = d["D"], d["I"], d["H"], d["D"] // d["H"]
    after = torch.argsort(d["perm"])                                # the head's row perm^-1(t) is token t's embedding
    seq = [d["prompt"]]
    for _ in range(case["new_tokens"] - 1):
        seq.append(after[seq[-1][:, -1:]])
    ids = torch.cat(seq, 1)
    n = ids.shape[1]
    pos = torch.arange(n, device="cuda")
    h = d["embed"][ids].double()
    causal = torch.ones(n, n, dtype=torch.bool, device="cuda").tril()
    for L in d["layers"]:
        q, k, v = (t.transpose(1, 2) for t in _heads64(_rms64(h, L["ln1"]), L, H, H, hd, D))
        q, k = _rope64(q, pos), _rope64(k, pos)
        p = torch.softmax(((q @ k.transpose(-1, -2)) / math.sqrt(hd)).masked_fill(~causal, -math.inf), -1)
        h = h + (p @ v).transpose(1, 2).reshape(h.shape) @ _w64(*L["o"], D, D).t()
        h = h + _mlp64(h, L, I, D)
    logits = _rms64(h[:, -1], d["norm"]) @ d["head"].double().t()
    return dict(tokens=None, logits=logits)


def _exact_a8w8(case, seed):
    d = _a8w8_inputs(case, seed)
    x = d["x"].double()
    rs = x.abs().amax(1, keepdim=True) / 127
    y = (torch.round(x / rs) @ d["w8"].double().t()) * rs * d["scale"].double().view(1, -1)
    return y + d["bias"].double() if d["bias"] is not None else y


_EXACT = dict(linear=_exact_linear, train=_exact_linear, decode=_exact_decode, generate=_exact_generate, a8w8=_exact_a8w8)
