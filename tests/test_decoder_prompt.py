"""FusedLlamaGreedyDecoder, what needs no kernel: which route a prompt takes, and that a call works with the model's weights as they are then."""
import pytest
import torch
from transformers import LlamaConfig, LlamaForCausalLM

from latentq_llm_b200.generate import FusedLlamaGreedyDecoder
from latentq_llm_b200.quant import QLinearA16W4

MODULES = ("self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj", "mlp.gate_proj", "mlp.up_proj", "mlp.down_proj")


def _int4_linear(n, k, g, cls=QLinearA16W4):
    lin = cls(k, n, bias=False)
    lin.scales.data = torch.rand(n * k // 128, 1, generator=g).to(torch.bfloat16)
    lin.zeros.data = torch.randint(0, 16, (n * k // 128, 1), generator=g).to(torch.bfloat16)
    lin.weight.set_value(torch.randint(-128, 128, (n * k // 2,), generator=g, dtype=torch.int64).to(torch.int8), [lin.scales, lin.zeros, lin.wshape])
    return lin


def _model(**cfg):
    g = torch.Generator().manual_seed(0)
    model = LlamaForCausalLM(LlamaConfig(**{**dict(hidden_size=256, intermediate_size=512, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2,
                                                   vocab_size=64, max_position_embeddings=128), **cfg})).to(torch.bfloat16)
    for layer in model.model.layers:
        for name in MODULES:
            part, leaf = name.split(".")
            old = getattr(getattr(layer, part), leaf)
            setattr(getattr(layer, part), leaf, _int4_linear(*old.weight.shape, g))
    return model


def _decoder(model):
    return FusedLlamaGreedyDecoder(model, batch=2, max_len=64)


def test_llama_prompts_go_through_the_kernels():
    for rope in (None, {"rope_type": "linear", "factor": 2.0, "rope_theta": 10000.0},
                 {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 32, "rope_theta": 10000.0}):
        assert _decoder(_model(**({"rope_parameters": rope} if rope else {})))._kernels_serve_prompts(), rope


class _OtherLinear(QLinearA16W4):
    def forward(self, x):
        return super().forward(x) * 2


def _replace(path, make):
    def change(model):
        owner = model.model.layers[1]                      # the last layer: every layer is looked at
        *parents, leaf = path.split(".")
        for name in parents:
            owner = getattr(owner, name)
        setattr(owner, leaf, make(getattr(owner, leaf)))
    return change


def _forward_of_its_own(module):
    old = module.forward
    module.forward = lambda *a, **k: old(*a, **k)


CHANGES = {
    "hook of a projection": lambda m: m.model.layers[1].mlp.up_proj.register_forward_hook(lambda *a: None),
    "hook before a layer": lambda m: m.model.layers[1].register_forward_pre_hook(lambda *a: None),
    "hook of the head": lambda m: m.lm_head.register_forward_hook(lambda *a: None),
    "hook of the model": lambda m: m.register_forward_hook(lambda *a: None),
    "forward of one object": lambda m: _forward_of_its_own(m.model.layers[1].self_attn),
    "linear of a subclass": _replace("self_attn.v_proj", lambda old: _int4_linear(*old.wshape, torch.Generator(), _OtherLinear)),
    "norm of another class": _replace("input_layernorm", lambda old: torch.nn.RMSNorm(256, dtype=torch.bfloat16)),
    "norm with another epsilon": lambda m: setattr(m.model.layers[1].post_attention_layernorm, "variance_epsilon", 1e-3),
    "other activation": _replace("mlp.act_fn", lambda old: torch.nn.GELU()),
    "scaled attention": lambda m: setattr(m.model.layers[1].self_attn, "scaling", 0.5),
    "embedding in fp32": lambda m: m.model.embed_tokens.float(),
    "head of another class": lambda m: setattr(m, "lm_head", torch.nn.Sequential(torch.nn.Linear(256, 64, bias=False))),
}


@pytest.mark.parametrize("change", CHANGES)
def test_models_that_do_something_else_run_their_prompt_themselves(change):
    model = _model()
    dec = _decoder(model)
    assert dec._kernels_serve_prompts()
    CHANGES[change](model)
    assert not dec._kernels_serve_prompts()
    if change not in ("head of another class", "linear of a subclass"):
        assert not _decoder(model)._kernels_serve_prompts()


@pytest.mark.parametrize("cfg", [{"rope_parameters": {"rope_type": "yarn", "factor": 4.0, "rope_theta": 10000.0}},
                                 {"rope_parameters": {"rope_type": "dynamic", "factor": 2.0, "rope_theta": 10000.0}},
                                 {"hidden_act": "gelu"}, {"sliding_window": 16}, {"attn_implementation": "eager"}], ids=str)
def test_configurations_that_the_kernels_do_not_compute(cfg):
    assert not _decoder(_model(**cfg))._kernels_serve_prompts()


def test_autocast_and_global_hooks_are_the_modules_business():
    dec = _decoder(_model())
    with torch.autocast("cpu", dtype=torch.bfloat16):
        assert not dec._kernels_serve_prompts()
    handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    try:
        assert not dec._kernels_serve_prompts()
    finally:
        handle.remove()
    assert dec._kernels_serve_prompts()


def _fresh_equals(dec, model):
    new = _decoder(model)
    for L, N in zip(dec.layers, new.layers):
        for name in ("qkv", "gu", "o", "down"):
            assert all(torch.equal(a, b) for a, b in zip(L[name], N[name])), name
        assert torch.equal(L["ln1"], N["ln1"]) and torch.equal(L["ln2"], N["ln2"])
    assert all(torch.equal(a, b) for a, b in zip(dec.ends, new.ends))


def test_a_call_takes_the_weights_as_they_are():
    model = _model()
    dec = _decoder(model)
    dec.graph = captured = object()
    held = [L[name][i].data_ptr() for L in dec.layers for name in ("qkv", "gu") for i in range(3)]
    g = torch.Generator().manual_seed(1)
    for li, layer in enumerate(model.model.layers):        # written in place: the captured step sees these where it reads them
        for lin in (layer.self_attn.k_proj, layer.self_attn.o_proj, layer.mlp.up_proj):
            lin.weight.data.copy_(torch.randint(-128, 128, lin.weight.data.shape, generator=g, dtype=torch.int64))
            lin.scales.data.add_(1)
        layer.input_layernorm.weight.data.mul_(0.5)
    dec._take_weights()
    _fresh_equals(dec, model)
    assert dec.graph is captured and held == [L[name][i].data_ptr() for L in dec.layers for name in ("qkv", "gu") for i in range(3)]

    q, v = model.model.layers[0].self_attn.q_proj, model.model.layers[1].self_attn.v_proj
    q.weight.set_value(q.weight.data.flip(0), [q.scales + 1, q.zeros, q.wshape])       # elsewhere, but copied
    v.weight.data = v.weight.data.flip(0)
    dec._take_weights()
    _fresh_equals(dec, model)
    assert dec.graph is captured and held == [L[name][i].data_ptr() for L in dec.layers for name in ("qkv", "gu") for i in range(3)]

    for move in (lambda: setattr(model.model.layers[1].mlp.down_proj.weight, "data", model.model.layers[1].mlp.down_proj.weight.data.flip(0)),
                 lambda: setattr(model.model.norm.weight, "data", model.model.norm.weight.data * 2),
                 lambda: setattr(model.lm_head.weight, "data", model.lm_head.weight.data * 2)):
        dec.graph = captured
        move()                                             # read where the model has them: the captured step reads the old place
        dec._take_weights()
        _fresh_equals(dec, model)
        assert dec.graph is None


def test_rows_that_are_not_whole_words_are_copied_too():
    """Codes at an odd address (a slice of a checkpoint's buffer): copied byte by byte."""
    model = _model()
    w = model.model.layers[0].self_attn.k_proj.weight
    dec = _decoder(model)
    odd = torch.empty(w.data.numel() + 1, dtype=torch.int8)[1:]
    w.data = odd.copy_(w.data.flip(0))
    dec._take_weights()
    _fresh_equals(dec, model)
    w.data.add_(1)
    dec._take_weights()
    _fresh_equals(dec, model)


def test_a_prompt_sees_the_present_weights_and_route(monkeypatch):
    """The order inside `generate`: the route and the weights of the call before its prompt."""
    model = _model()
    dec = _decoder(model)
    seen = []
    monkeypatch.setattr(dec, "_prompt_step", lambda prompt: (seen.append(("kernels", dec.layers[0]["qkv"][0][0].item())), torch.zeros(2, 64))[1])
    prompt = torch.zeros((2, 5), dtype=torch.long)
    for value in (3, 4):
        model.model.layers[0].self_attn.q_proj.weight.data.fill_(value)
        dec.generate(prompt, 1, use_graph=False)
    assert seen == [("kernels", 3), ("kernels", 4)]
    model.model.rotary_emb.inv_freq.mul_(0.5)
    dec.generate(prompt, 1, use_graph=False)
    assert torch.equal(dec.inv_freq, model.model.rotary_emb.inv_freq.float())
    fired = []
    model.model.embed_tokens.register_forward_hook(lambda *a: (fired.append(1), 1 / 0))
    with pytest.raises(ZeroDivisionError):                 # through the modules, whose kernels need a GPU: as far as the first hook
        dec.generate(prompt, 1, use_graph=False)
    assert fired and len(seen) == 3
