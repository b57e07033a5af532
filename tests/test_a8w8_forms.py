"""Forms of scale, bias and clamp value that the A8W8 linear takes: the one-launch forward is for a scale and a bias of one element per
output channel and a clamp value of one element; everything else is broadcast, or refused, as the tensor operations do it.  The two
launches are stood in for by plain torch, which refuses to read past an operand."""
import pytest
import torch

from latentq_llm_b200 import quant

M, N, K = 6, 8, 128


def _acc(x8, w8):
    return x8.float() @ w8.float().t()


def _gemm_a8w8(x8, w8, row_scale=None, col_scale=None, alpha=1.0, bias=None):
    assert row_scale.shape == (M,) and col_scale is None and alpha == 1.0
    assert bias.is_contiguous() and bias.dtype == torch.bfloat16 and bias.numel() >= N, "bias read past its end"
    return (_acc(x8, w8) * row_scale[:, None] + bias.reshape(-1)[:N].float()).to(torch.bfloat16)


def _gemm_a8w8_module(x8, w8, clampv, alpha, bias, qscales):
    assert qscales.numel() == N and (bias is None or bias.numel() == N) and (clampv is None or clampv.numel() == 1), "operand read past its end"
    a = alpha if clampv is None else float(clampv.to(torch.bfloat16) / 127.)
    qs = qscales.reshape(-1)
    b = (0 * qs if bias is None else bias / qs).to(torch.bfloat16)
    return (_acc(x8, w8) * a + b.float()).to(torch.bfloat16) * qs


@pytest.fixture
def case(monkeypatch):
    monkeypatch.setattr(quant.ops, "gemm_a8w8", _gemm_a8w8)
    monkeypatch.setattr(quant.ops, "gemm_a8w8_module", _gemm_a8w8_module)
    g = torch.Generator().manual_seed(0)
    return dict(x=torch.randint(-128, 128, (M, K), generator=g, dtype=torch.int8), w=torch.randint(-128, 128, (N, K), generator=g, dtype=torch.int8),
                clampv=torch.tensor([2.5]), qs=(torch.rand(N, 1, generator=g) * 0.01 + 1e-3).to(torch.bfloat16),
                bias=torch.randn(N, generator=g).to(torch.bfloat16))


@pytest.mark.parametrize("static", [True, False])
@pytest.mark.parametrize("scale", ["channel", "one"])
@pytest.mark.parametrize("bias", ["channel", "row", "one", "none"])
def test_accepted_forms(case, static, scale, bias):
    qs = case["qs"] if scale == "channel" else case["qs"][:1]
    b = {"channel": case["bias"], "row": case["bias"][None], "one": case["bias"][:1], "none": None}[bias]
    a = 2.5 / 127. if static else float(torch.tensor(2.5).to(torch.bfloat16) / 127.)
    shift = ((0 * qs.view(-1)) if b is None else b / qs.view(-1)).to(torch.bfloat16)
    want = (_acc(case["x"], case["w"]) * a + shift.float()).to(torch.bfloat16) * qs.view(1, -1)
    assert torch.equal(quant._a8w8_forward(case["x"], 2.5 if static else case["clampv"], case["w"], qs, b), want)


@pytest.mark.parametrize("scale", ["channel", "one"])
@pytest.mark.parametrize("length", [2, N - 1])
def test_a_shorter_bias_is_refused(case, scale, length):
    with pytest.raises(RuntimeError):
        quant._a8w8_forward(case["x"], case["clampv"], case["w"], case["qs"] if scale == "channel" else case["qs"][:1], case["bias"][:length])


def test_a_clamp_value_of_two_elements_is_refused(case):
    with pytest.raises(RuntimeError):
        quant._a8w8_forward(case["x"], torch.tensor([2.5, 3.0]), case["w"], case["qs"], case["bias"])


def test_grad_input_scales_rows_only_with_a_column_of_scales(case, monkeypatch):
    """A flat scale multiplies the weight's columns or is refused, as the tensor product does it."""
    monkeypatch.setattr(quant.ops, "i8_dequant", lambda codes, row_scales=None, clampv=None: codes.to(torch.bfloat16) * row_scales.view(-1, 1))
    ctx = type("Ctx", (), dict(needs_input_grad=(True, False, False, False)))()
    w = case["w"][:, :N].contiguous()                                    # square: the flat scale broadcasts along the columns
    dy, x = torch.randn(M, N).to(torch.bfloat16), torch.randn(M, N).to(torch.bfloat16)
    for qs in (case["qs"], case["qs"].view(-1)):
        dx = quant._a8w8_backward(ctx, dy, x, w, qs, None)[0]
        quant.dict_temp.pop()
        assert torch.equal(dx, dy.mm(w.to(torch.bfloat16) * qs))
    with pytest.raises(RuntimeError):
        quant._a8w8_backward(ctx, dy, torch.randn(M, K).to(torch.bfloat16), case["w"], case["qs"].view(-1), None)
