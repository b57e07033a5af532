"""The division by a scale that many elements share, against torch's IEEE division: dividends within a few units in the last place of a
value where the rounded quotient changes, and random ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _near_ties(s, k, g):
    """fp32 dividends a with a / s within a few units in the last place of k + 1/2."""
    a = ((k.double() + 0.5) * s.double()).float()
    return (a.view(torch.int32) + torch.randint(-3, 4, a.shape, device="cuda", generator=g, dtype=torch.int32)).view(torch.float32)


@pytest.mark.parametrize("block", [128, 2048, 8192])
def test_optimizer_state_codes_at_the_ties_of_the_quotient(block):
    from latentq_llm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(block)
    blocks = 256
    x = torch.zeros(blocks, block, device="cuda")
    x[:, 0] = -torch.exp2(torch.rand(blocks, device="cuda", generator=g) * 80 - 40)           # the range; the maximum stays 0
    s = ops.opt8_quant(x, block)[1]
    near = _near_ties(s, torch.randint(0, 254, (blocks, block - 2), device="cuda", generator=g), g)
    rand = -x[:, :1] * torch.rand(blocks, block - 2, device="cuda", generator=g)
    x[:, 2:] = -torch.where(torch.rand(near.shape, device="cuda", generator=g) < 0.8, near, rand).minimum(-x[:, :1])
    q, s2, tmax = ops.opt8_quant(x, block)
    assert torch.equal(s, s2) and not tmax.any()
    assert torch.equal(q, torch.round(-x / s).clamp(0, 255).to(torch.uint8))


def test_int8_codes_at_the_ties_of_the_quotient():
    from latentq_llm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    rows, cols = 512, 4096
    s = torch.exp2(torch.rand(rows, 1, device="cuda", generator=g) * 60 - 30)
    s[:8, 0] = torch.tensor([2.0 ** -40, 2.0 ** 40, 1.0, 1.9999998807907104, 2.0 ** -45, 2.0 ** 50, 1.0000001192092896, 3.0])
    w = _near_ties(s, torch.randint(-127, 126, (rows, cols), device="cuda", generator=g), g)
    w[:, ::7] = s * 300 * (torch.rand(rows, cols, device="cuda", generator=g)[:, ::7] - 0.5)
    w[:, :3] = torch.tensor([0.0, 1e-30, 1e25], device="cuda")
    codes, _ = ops.a8w8_requant(w, s, ops.make_opts(codec=ops.CODEC_NONE, math_dtype=torch.float32))
    assert torch.equal(codes, torch.round(w / s).clamp(-128, 127).to(torch.int8))
