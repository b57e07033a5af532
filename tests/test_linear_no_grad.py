"""The linear's no-gradient route: calls the autograd function's forward directly, and leaves every case that autograd has a say in
(gradients on, forward-mode duals, functorch transforms, traces) to `apply`."""
import ctypes

import torch
import torch.autograd.forward_ad as fwd

from latentq_llm_b200 import quant


class _Double(torch.autograd.Function):
    applied = 0

    @staticmethod
    def forward(x):
        return 2 * x

    @staticmethod
    def setup_context(ctx, inputs, output):
        _Double.applied += 1

    @staticmethod
    def backward(ctx, g):
        return 2 * g


def _went_through_apply(x):
    before = _Double.applied
    try:
        quant._apply(_Double, x)
    except Exception:           # apply refuses what has no rule: that is its answer, not the direct call's
        return True
    return _Double.applied != before


def test_direct_call_only_where_autograd_has_no_say():
    x = torch.randn(3)
    with torch.no_grad():
        assert not _went_through_apply(x)
        assert torch.equal(quant._apply(_Double, x), 2 * x)
        with fwd.dual_level():
            assert _went_through_apply(fwd.make_dual(x, torch.ones_like(x)))
        seen = []

        def under_vmap(v):
            seen.append(_went_through_apply(v))
            return v
        torch.func.vmap(under_vmap)(torch.randn(2, 3))
        assert seen == [True]
    assert _went_through_apply(x)
    with torch.inference_mode():
        assert torch.equal(quant._apply(_Double, x), 2 * x)


class _Foreign(torch.autograd.Function):
    """Writes its output behind torch's back, as the kernels do."""

    @staticmethod
    def forward(x):
        y = torch.empty_like(x)
        ctypes.memmove(y.data_ptr(), x.data_ptr(), x.numel() * x.element_size())
        return y

    @staticmethod
    def setup_context(ctx, inputs, output):
        pass


def test_a_trace_records_the_function():
    with torch.no_grad():
        traced = torch.jit.trace(lambda v: quant._apply(_Foreign, v), torch.randn(64), check_trace=False)
        assert "Foreign" in str(traced.graph)
        for i in range(4):
            x = torch.randn(64)
            assert torch.equal(traced(x), x)
