"""What the plan of a GEMM launch depends on, seen through the scratch it asks for (no GPU needed)."""
import pytest

from latentq_llm_b200 import _lib

FWD, DGRAD = _lib.GEMM_A16W4_FWD, _lib.GEMM_A16W4_DGRAD
SHAPES = [(M, N, K) for M in (65, 100, 129, 200, 300, 500) for N, K in ((1024, 2048), (512, 1024), (2048, 1024))]


def _scratch(kind):
    return [_lib.lib.lq_gemm_workspace_bytes(kind, *s) for s in SHAPES]


@pytest.fixture(autouse=True)
def _default_plan(monkeypatch):
    for k in ("LQ_GEMM_BALANCE", "LQ_GEMM_A_OPERAND", "LQ_GEMM_DGRAD_TRANSPOSE", "LQ_GEMM_NO_SKINNY", "LQ_SKINNY_SPLIT"):
        monkeypatch.delenv(k, raising=False)


@pytest.mark.parametrize("kind", [FWD, DGRAD])
def test_balance_switched_off_is_the_default_plan(monkeypatch, kind):
    default = _scratch(kind)
    assert any(default)
    monkeypatch.setenv("LQ_GEMM_BALANCE", "0")
    assert _scratch(kind) == default


def test_balanced_forward_leaves_the_grad_input_plan_alone(monkeypatch):
    default = _scratch(DGRAD)
    monkeypatch.setenv("LQ_GEMM_BALANCE", "1")
    assert _scratch(DGRAD) == default
