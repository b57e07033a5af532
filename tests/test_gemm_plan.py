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


# (tokens, out, in) and whether the grad-input goes through the transposed copy: measured 7 % and more apart (us, copy / stored), and the
# kernel on the stored weight needs no scratch of its own there
@pytest.mark.parametrize("M,N,K,copy", [
    (2048, 4096, 11008, True),       # 144 / 158
    (2048, 8192, 2048, True),        # 58 / 73
    (1792, 4096, 4096, True),        # 58 / 68
    (4096, 2048, 2048, True),        # 35 / 40
    (1791, 4096, 4096, False),       # below the range
    (2048, 8192, 1024, False),       # 53 / 48: 64 tiles of 256 tokens on 148 SMs
    (1792, 512, 8192, False),        # 29 / 26
    (1920, 2048, 5632, False),       # 51 / 44
    (2560, 2048, 2048, False),       # 33 / 31: a second wave of 12 tiles
])
def test_route_of_the_grad_input(M, N, K, copy):
    need = _lib.lib.lq_gemm_workspace_bytes(DGRAD, M, N, K)
    assert need == (N * K // 2 + N * K // 128 * 4 if copy else 0)


def test_split_of_a_forward_without_two_block_stages():
    """Nine groups per row: 18 k-blocks in four splits, not three of an even number."""
    assert _lib.lib.lq_gemm_workspace_bytes(FWD, 8, 1088, 1152) == 4 * 8 * 1088 * 4


def test_tiles_of_a_forward_without_staged_group_parameters():
    """31 groups per row, 128 tokens: one 128-token tile in four splits, not four 32-token tiles."""
    assert _lib.lib.lq_gemm_workspace_bytes(FWD, 128, 4096, 3968) == 4 * 128 * 4096 * 4
