"""The GEMM kernel's waits are bounded, and a lane may give up at another poll than its neighbours.  The epilogue and dequant warps do
warp-collective work behind their waits (tensor-memory loads and stores, votes), so there every wait's outcome is voted on: a warp
that went on in part would wait for the lanes that left, without a limit."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "latentq_llm_b200", "csrc")


def test_collective_roles_vote_on_every_wait():
    with open(os.path.join(CSRC, "lq_gemm_tc.cu")) as f:
        src = f.read()
    begin = src.index("} else if (warp < 6 || warp >= C::FIRST_EXTRA_EPI) {")           # epilogue, then dequant
    roles = src[begin:src.index("// split-K reduction", begin)]
    ready = re.search(r"auto stage_ready = .*?\n            \};", roles, re.S)
    assert ready and re.search(r"return warp_vote\(r\);\s*\};$", ready.group(0)), "stage_ready returns the warp's vote"
    assert len(re.findall(r"\breturn\b", ready.group(0))) == 1
    rest = roles.replace(ready.group(0), "")
    waits = [line.strip() for line in rest.splitlines() if re.search(r"\bmbar_wait(_t)?\(", line)]
    assert len(waits) >= 3
    for line in waits:
        assert re.search(r"warp_vote\(mbar_wait(_t)?\(", line), line
