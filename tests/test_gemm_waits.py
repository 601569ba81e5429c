"""A warp of the large-batch GEMM whose wait gave up issues nothing more: read from the source, because a wait runs out on a GPU only
where something is already wrong."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "candle_b200", "csrc", "expert_gemm.cu")
ROLES = ("WARP_LOAD", "WARP_D8", "WARP_TMA", "WARP_MMA")


def _role(name):
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    body = text[text.index("expert_gemm_kernel(const"):]
    body = body[body.index(f"if (warp == {name}) {{"):]
    ends = [body.index(f"else if (warp == {r}) {{") for r in ROLES if f"else if (warp == {r}) {{" in body[10:]]
    return body[:min(ends)] if ends else body[:body.index("tc5_fence_before_sync();\n    __syncthreads();")]


@pytest.mark.parametrize("role", ["WARP_LOAD", "WARP_TMA"])
def test_copying_warps_issue_nothing_after_a_wait_that_gave_up(role):
    body = _role(role)
    waits = [m.start() for m in re.finditer(r"mbar_wait_tight\(", body)]
    assert waits
    for at in waits:
        assert re.search(r"\bok = (ok && )?$", body[:at]), body[max(0, at - 120):at + 40]
    elected = list(re.finditer(r"if \(elect_one\(\)([^{]*)\) \{", body))
    assert elected
    for m in elected:
        # in the condition itself, or by leaving the loop on the whole warp's answer just before
        left = re.search(r"if \(!\(ok = __all_sync\(0xffffffffu, ok\)\)\) break;\s*$", body[:m.start()])
        assert "&& ok" in m.group(1) or left, body[max(0, m.start() - 160):m.end()]


def test_mma_warp_issues_nothing_after_a_wait_that_gave_up():
    body = _role("WARP_MMA")
    # one place waits, with the whole warp's answer ...
    assert len(re.findall(r"mbar_wait_tight\(", body)) == 1
    assert re.search(r"const auto wait = [^;]*return \(bool\)__all_sync\(0xffffffffu, known \|\| mbar_wait_tight\(", body)
    uses = list(re.finditer(r"\bwait\((?!known)", body))
    assert len(uses) == 2
    for m in uses:  # ... that leaves the block ...
        assert body[:m.start()].endswith("!") and re.match(r"[^;]*\)\) return false;", body[m.start():]), body[m.start():m.start() + 120]
    blocks = list(re.finditer(r"\bblock\(std::integral_constant", body))
    assert len(blocks) == 2
    for m in blocks:  # ... and the tile loop
        assert re.match(r"if \(!block\(std::integral_constant<int, [01]>\{\}\)\) goto mma_end;", body[m.start() - 5:]), body[m.start() - 5:m.start() + 80]
    assert body[body.index("mma_end:"):].strip() in ("mma_end:;\n    }", "mma_end:;")
