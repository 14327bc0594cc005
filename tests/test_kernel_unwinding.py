"""How a fused kernel unwinds after a wait that ran out: no warp may be left in a wait without a limit.  Each lane times its own wait,
so where a barrier completes as the limit runs out, the lanes of a warp, or the warps of a role, would part: those that go on to
something all of them have to reach would wait there for good.  (What happens then cannot be run; read here.)"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "georefine_b200" / "csrc"
KERNELS = sorted(CSRC.glob("bx?_kernels.cuh"))


def _without(text, opening):
    """The text without the blocks that `opening` (a pattern ending at a brace) begins."""
    while (m := re.search(opening, text)):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        text = text[:m.start()] + text[at:]
    return text


@pytest.mark.parametrize("path", KERNELS, ids=lambda p: p.name)
def test_no_meeting_of_warps_without_a_limit(path):
    text = path.read_text()
    assert "bar.sync" not in text and "named_barrier" not in text
    # whole CTAs and clusters meet at the set-up and once every role is through, on every path
    roles = text[text.index("if (warp < kDecoderWarps) {\n    // ---"):]
    for meeting in re.findall(r"^( *).*\b(__syncthreads|cluster_sync)\(\)", roles, re.M):
        assert len(meeting[0]) <= 4


@pytest.mark.parametrize("path", KERNELS, ids=lambda p: p.name)
def test_a_warp_has_one_verdict_on_a_wait(path):
    text = path.read_text()
    kernel = text[text.index("_kernel(const BxrArgs args"):]
    single = _without(kernel, r"if \([^;{}]*lane == 0[^;{}]*\) \{")      # blocks of one lane have nobody to part from
    lines = [line.strip() for line in single.splitlines()]
    for i, line in enumerate(lines):
        if not re.search(r"\bctx\.wait\(", line):
            continue
        # the lane goes on, whatever its verdict, to a vote that decides for the warp before anything else can end the loop
        assert re.match(r"(bool )?ok = ctx\.wait\(", line), line
        rest = lines[i + 1:]
        vote = next(n for n, after in enumerate(rest) if "live = __all_sync(0xFFFFFFFFu, ok)" in after)
        assert not any(re.search(r"\b(break|return|continue)\b", after.split("//")[0]) for after in rest[:vote])
        assert rest[vote + 1].startswith("if (!live) break;")
    helpers = (CSRC / "bxr_kernels.cuh").read_text()
    assert "return __all_sync(0xFFFFFFFFu, !aborted() && wait(bar, parity));" in helpers     # go_warp
    assert "return wait_warp(bar, met++ & 1);" in helpers                                    # meet
