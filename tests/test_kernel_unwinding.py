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
    assert "ctx.wait(" not in single
    # a wait without a verdict: nobody leaves after it, so nobody parts
    for line in re.findall(r".*wait_or_go_on.*", single):
        assert re.match(r" +ctx\.wait_or_go_on\(.*\);( +//.*)?$", line)
    helpers = (CSRC / "bxr_kernels.cuh").read_text()
    assert "return __all_sync(0xFFFFFFFFu, !aborted() && wait(bar, parity));" in helpers     # go_warp
    assert "return wait_warp(bar, met++ & 1);" in helpers                                    # meet


@pytest.mark.parametrize("path", KERNELS, ids=lambda p: p.name)
def test_a_cta_that_gives_up_outlives_its_copies(path):
    """Decoders that no longer leave at the limit must not take the CTA to its end while its copies and multiplies are under way."""
    helpers = (CSRC / "bxr_kernels.cuh").read_text()
    wait = helpers[helpers.index("void wait_or_abort("):]
    wait = wait[:wait.index("\n}\n")]
    assert re.search(r"if \(aborted && [^;]*> kLingerNs\) return;", wait) and wait.count("return;") == 2     # (the other: the phase is complete)
    text = path.read_text()
    # blobs, and activation tiles that have barriers of their own, are waited for (an entropy-coded image's tiles share the operand stages')
    waited = [bar for bar in ("bar_in_full", "bar_x_full") if f"mbar_wait({bar} + 8 * (u %" in text]
    assert waited == (["bar_in_full"] if path.name == "bxr_kernels.cuh" else ["bar_in_full", "bar_x_full"])
