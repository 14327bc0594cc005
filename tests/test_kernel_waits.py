"""Waits of warps that act together: the bounded wait of each lane may end differently, so a warp that elects a lane after it
needs one verdict for all of them.  (What happens without cannot be run: the lanes that go on wait for those that left.)"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "georefine_b200" / "csrc"


def roles(text):
    """The branches of a kernel's role dispatch (an `else if` on the warp at the kernel's outermost indentation)."""
    return re.split(r"\n  \} else if \(|\n  if \(warp|\n  \}\n", text)


def test_a_role_that_elects_a_lane_waits_as_one_warp():
    electing = [(p.name, role) for p in sorted(CSRC.glob("*_kernels.cuh")) for role in roles(p.read_text()) if "elect_one()" in role]
    assert electing
    for name, role in electing:
        waits = [line.strip() for line in role.splitlines() if re.search(r"\bwait(_warp)?\(", line)]
        assert waits
        for line in waits:
            assert "__all_sync(0xFFFFFFFFu" in line or "ctx.wait_warp(" in line, (name, line)
    assert "return __all_sync(0xFFFFFFFFu, wait(bar, parity));" in (CSRC / "bxr_kernels.cuh").read_text()
