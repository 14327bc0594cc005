"""The protocol of the closing reduction of the 4-bit window kernel (bxq_kernels.cuh), read in its source: who adds a row block up, what
it waits for, and what is left behind when a wait runs out.  (The sums themselves are tested on the GPU.)"""
from pathlib import Path

KERNEL = (Path(__file__).resolve().parents[1] / "georefine_b200" / "csrc" / "bxq_kernels.cuh").read_text()
EPILOGUE = KERNEL[KERNEL.index("warp >= kWideWarpEpilogue) {\n    // ---"):KERNEL.index("if (MODE == kUmma && args.cluster > 1) {")]


def test_a_first_item_is_declared_when_its_cta_starts():
    """Declared with its tile it could be the last of its row block, and its CTA would add up that one and its last item's."""
    before, loop = EPILOGUE.split("for (uint32_t it = item_begin;", 1)
    assert "first_declared = atomicAdd(args.counters + item.row_block, 1u);" in before
    assert before.index("grid_dependency_wait();") < before.index("first_declared = atomicAdd(")     # (the counters may be the launch before's)
    stored = loop[loop.index("stg32(dst"):]
    assert "atomicAdd(args.counters + item.row_block, 1u << 16);" in stored and "0x10001u" not in EPILOGUE


def test_a_counter_is_cleared_only_when_all_its_parts_are_in_memory():
    """A part published after the wait for it ran out would stay counted, and a later launch add its tile too early."""
    assert KERNEL.count("args.counters[") == 1
    wait = KERNEL[KERNEL.index("bool bxq_parts_in_memory("):]
    wait = wait[:wait.index("\n}\n")]
    assert wait.index("while ((ld_acquire_gpu(") < wait.index("return false;") < wait.index("args.counters[row_block] = 0;")


def test_the_warp_that_asks_for_tiles_waits_for_them():
    """(With the wait in the epilogue, a fence and a barrier stood between a tile's arrival and its copy: short launches got slower.)"""
    assert "bxq_parts_in_memory(" not in EPILOGUE
    closing = KERNEL[KERNEL.index("// Row blocks that fell to this CTA are added up"):]
    asked = closing.index("if (warp == kWideWarpSlices && lane == 0)")
    assert asked < closing.index("bxq_parts_in_memory(") < closing.index("bulk_g2s(") and "__threadfence" not in closing
