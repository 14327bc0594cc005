"""Memory that ordinary stores write and bulk copies then read or overwrite: the two go through different proxies, and only a
proxy fence between them orders them.  (A missing one shows as stale data now and then, if at all: read here, not run.)"""
from pathlib import Path

KERNEL = (Path(__file__).resolve().parents[1] / "georefine_b200" / "csrc" / "bxq_kernels.cuh").read_text()


def _in_order(text, *parts):
    at = 0
    for part in parts:
        at = text.find(part, at)
        assert at >= 0, part
        at += len(part)


def test_partial_tiles_are_fenced_before_they_are_counted():
    epilogue = KERNEL[KERNEL.index("warp >= kWideWarpEpilogue) {\n    // ---"):]
    _in_order(epilogue, "stg32(dst", "fence_proxy_async_all();", "__threadfence();", "1u << 16")     # stored tile by tile
    _in_order(epilogue, "drain_to_smem(n_item, 0, smem);", "fence_proxy_async_smem();", "bulk_s2g(")    # sent from shared memory


def test_slices_are_asked_for_after_a_fence():
    closing = KERNEL[KERNEL.index("// Row blocks that fell to this CTA are added up"):]
    _in_order(closing, "bar_final, 0)", "bxq_parts_in_memory(", "fence_proxy_async_all();", "bulk_g2s(")
