"""Batches above 128 rows by pairs of CTAs against passes of at most 128 rows, bit for bit, and against a 64-bit product (needs a B200)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# rows x columns, workers: shares of one and of several row blocks, ragged edges, an unaligned y (500 rows), clusters of 2, 3 and 4
# parts a row block (4, 6 and 8 CTAs), one CTA per SM with first, whole and last items
SHAPES = [((512, 2048), 4), ((512, 2048), 6), ((500, 2040), 6), ((1280, 1160), 8), ((512, 2048), 8), ((508, 2048), 12), ((512, 2048), 16),
          ((5120, 4096), 148)]
_cache = {}


def _weight(shape, workers):
    from georefine_b200.resident import ResidentWeight

    if (shape, workers) not in _cache:
        _cache.clear()
        w = (torch.randn(*shape, generator=torch.Generator().manual_seed(sum(shape))) * 0.02).to(torch.bfloat16)
        r = ResidentWeight.from_words(w.view(torch.int16).numpy().view(np.uint16), torch.device("cuda:0"), workers=workers, layout="window4")
        _cache[shape, workers] = r, w.cuda().double()
    return _cache[shape, workers]


@pytest.mark.parametrize("shape,workers", SHAPES)
@pytest.mark.parametrize("m", [129, 192, 193, 256, 257, 384, 385, 520])
@pytest.mark.parametrize("biased", [False, True])
def test_rows_equal_those_of_narrow_passes(shape, workers, m, biased):
    n, k = shape
    r, w = _weight(shape, workers)
    g = torch.Generator().manual_seed(n + m)
    x = torch.randn(m, (k + 7) // 8 * 8, generator=g).to(torch.bfloat16).cuda()[:, :k]
    bias = torch.randn(n, generator=g).to(torch.bfloat16).cuda() if biased else None
    want, y, again = (torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(3))
    for lo in range(0, m, 64):
        r.gemm(x[lo:lo + 64], want[lo:lo + 64], bias)
    r.gemm(x, y, bias)
    r.gemm(x, again, bias)                                   # counters left at zero, scratch reused
    assert r.check_status() == 0
    assert torch.equal(y, want) and torch.equal(again, want)
    exact = x.double() @ w.T + (0 if bias is None else bias.double())
    # one BF16 rounding (2^-9 relative), and the FP32 sum's error, far below 2^-14 of the norm product
    bound = exact.abs() * 2.0**-8 + 2.0**-14 * x.double().norm(dim=1, keepdim=True) * w.norm(dim=1)
    assert bool(((y.double() - exact).abs() <= bound).all())


def test_passes_are_as_wide_as_the_scratch_allows():
    """Lent partial tiles for 384, 256, 192 and 128 rows and for one row less than each: the same bits."""
    r, _ = _weight((1280, 1160), 8)
    assert r.header.paired == 1
    row = int(r.header.partial_slots) * 512
    assert r.wide_scratch_bytes == 384 * row
    x = torch.randn(500, 1160, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    want, y = torch.empty(500, 1280, dtype=torch.bfloat16, device="cuda"), torch.empty(500, 1280, dtype=torch.bfloat16, device="cuda")
    for lo in range(0, 500, 64):
        r.gemm(x[lo:lo + 64], want[lo:lo + 64])
    for rows in (384, 383, 256, 255, 192, 191, 128):
        lent = torch.full((rows * row,), 255, dtype=torch.uint8, device="cuda")
        r.gemm(x, y.fill_(float("nan")), scratch=lent)
        assert torch.equal(y, want), rows
    assert r.check_status() == 0
