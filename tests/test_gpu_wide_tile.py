"""Batches above 128 rows: the 192-column tile of the 4-bit window kernel against the 128-column one, bit for bit (needs a B200)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# rows x columns, workers: one row block, ragged edges, row blocks cut by several CTAs, clusters of 2 and 5, one CTA per
# SM with several items each (first, whole and last ones), an unaligned y
SHAPES = [((100, 136), 1), ((777, 1032), 5), ((300, 2056), 7), ((256, 1024), 4), ((384, 2560), 15), ((5000, 1152), 148), ((1025, 640), 20)]


@pytest.mark.parametrize("shape,workers", SHAPES)
@pytest.mark.parametrize("m", [129, 160, 192, 193, 257, 384, 449])
def test_rows_equal_those_of_narrow_passes(shape, workers, m):
    from georefine_b200.resident import ResidentWeight

    n, k = shape
    g = torch.Generator().manual_seed(n + m)
    w = (torch.randn(n, k, generator=g) * 0.02).to(torch.bfloat16)
    r = ResidentWeight.from_words(w.view(torch.int16).numpy().view(np.uint16), torch.device("cuda:0"), workers=workers, layout="window4")
    x = torch.randn(m, k, generator=g).to(torch.bfloat16).cuda()
    bias = torch.randn(n, generator=g).to(torch.bfloat16).cuda()
    want, y = (torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    for lo in range(0, m, 128):
        r.gemm(x[lo:lo + 128], want[lo:lo + 128], bias)
    r.gemm(x, y, bias)
    again = torch.full_like(y, float("nan"))
    r.gemm(x, again, bias)                                   # counters left at zero, scratch reused
    assert r.check_status() == 0
    assert torch.equal(y, want) and torch.equal(again, want)
    exact = x.double() @ w.cuda().double().T + bias.double()
    # one BF16 rounding (2^-9 relative), and the FP32 sum's error, far below 2^-14 of the norm product
    bound = exact.abs() * 2.0**-8 + 2.0**-14 * x.double().norm(dim=1, keepdim=True) * w.cuda().double().norm(dim=1)
    assert bool(((y.double() - exact).abs() <= bound).all())


def test_scratch_of_128_rows_still_serves_any_batch():
    """Inside a capture nothing is allocated: the batch runs in passes of 128 rows, with the same bits."""
    from georefine_b200.resident import ResidentWeight

    g = torch.Generator().manual_seed(3)
    w = (torch.randn(3000, 1152, generator=g) * 0.02).to(torch.bfloat16)
    r = ResidentWeight.from_words(w.view(torch.int16).numpy().view(np.uint16), torch.device("cuda:0"), layout="window4")
    x = torch.randn(400, 1152, generator=g).to(torch.bfloat16).cuda()
    y, want = torch.empty(400, 3000, dtype=torch.bfloat16, device="cuda"), torch.empty(400, 3000, dtype=torch.bfloat16, device="cuda")
    r.gemm(x[:8], y[:8])                                     # (kernels loaded outside the capture)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        r.gemm(x, y)
    assert r.max_m == 128
    r.gemm(x, want)                                          # wide scratch from here on; the graph keeps its own
    assert r.max_m == 400
    graph.replay()
    assert r.check_status() == 0 and torch.equal(y, want)


@pytest.mark.parametrize("length", [128, 129, 256, 257, 513, 640, 1000])
def test_prompt_in_wide_chunks_equals_chunks_of_a_step(length):
    from georefine_b200 import serve

    dev = torch.device("cuda:0")
    cfg = serve.DecoderConfig(hidden=640, layers=2, heads=10, kv_heads=2, ffn=1792, vocab=1000)
    weights = serve.DecoderWeights.synthetic(cfg, dev, seed=5)
    ids = torch.randint(0, cfg.vocab, (length,), generator=torch.Generator().manual_seed(length)).tolist()
    got = []
    for wide in (False, True):
        d = serve.BatchDecoder(weights, max_rows=128, max_slots=2, max_context=1024, device=dev)
        assert d.prompt_rows == serve.PROMPT_ROWS
        b = serve.Batcher(d)
        if not wide:
            b._absorb = None
        slot = b.admit(ids)
        tokens = list(b.active[slot]["tokens"]) + [b.step()[slot] for _ in range(3)]
        got.append((tokens, d.kv.clone(), d.logits[:1].clone()))
    assert got[0][0] == got[1][0] and torch.equal(got[0][1][:, :, :-1], got[1][1][:, :, :-1]) and torch.equal(got[0][2], got[1][2])
