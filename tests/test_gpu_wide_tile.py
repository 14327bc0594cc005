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
    """Inside a capture as outside: the weight's own scratch stays what 128 rows need, and the bits are the same."""
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
    r.gemm(x, want)
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


def _weight(n, k, workers, max_m=128):
    from georefine_b200.resident import ResidentWeight

    w = (torch.randn(n, k, generator=torch.Generator().manual_seed(n)) * 0.02).to(torch.bfloat16)
    r = ResidentWeight.from_words(w.view(torch.int16).numpy().view(np.uint16), torch.device("cuda:0"), layout="window4", workers=workers, max_m=max_m)
    return r, lambda m: torch.randn(m, k, generator=torch.Generator().manual_seed(m)).to(torch.bfloat16).cuda()


@pytest.mark.parametrize("entry", ["gemm", "linear"])
def test_graphs_keep_their_scratch_whatever_is_multiplied_afterwards(entry):
    """Graphs captured below and above 128 rows, on a weight whose scratch has to grow in between, replayed at the end;
    eager calls between a capture and its first replay."""
    r, rows = _weight(3000, 1152, 37, max_m=8)               # 37 workers: no clusters, row blocks shared by CTAs
    assert r.wide_scratch_bytes > 0
    sizes = (8, 100, 400) if entry == "linear" else (8, 400)
    full, _ = _weight(3000, 1152, 37)
    want = {m: torch.empty(m, 3000, dtype=torch.bfloat16, device="cuda") for m in (8, 100, 400)}
    x = {m: rows(m) for m in want}
    for m in want:
        for lo in range(0, m, 128):
            full.gemm(x[m][lo:lo + 128], want[m][lo:lo + 128])
    graphs, first = {}, r.workspace
    out = {m: torch.full_like(want[m], float("nan")) for m in want}
    for m in sizes:
        if entry == "gemm" and m > 8:
            r.reserve(128)
        graphs[m] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graphs[m]):
            if entry == "linear":
                r.linear(x[m], out=out[m])
            else:
                r.gemm(x[m], out[m])
    for m in (8, 100, 400, 100, 8):                          # before any replay
        assert torch.equal(r.linear(x[m]), want[m]), m
    assert first.data_ptr() in [ws.data_ptr() for ws in (r.workspace, *r._outgrown)]
    for _ in range(2):
        for m in sizes:
            out[m].fill_(float("nan"))
            graphs[m].replay()
            assert torch.equal(out[m], want[m]), m
    assert r.check_status() == 0


def test_wide_batches_leave_no_memory_behind(monkeypatch):
    import gc

    r, rows = _weight(5000, 1152, 148)
    x, want = rows(400), torch.empty(400, 5000, dtype=torch.bfloat16, device="cuda")
    y = torch.empty_like(want)
    for lo in range(0, 400, 128):
        r.gemm(x[lo:lo + 128], want[lo:lo + 128])
    gc.collect()
    held, said = torch.cuda.memory_allocated(), r.resident_bytes
    r.gemm(x, y)
    assert torch.equal(y, want)
    assert torch.cuda.memory_allocated() == held and r.resident_bytes == said == r.bytes + r.workspace.numel() + 4
    lent = torch.empty(r.wide_scratch_bytes, dtype=torch.uint8, device="cuda").fill_(255)     # contents of no account
    r.gemm(x, y.fill_(float("nan")), scratch=lent)
    assert torch.equal(y, want)
    r.gemm(x, y.fill_(float("nan")), scratch=lent[:-256])    # too little: passes of 128 rows
    assert torch.equal(y, want)

    empty = torch.empty

    def none_left(*size, **kw):
        if kw.get("dtype") is torch.uint8:
            raise torch.cuda.OutOfMemoryError("no memory left")
        return empty(*size, **kw)

    monkeypatch.setattr(torch, "empty", none_left)
    r.gemm(x, y.fill_(float("nan")))
    assert torch.equal(y, want) and r.check_status() == 0


def test_a_long_prompt_leaves_no_memory_behind():
    from georefine_b200 import serve

    dev = torch.device("cuda:0")
    cfg = serve.DecoderConfig(hidden=640, layers=2, heads=10, kv_heads=2, ffn=1792, vocab=1000)
    weights = serve.DecoderWeights.synthetic(cfg, dev, seed=5)
    d = serve.BatchDecoder(weights, max_rows=128, max_slots=2, max_context=1024, device=dev)
    b = serve.Batcher(d)
    said = sum(w.resident_bytes for w in weights.linears())
    b.admit([1, 2, 3])                                       # (libraries loaded)
    held = torch.cuda.memory_allocated()
    b.admit([i % 1000 for i in range(900)])
    assert torch.cuda.memory_allocated() == held and sum(w.resident_bytes for w in weights.linears()) == said


def test_more_rows_than_a_pass_takes_are_refused():
    from georefine_b200 import serve

    dev = torch.device("cuda:0")
    cfg = serve.DecoderConfig(hidden=640, layers=1, heads=10, kv_heads=2, ffn=1792, vocab=1000)
    d = serve.BatchDecoder(serve.DecoderWeights.synthetic(cfg, dev, seed=5), max_rows=128, max_slots=2, max_context=1024, device=dev)
    before = d.tokens.clone(), d.row_seq.clone(), d.row_pos.clone()
    for put, n in ((d.set_rows, 129), (d.queue_rows, d.prompt_rows), (d.absorb, d.prompt_rows + 1)):
        with pytest.raises(ValueError):
            put([0] * n, range(n), [1] * n)
    assert all(torch.equal(a, b) for a, b in zip(before, (d.tokens, d.row_seq, d.row_pos)))
    d.set_rows([0] * 128, range(128), [1] * 128)
    assert d.row_pos[:128].tolist() == list(range(128))


def test_rows_reach_the_device_in_order_without_allocating():
    """Passes queued far ahead of the device, of sizes never seen before: every one finds its own rows."""
    from georefine_b200 import serve

    dev = torch.device("cuda:0")
    cfg = serve.DecoderConfig(hidden=640, layers=1, heads=10, kv_heads=2, ffn=1792, vocab=1000)
    d = serve.BatchDecoder(serve.DecoderWeights.synthetic(cfg, dev, seed=5), max_rows=128, max_slots=2, max_context=1024, device=dev)
    pinned = torch.cuda.host_memory_stats()["num_host_alloc"]
    sizes, seen = [1, 2, 3, 7, 128, 64, 5, 33, 127, 1, 100, 17], []
    torch.cuda._sleep(20_000_000)                            # some 10 ms of work before them
    for i, n in enumerate(sizes):
        d.queue_rows([i % 2] * n, range(i, i + n), [100 * i + j for j in range(n)])
        seen.append((d.row_seq[:n].clone(), d.row_pos[:n].clone(), d.tokens[:n].clone()))
    for i, (n, (seq, pos, tok)) in enumerate(zip(sizes, seen)):
        assert seq.tolist() == [i % 2] * n and pos.tolist() == list(range(i, i + n)) and tok.tolist() == [100 * i + j for j in range(n)]
    d.set_rows([1] * 50, range(50), [9] * 50)
    d.run("ar", 50)
    for _ in range(3):
        d.set_rows([1] * 51, range(51), [9] * 51)
        d.run("ar", 51)
    assert torch.cuda.host_memory_stats()["num_host_alloc"] == pinned
