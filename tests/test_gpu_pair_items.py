"""Pair launches with many items a CTA, inside a captured graph, and on two streams at a time, bit for bit against passes of at most
64 rows (needs a B200)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# rows x columns, workers, items of each worker: split first / whole / split last items, and ten whole ones beside a split one (an
# accumulator's place used again and again)
SHAPES = [((2560, 1152), 6, [4, 4, 4, 4, 4, 4]), ((4864, 1152), 4, [10, 10, 10, 10]), ((2440, 1096), 6, [4, 4, 4, 4, 4, 4])]
_cache = {}


def _weight(shape, workers):
    from georefine_b200.resident import ResidentWeight

    if (shape, workers) not in _cache:
        _cache.clear()
        w = (torch.randn(*shape, generator=torch.Generator().manual_seed(sum(shape))) * 0.02).to(torch.bfloat16)
        _cache[shape, workers] = ResidentWeight.from_words(w.view(torch.int16).numpy().view(np.uint16), torch.device("cuda:0"), workers=workers, layout="window4")
    return _cache[shape, workers]


def _narrow(r, x):
    y = torch.empty(x.shape[0], r.N, dtype=torch.bfloat16, device="cuda")
    for lo in range(0, x.shape[0], 64):
        r.gemm(x[lo:lo + 64], y[lo:lo + 64])
    return y


def _rows(m, k, seed):
    return torch.randn(m, k, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).cuda()


@pytest.mark.parametrize("shape,workers,items", SHAPES)
@pytest.mark.parametrize("m", [129, 192, 200, 256, 300, 384, 500])
def test_many_items_a_cta(shape, workers, items, m):
    r = _weight(shape, workers)
    h = r.header
    at = h.worker_items_at
    assert h.paired == 1 and np.diff(r.image[at:at + 4 * (workers + 1)].cpu().numpy().view(np.uint32)).tolist() == items
    x = _rows(m, shape[1], m)
    want, y = _narrow(r, x), torch.full((m, shape[0]), float("nan"), dtype=torch.bfloat16, device="cuda")
    for _ in range(3):
        r.gemm(x, y.fill_(float("nan")))
        assert torch.equal(y, want)
    assert r.check_status() == 0


@pytest.mark.parametrize("lent", [True, False])
def test_inside_a_graph(lent):
    r = _weight(*SHAPES[0][:2])
    r.reserve(128)
    x, y = _rows(300, 1152, 1), torch.empty(300, 2560, dtype=torch.bfloat16, device="cuda")
    scratch = torch.empty(r.wide_scratch_bytes, dtype=torch.uint8, device="cuda") if lent else None
    r.gemm(x, y, scratch=scratch)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(3):
            r.gemm(x, y, scratch=scratch)
    for seed in (2, 3):
        x.copy_(_rows(300, 1152, seed))
        want = _narrow(r, x)
        y.fill_(float("nan"))
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
    assert r.check_status() == 0
    del graph


def test_on_two_streams_at_a_time():
    first = _weight(*SHAPES[0][:2])
    weights = [first, first.clone()]          # (a workspace belongs to one stream at a time)
    streams = [torch.cuda.Stream() for _ in weights]
    xs = [_rows(384, 1152, 5), _rows(256, 1152, 6)]
    wants = [_narrow(first, x) for x in xs]
    lent = [torch.empty(first.wide_scratch_bytes, dtype=torch.uint8, device="cuda") for _ in weights]
    ys = [[torch.full_like(want, float("nan")) for _ in range(8)] for want in wants]
    torch.cuda.synchronize()
    for i in range(8):
        for w, stream, x, y, scratch in zip(weights, streams, xs, ys, lent):
            with torch.cuda.stream(stream):
                w.gemm(x, y[i], scratch=scratch)
    torch.cuda.synchronize()
    for w, y, want in zip(weights, ys, wants):
        assert w.check_status() == 0 and all(torch.equal(got, want) for got in y)
