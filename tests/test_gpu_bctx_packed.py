"""The shared-memory kernel for indexed decoding (csrc/bctx_packed.cuh) at the edges of its range, bit for bit (needs a B200)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = [((16, 16), 128), ((3, 129), 16), ((257, 272), 64), ((300, 1000), 128), ((97, 4111), 1024), ((64, 4096), 48), ((7, 24576), 128), ((333, 1024), 256),
         ((5, 24577), 128), ((4, 15), 128)]     # the last two: one column too many, one too few for the kernel


@pytest.mark.parametrize("shape,stride", CASES)
@pytest.mark.parametrize("coarse", [False, True])     # True: three mantissa bits are zero, so that coded residuals (mode 128) win
@pytest.mark.parametrize("classes", [(16, 4), (1, 1), (64, 16)])
def test_packed_decode_and_row_gather_are_exact(orc, shape, stride, classes, coarse):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from georefine_b200 import codec
    from georefine_b200.gpu import CudaContextTensor

    words = orc.synthetic_weight_words(*shape, 3)
    words[0, :5] = (0, 0x8000, 0x7F80, 1, 0xFFFF)             # far-off symbols: rare entries at the ends of the tables
    if coarse:
        words &= 0xFFF8
    t = CudaContextTensor(codec.encode(words, row_classes=classes[0], col_classes=classes[1]), stride=stride, walk_stride=stride,
                          device="cuda:0", fused=False)
    assert not coarse or words.size < 20000 or t.mode == 128
    if t.mode != 1:
        assert (t._packed is not None) == (stride % 16 == 0 and 16 <= shape[1] <= 24576 and
                                           (shape[1] % stride == 0 or classes != (64, 16)))
    for check in (True, False):
        assert np.array_equal(t.decode(check=check).view(torch.uint16).cpu().numpy(), words)
    ids = torch.tensor([[shape[0] - 1, 0], [shape[0] // 2, 0]])
    assert np.array_equal(t.gather_rows(ids).view(torch.uint16).cpu().numpy(), words[ids.numpy()])
    assert int(t.error.item()) == 0
    for wrong in (-1, shape[0]):
        with pytest.raises(IndexError):
            t.gather_rows(torch.tensor([0, wrong]))
    assert np.array_equal(t.gather_rows(ids).view(torch.uint16).cpu().numpy(), words[ids.numpy()])


# More blocks than a CTA has lanes (at most 1024): every lane walks a second block through the ring that the first one used.
# rows that are whole blocks (decoded class by class; also one row of 1536 blocks gathered), rows of whole runs of 16, any rows
ROUNDS = [((4100, 1024), 16), ((3, 24576), 16), ((4100, 2064), 32), ((4100, 1030), 16)]


@pytest.mark.parametrize("shape,stride", ROUNDS)
@pytest.mark.parametrize("coarse", [False, True])
def test_lanes_that_walk_several_blocks(orc, shape, stride, coarse):
    from georefine_b200 import codec
    from georefine_b200.gpu import CudaContextTensor

    words = orc.synthetic_weight_words(*shape, 11)
    if coarse:
        words &= 0xFFF8
    t = CudaContextTensor(codec.encode(words), stride=stride, walk_stride=stride, device="cuda:0", fused=False)
    assert t._packed is not None and t.mode == (128 if coarse else 0)
    if shape[0] > 148:
        assert -(-words.size // stride) > 148 * 1024
    for _ in range(3):
        assert np.array_equal(t.decode().view(torch.uint16).cpu().numpy(), words)
    ids = torch.arange(shape[0]).flip(0)[:200]
    assert np.array_equal(t.gather_rows(ids).view(torch.uint16).cpu().numpy(), words[ids.numpy()])


def test_threads_that_share_a_tensor_see_their_own_outcome(orc):
    """One thread asks for rows that exist, the other for one that does not: neither's verdict reaches the other."""
    import threading

    from georefine_b200 import codec
    from georefine_b200.gpu import CudaContextTensor

    words = orc.synthetic_weight_words(64, 4096, 5)
    t = CudaContextTensor(codec.encode(words), device="cuda:0", fused=False)
    wrong, rounds = [], 300

    def ask(ids, bad):
        stream, ids = torch.cuda.Stream(), ids.cuda()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for _ in range(rounds):
                try:
                    rows = t.gather_rows(ids)
                    if bad or not torch.equal(rows.view(torch.int16), want):
                        wrong.append("no error for a row outside" if bad else "wrong words")
                except IndexError:
                    if not bad:
                        wrong.append("the other thread's error")

    good = torch.arange(64).flip(0)
    want = torch.from_numpy(words[good.numpy()].view(np.int16)).cuda()
    threads = [threading.Thread(target=ask, args=a) for a in ((good, False), (torch.tensor([0, 64]), True)) for _ in range(2)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not wrong, (len(wrong), wrong[:3])


def test_a_replay_clears_the_error_word_of_the_one_before(orc):
    from georefine_b200 import codec
    from georefine_b200.gpu import CudaContextTensor

    words = orc.synthetic_weight_words(64, 512, 5)
    t = CudaContextTensor(codec.encode(words), device="cuda:0", fused=False)
    assert np.array_equal(t.decode().view(torch.uint16).cpu().numpy(), words)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = t.decode(check=False)
    for eager in (lambda: t.decode(check=False), t.decode):
        t.error.fill_(4)                                     # as a replay over broken streams leaves it
        graph.replay()
        assert int(t.error.item()) == 0 and np.array_equal(out.view(torch.uint16).cpu().numpy(), words)
        t.error.fill_(4)
        eager()
        assert int(t.error.item()) == 0


@pytest.mark.parametrize("shape,classes", [((6000, 128), (16, 4)), ((6000, 130), (16, 4)), ((2600, 256), (64, 16)), ((40, 512), (16, 4))])
@pytest.mark.parametrize("coarse", [False, True])
def test_gathers_on_both_sides_of_the_packed_limit(orc, shape, classes, coarse):
    """Rows by the packed kernel, by the general one and out of a whole decode are the same bits, and refuse the same."""
    from georefine_b200 import codec
    from georefine_b200.gpu import CudaContextTensor

    words = orc.synthetic_weight_words(*shape, 9)
    if coarse:
        words &= 0xFFF8
    t = CudaContextTensor(codec.encode(words, row_classes=classes[0], col_classes=classes[1]), device="cuda:0", fused=False)
    limits = {t._gather_limit} if shape[1] % t.walk_stride else {t._gather_limit, 100, shape[0] + 100}
    if shape[0] <= t._gather_limit:
        limits -= {100}                                      # no tables for the general kernel: it would not be taken
    for limit in sorted(limits):
        t._gather_limit = limit
        for count in (limit, limit + 1, shape[0], shape[0] + 1):
            if not 0 < count * shape[1] < 40_000_000:
                continue
            ids = torch.randint(0, shape[0], (count,), generator=torch.Generator().manual_seed(count))
            ids[0], ids[-1] = shape[0] - 1, 0
            rows = t.gather_rows(ids.reshape(1, -1))
            assert rows.shape == (1, count, shape[1]) and np.array_equal(rows[0].view(torch.uint16).cpu().numpy(), words[ids.numpy()])
            for wrong in (-1, shape[0]):
                ids[count // 2] = wrong
                with pytest.raises(IndexError):
                    t.gather_rows(ids)


def test_tensors_share_one_pinned_block(orc):
    """Outcomes of checked decodes need no pinned allocation per tensor, and every place comes back, also after an error."""
    from georefine_b200 import codec, gpu

    words = orc.synthetic_weight_words(32, 256, 5)
    frame = codec.encode(words)
    gpu.CudaContextTensor(frame, device="cuda:0", fused=False).decode()
    pinned = torch.cuda.host_memory_stats()["num_host_alloc"]
    tensors = [gpu.CudaContextTensor(frame, device="cuda:0", fused=False) for _ in range(5)]
    places = len(gpu._Outcome.free)
    for t in tensors:
        assert np.array_equal(t.decode().view(torch.uint16).cpu().numpy(), words)
        with pytest.raises(IndexError):
            t.gather_rows(torch.tensor([32]))
        assert len(t.gather_rows(torch.tensor([31]))) == 1
    assert len(gpu._Outcome.free) == places and torch.cuda.host_memory_stats()["num_host_alloc"] == pinned
