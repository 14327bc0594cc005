"""Edges of the decode step's small kernels: runs of rows that share a KV tile, row widths at the switch of the norm (needs a B200)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,nkv", [(8, 8), (8, 4), (16, 4), (10, 2), (8, 1), (5, 1)])
def test_rows_of_mixed_runs_equal_rows_alone(nq, nkv):
    """Runs that start and end anywhere in a group, a sequence that comes back after another one, rows whose context ends
    before a part that their neighbours see; every row has the bits it has alone."""
    from georefine_b200 import ops

    g = torch.Generator().manual_seed(nq + nkv)
    slots, pages = 4, 3
    cos, sin = ops.rope_tables(pages * ops.PAGE, device="cuda:0")
    table = torch.randperm(slots * pages, generator=g).reshape(slots, pages).to(torch.int32).cuda()
    kv = [torch.randn(slots * pages, nkv, ops.PAGE, 128, generator=g).to(torch.bfloat16).cuda() for _ in range(2)]
    attn = ops.PagedAttention(nq, nkv, max_rows=64, max_pages=pages, device="cuda:0")
    seqs = [0, 0, 1, 0, 2, 2, 2, 3, 1, 1, 1, 1, 1, 3, 3, 0, 2]
    at = [3, 600, 127, 700, 128, 129, 400, 0, 255, 256, 257, 500, 767, 383, 384, 5, 6]
    seqs, at = seqs + seqs[::-1], at + [(p + 13) % (pages * ops.PAGE) for p in at[::-1]]
    rows = len(seqs)
    qkv = torch.randn(rows, (nq + 2 * nkv) * 128, generator=g).to(torch.bfloat16).cuda()
    rs, rp = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in (seqs, at))
    assert len(set(zip(seqs, at))) == rows                  # no two rows append to the same place
    out = torch.full((rows, nq * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    attn(qkv, cos, sin, rs, rp, table, *kv, out)            # appends every row's keys and values
    for r in range(rows):                                   # (appending again writes the same bits)
        solo = torch.full((1, nq * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
        attn(qkv[r:r + 1], cos, sin, rs[r:r + 1], rp[r:r + 1], table, *kv, solo)
        assert torch.equal(solo[0], out[r]), (r, seqs[r], at[r])


@pytest.mark.parametrize("hidden", [8184, 8192, 8200])
def test_rmsnorm_at_the_switch_of_its_width(hidden):
    from georefine_b200 import ops

    g = torch.Generator().manual_seed(hidden)
    h, delta = (torch.randn(3, hidden, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    w = (1 + 0.2 * torch.randn(hidden, generator=g)).to(torch.bfloat16).cuda()
    summed = (h.float() + delta.float()).to(torch.bfloat16).double()
    want = summed * torch.rsqrt(summed.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    out = torch.empty_like(h)
    ops.rmsnorm(h, w, out, delta=delta)
    assert torch.equal(h.double(), summed)
    assert bool(((out.double() - want).abs() <= want.abs() * 2.0**-8 + 1e-30).all())     # one BF16 rounding, 2^-9, and FP32 noise
