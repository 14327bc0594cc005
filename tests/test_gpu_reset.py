"""What is left to the host after a launch that gave up (needs a B200).  The launch itself is not run: its leftovers, counted parts and a
status, are put in place by the host, and no kernel reads them before they are cleared."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["window4", "window", "rans"])
def test_reset_after_a_timeout(layout):
    from georefine_b200.resident import ResidentWeight

    w = (torch.randn(640, 2048, generator=torch.Generator().manual_seed(3)) * 0.02).to(torch.bfloat16)
    r = ResidentWeight.from_words(w.view(torch.int16).numpy().view(np.uint16), torch.device("cuda:0"), max_m=16, workers=37, layout=layout)
    x = torch.randn(40, 2048, generator=torch.Generator().manual_seed(4)).to(torch.bfloat16).cuda()
    want, y = (torch.empty(40, 640, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    r.reserve(40)                                                # (a second workspace; the first is kept)
    r.gemm(x, want)
    assert r.check_status() == 0
    for scratch in (r.workspace, *r._outgrown):
        scratch[:4 * int(r.header.row_blocks)].fill_(1)
    r.status.fill_(16)
    assert torch.equal(r.decode(), w.cuda())                     # does not touch the counters, and does not hide the timeout
    assert r.check_status() == 16
    r.reset()
    assert r.check_status() == 0
    r.gemm(x, y)
    assert r.check_status() == 0 and torch.equal(y, want)
    for scratch in (r.workspace, *r._outgrown):
        assert not bool(scratch[:4 * int(r.header.row_blocks)].any())
