"""A prompt in chunks as wide as a pass, the last of which gives logits for its last rows, against chunks of a step (needs a B200)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [100, 128, 129, 255, 384, 385, 513, 900, 1000])
def test_same_tokens_logits_and_pages(length):
    from georefine_b200 import serve

    dev = torch.device("cuda:0")
    cfg = serve.DecoderConfig(hidden=640, layers=2, heads=10, kv_heads=2, ffn=1792, vocab=1000)
    weights = serve.DecoderWeights.synthetic(cfg, dev, seed=6)
    ids = torch.randint(0, cfg.vocab, (length,), generator=torch.Generator().manual_seed(length)).tolist()
    got = []
    for wide, rows in ((False, 128), (True, 128), (True, 200), (True, 48)):     # (48: a decoder whose prompts are as narrow as its steps)
        d = serve.BatchDecoder(weights, max_rows=rows, max_slots=1, max_context=1100, device=dev)
        b = serve.Batcher(d)
        if not wide:
            b._absorb = None
        slot = b.admit(ids)
        got.append((b.active[slot]["tokens"], d.kv[:, :, :-1].clone(), d.logits[(length - 1) % rows].clone()))
    for tokens, kv, logits in got[1:]:
        assert tokens == got[0][0] and torch.equal(kv, got[0][1]) and torch.equal(logits, got[0][2])
    with pytest.raises(ValueError):
        d.absorb([slot] * 49, range(49), [1] * 49, 0)
