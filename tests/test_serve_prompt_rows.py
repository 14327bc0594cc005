"""How a prompt's rows reach a decoder: whole ones of this package, and a user's own with fewer entry points (host only)."""
import pytest

from georefine_b200 import serve
from test_serve_host_logic import FakeDecoder, greedy


class ThreeArguments(FakeDecoder):
    """Takes rows in without logits, three arguments, in passes wider than a step."""

    def __init__(self, **kw):
        super().__init__(**kw)
        self.prompt_rows = 3 * self.max_rows
        self.absorbed = []

    def absorb(self, slots, positions, tokens):
        assert 0 < len(slots) <= self.prompt_rows
        self.absorbed.append(len(slots))
        for slot, pos, tok in zip(slots, positions, tokens):
            self.cache[slot][pos] = tok


class WithHead(ThreeArguments):
    def absorb(self, slots, positions, tokens, head=None):
        super().absorb(slots, positions, tokens)
        if head is not None:
            assert 0 < len(slots) - head <= self.max_rows
            for row, (slot, pos) in enumerate(list(zip(slots, positions))[head:]):
                self.next_token[row] = greedy([self.cache[slot][p] for p in range(pos + 1)], 1)[0]


@pytest.mark.parametrize("length", [1, 7, 8, 9, 16, 17, 24, 25, 31, 32, 33, 60])
@pytest.mark.parametrize("kind", [FakeDecoder, ThreeArguments, WithHead])
def test_first_token_of_a_prompt(kind, length):
    d = kind(max_rows=8)
    b = serve.Batcher(d)
    ids = [(7 * i + length) % 50 for i in range(length)]
    slot = b.admit(ids)
    assert b.active[slot]["tokens"] == greedy(ids, 1)
    assert [d.cache[slot][p] for p in range(length)] == ids
    if kind is ThreeArguments:      # as before: all but the last rows taken in, the last of them a step of their own
        last = (length - 1) // 8 * 8
        assert sum(d.absorbed) == last and d.runs == [("verify", length - last, False)]
