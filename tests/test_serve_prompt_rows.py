"""How a prompt's rows reach a decoder: whole ones of this package, and a user's own with fewer entry points (host only)."""
import types

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


@pytest.mark.parametrize("rows,head", [(200, 0), (200, 71), (100, -5), (100, 100), (100, 101)])
def test_absorb_refuses_rows_it_has_no_logits_for(rows, head):
    # (200 rows fit the pass: nothing but the check of the head may refuse them)
    d = types.SimpleNamespace(max_rows=128, prompt_rows=384)
    with pytest.raises(ValueError, match="logits"):
        serve.BatchDecoder.absorb(d, [0] * rows, range(rows), [1] * rows, head)
