"""Layered engine, host side of a step: the choice between a captured step and an eager one for every way to ask for heads."""
from types import SimpleNamespace

import pytest
import torch

from sparkflash_b200.models import layered as LY

VOCAB = 50


class _Model:
    """Nothing but the sizes that staging reads; ``forward`` keeps the Step it was given."""
    cfg, vocab, device, dtype, kv_runs = None, VOCAB, "cpu", torch.float32, [(1, 4, 4)]

    def __init__(self, windows=(), tc=False):
        self.windows, self.tc_attention, self.tc_state, self.seen = windows, tc, tc, None

    def bind(self, engine):
        pass

    def forward(self, s):
        self.seen = s
        return torch.zeros(s.nhead, VOCAB)


@pytest.fixture
def engine(monkeypatch):
    """An engine whose sampler names every head's position and whose captured steps do the same for all rows."""
    eng = LY.LayeredEngine(_Model(), max_lanes=4, max_context=512, max_rows=64)
    eng.replays = 0

    def sample(logits, hpos, temp, seed, mask, best_val, best_id, n):
        best_id[:n] = hpos + 1000
    monkeypatch.setattr(LY.R, "sample", sample)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: SimpleNamespace(synchronize=lambda: None))

    def replay():
        eng.replays += 1
        n = eng.captured_rows
        eng.best_id[:n] = torch.tensor([eng.state.rows(lane) for lane in range(n)]) + 1000
    eng.capture = lambda n: (setattr(eng, "captured_rows", n), eng.graphs.update({(n, 16, True): SimpleNamespace(replay=replay)}))
    return eng


@pytest.mark.parametrize("n,head,replayed", [(1, True, True), (1, "last", True), (1, [0], True), (1, [-1], True), (2, True, True), (2, [0, 1], True), (2, [-2, -1], True),
                                             (2, [0, -1], True), (2, [-1, 0], False), (2, [1], False), (2, [-1], False), (2, [0, 0], False), (2, False, False)])
@pytest.mark.parametrize("captured", [False, True])
def test_a_decoded_row_is_answered_however_its_head_is_named(engine, n, head, replayed, captured):
    """Rows may be counted from the end.  Where a captured step answers, no index arrays are made; where none does, all of them are."""
    engine.use_graphs = captured
    for lane in range(n):
        engine.step([1] * (3 + lane), [lane] * (3 + lane), list(range(3 + lane)), head=False)
    engine.capture(n)
    out = engine.step([7] * n, list(range(n)), [3 + i for i in range(n)], head=head)
    heads = range(n) if head is True else [] if head is False else [n - 1] if head == "last" else [h % n for h in head]
    assert out.tolist() == [1003 + i if i in heads else 0 for i in range(n)]
    assert engine.replays == int(captured and replayed)
    if not engine.replays:
        s = engine.model.seen
        assert s.tokens.tolist() == [7] * n and s.row_pos.tolist() == [3 + i for i in range(n)] and s.hpos.tolist() == [3 + i for i in heads]
    assert [engine.state.rows(lane) for lane in range(n)] == [4 + i for i in range(n)]


@pytest.mark.parametrize("head", [[1], [-2]])
def test_heads_that_are_no_rows_are_refused(engine, head):
    with pytest.raises(IndexError):
        engine.step([1], [0], [0], head=head)
