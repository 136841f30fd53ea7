"""Layered engine, host side of a step: which rows of the index buffer a step's kernels read, against a count row by row, and the choice between a
captured step and an eager one for every way to ask for heads."""
import random
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from sparkflash_b200.kv.paged import PAGE
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


def _row_by_row(eng, segs, advs, heads, temps, seeds):
    """The arrays of a step, one row at a time."""
    m, w = eng.model, {k: [] for k in ("tokens", "row_pos", "row_lane", "row_seg", "seg_row0", "seg_len", "chunk_seg", "chunk_row0", "chunk_rows", "chunk_first",
                                       "short_segs", "long_seg", "long_first", "long_row0", "long_rows")}
    back, short, tiles = [], [], []
    for k, ((lane, p0, toks, _), adv) in enumerate(zip(segs, advs)):
        run, r0, c0 = adv.replay + list(toks), len(w["tokens"]), len(w["chunk_seg"])
        w["seg_row0"].append(r0); w["seg_len"].append(len(run))
        for i, t in enumerate(run):
            w["tokens"].append(t); w["row_pos"].append(adv.start + i); w["row_lane"].append(lane); w["row_seg"].append(k)
            if i >= len(adv.replay):
                back.append(r0 + i)
        for i in range(0, len(run), eng.chunk_rows):
            w["chunk_seg"].append(k); w["chunk_row0"].append(r0 + i); w["chunk_rows"].append(min(eng.chunk_rows, len(run) - i)); w["chunk_first"].append(c0)
        long = m.tc_attention and len(run) >= LY.TC_MIN_ROWS
        if long:
            tiles += [(adv.start + i, r0 + i, min(LY.TC_TILE, len(run) - i), k) for i in range(0, len(run), LY.TC_TILE)]
            w["long_seg"].append(k); w["long_first"].append(len(w["long_row0"]))
            for i in range(0, len(run), LY.STATE_CHUNK):
                w["long_row0"].append(r0 + i); w["long_rows"].append(min(LY.STATE_CHUNK, len(run) - i))
        else:
            short += range(r0, r0 + len(run)); w["short_segs"].append(k)
    w["long_first"].append(len(w["long_row0"]))
    tiles.sort(reverse=True)
    hrows = [back[i] for i in heads]
    w["hpos"] = [w["row_pos"][r] for r in hrows]
    w["seg_src"], w["seg_dst"] = [a.src for a in advs], [a.dst for a in advs]
    w["seed"] = [(seeds[i] if seeds is not None else 0) & 0xFFFFFFFFFFFFFFFF for i in heads]
    w["temp"] = [float(temps[i]) if temps is not None else 0.0 for i in heads]
    w["head_rows"] = None if hrows == list(range(len(w["tokens"]))) else hrows
    w["tiles"], w["short_rows"] = [x for _, r, c, _ in tiles for x in (r, c)], short if tiles else None
    if not m.tc_state:
        w["short_segs"] = None
        for k in ("long_seg", "long_first", "long_row0", "long_rows"):
            del w[k]
    if len(segs) == len(w["tokens"]):
        w["short_segs"] = w["short_rows"] = None
        for k in ("tiles", "long_seg", "long_first", "long_row0", "long_rows"):
            w.pop(k, None)
    expand = {}
    for win in m.windows if tiles else ():
        pages, offs = [], {}
        for k, (adv, n) in enumerate(zip(advs, w["seg_len"])):
            if n >= LY.TC_MIN_ROWS:
                lo, hi = max(0, adv.start - win + 1) // PAGE, (adv.start + n - 1) // PAGE + 1
                offs[k] = len(pages) - lo
                pages += eng.kv.pages[segs[k][0]][lo:hi]
        expand[win] = (pages, [offs[k] for _, _, _, k in tiles])
    return w, expand


@pytest.mark.parametrize("tc,windows", [(False, ()), (True, ()), (True, (70, 300))])
@pytest.mark.parametrize("kind", [list, tuple, np.array])
def test_staged_arrays_are_those_of_a_count_row_by_row(tc, windows, kind):
    """Random mixes of decoded rows, short and long runs, and runs that begin inside a lane's latest step (whose first tokens run again)."""
    eng = LY.LayeredEngine(_Model(windows, tc), max_lanes=6, max_context=4096, max_rows=1200)
    rng = random.Random(3)
    for turn in range(40):
        toks, lanes, pos, budget = [], [], [], 500
        for lane in rng.sample(range(6), rng.randint(1, 6)):
            s = eng.state.lanes[lane]
            p0 = 0 if s.rows > 2500 else rng.randint(s.start, s.rows) if s.tokens and rng.random() < 0.3 else s.rows
            n = min(budget, 1 if turn % 4 == 0 else rng.choice([1, 2, 31, 32, 33, 64, 127, 128, 129, 256, 257]))
            if n:
                toks += [rng.randrange(VOCAB) for _ in range(n)]; lanes += [lane] * n; pos += range(p0, p0 + n)
            budget -= n
        n = len(toks)
        heads = rng.choice([list(range(n)), [], [n - 1], [-1], sorted(rng.sample(range(n), rng.randint(1, n))), [rng.randrange(-n, n) for _ in range(3)]])
        temps = rng.choice([None, [rng.random() for _ in range(n)]])
        seeds = rng.choice([None, [rng.getrandbits(64) - 2 ** 63 for _ in range(n)]])
        segs = eng._segments(kind(toks), kind(lanes), kind(pos))
        advs = [eng.state.plan(lane, p0) for lane, p0, _, _ in segs]
        for lane, p0, t, _ in segs:
            eng.kv.ensure(lane, p0 + len(t))
        s = eng._stage(segs, advs, heads, temps, seeds)
        want, expand = _row_by_row(eng, segs, advs, heads, temps, seeds)
        for name, values in want.items():
            got = getattr(s, name)
            if name == "seed":
                got = [x & 0xFFFFFFFFFFFFFFFF for x in got.tolist()]
            elif got is not None:
                got = got.tolist()
            if name == "temp":
                values = torch.tensor(values, dtype=torch.float32).tolist()
            assert got == values, (turn, name)
        assert {k: (p.tolist(), o.tolist()) for k, (p, _, o) in s.expand.items()} == expand and all(c == len(p) for p, c, _ in s.expand.values())
        assert s.n == len(want["tokens"]) and s.nhead == len(heads) and s.max_pos == max(want["row_pos"]) and s.chunks == len(want["chunk_seg"])
        for (lane, p0, t, _), adv in zip(segs, advs):
            eng.state.commit(adv, adv.replay + list(t))


@pytest.mark.parametrize("runs", [[1], [2], [3], [7, 8, 9], [1, 1, 1], [15, 1, 16, 17], [31, 33, 64]])
def test_runs_of_a_lane_end_where_the_next_one_begins(runs):
    values = [k for k, m in enumerate(runs) for _ in range(m)]
    i, ends = 0, []
    while i < len(values):
        i = LY._run_end(values, i, len(values))
        ends.append(i)
    assert ends == np.cumsum(runs).tolist()


@pytest.mark.parametrize("tokens,lanes,positions,message", [
    ([1, 1, 1], [0, 0, 0], [0, 1, 3], "consecutive"), ([1, 1, 1], [0, 0, 0], [2, 1, 0], "consecutive"), ([1, 1, 1], [0, 1, 0], [0, 0, 1], "not together"),
    ([1], [4], [0], "out of range"), ([1], [-1], [0], "out of range"), ([1], [0], [-1], "beyond the context"), ([1, 1], [0, 0], [511, 512], "beyond the context"),
    ([VOCAB], [0], [0], "vocabulary"), ([-1], [0], [0], "vocabulary"), ([], [], [], "rows 0"), ([1] * 65, [0] * 65, list(range(65)), "rows 65")])
def test_rows_that_make_no_step_are_refused(engine, tokens, lanes, positions, message):
    with pytest.raises(ValueError, match=message):
        engine.step(tokens, lanes, positions)


@pytest.mark.parametrize("kind", [list, tuple, np.array])
def test_a_continued_step_is_staged_as_any_other(engine, kind):
    """Captured steps of one row per lane through the short way and through segments: the same index buffer, pages, states, errors and answers, for rows
    that go on, begin again at 0, repeat the latest position or are none of these."""
    other = LY.LayeredEngine(_Model(), max_lanes=4, max_context=512, max_rows=64)
    other._continue = lambda *a: False
    rng, short = random.Random(5), 0
    engine._continue = lambda *a, go=engine._continue: go(*a) and (setattr(engine, "taken", engine.taken + 1) or True)
    engine.taken = 0
    staged = {}

    def replay(e):
        staged[e] = e._meta[:9 * len(lanes)].tolist()
        e.best_id[:len(lanes)] = e._meta[3 * len(lanes):4 * len(lanes)] + 1000
    for e in (engine, other):
        e.graphs.update({(n, b, s): SimpleNamespace(replay=lambda e=e: replay(e)) for n in range(1, 5) for b in (16,) for s in (True, False)})
        for lane in range(4):
            lanes = [lane] * (40 + lane)
            e.step([1] * len(lanes), lanes, list(range(len(lanes))), head=False)
    for turn in range(150):
        lanes = rng.sample(range(4), rng.randint(1, 4))
        rows = [engine.state.lanes[lane] for lane in lanes]
        pos = [0 if rng.random() < 0.05 else s.start if rng.random() < 0.2 else s.rows + (rng.random() < 0.02) for s in rows]
        toks = [rng.randrange(VOCAB + (rng.random() < 0.02)) for _ in lanes]
        kw = dict(temperature=rng.choice([None, [rng.random() for _ in lanes]]), seeds=rng.choice([None, [rng.getrandbits(64) - 2 ** 63 for _ in lanes]]), sample=rng.random() < 0.8)
        got = []
        for e in (engine, other):
            staged[e] = None
            try:
                got.append(e.step(kind(toks), kind(lanes), kind(pos), **kw).tolist())
            except ValueError as x:
                got.append(str(x))
        assert got[0] == got[1] and staged[engine] == staged[other], turn
        assert [vars_of(s) for s in engine.state.lanes] == [vars_of(s) for s in other.state.lanes] and engine.kv.pages == other.kv.pages, turn
    assert engine.taken > 75


def vars_of(lane):
    return lane.rows, lane.version, lane.start, lane.start_slot, list(lane.tokens)
