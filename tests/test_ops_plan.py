"""Planning layer: parts catalogue vs the built library, step plans, collective plans.
Reference tests: crates/sparkflash-ops (parts.rs asserts on the catalogue, collective.rs plan choices)."""
import pytest

from sparkflash_b200.ops import plan as P


def test_every_catalogued_entry_point_is_exported_by_the_library():
    r = P.KernelResolver()
    assert r.missing() == []
    assert r.resolve("attention", "tc") == "sfb_attn_tc"
    with pytest.raises(KeyError):
        r.resolve("attention", "nonexistent")
    with pytest.raises(KeyError):
        r.resolve("no_such_part", "x")


def test_resolver_reports_a_dropped_symbol():
    class Fake:
        def __getattr__(self, name):
            if name == "sfb_attn_tc":
                raise AttributeError(name)
            return object()
    r = P.KernelResolver(lib=Fake())
    assert ("attention", "tc", "sfb_attn_tc") in r.missing()
    with pytest.raises(LookupError):
        r.resolve("attention", "tc")


def test_step_plan_switches_variants_at_the_engine_thresholds():
    from sparkflash_b200.models.deepseek_v41.engine import Engine
    assert Engine.GROUP_MIN_ROWS == P.GROUP_MIN_ROWS and Engine.GROUP_WIDE_ROWS == P.GROUP_WIDE_ROWS
    one, few, chunk, bulk = (P.plan_step(n) for n in (1, 16, 128, 1024))
    assert (one.dense, one.attention, one.moe, one.coef, one.fold) == ("skinny", "rows", "token", "rows", "cluster")
    assert few.moe == "seg16" and few.attention == "rows"
    assert chunk.attention == "tc" and chunk.wo_a == "pair_bulk" and chunk.dense == "skinny"
    assert (bulk.dense, bulk.moe, bulk.coef, bulk.fold, bulk.gate) == ("bulk", "seg64", "gemm", "rows", "gemm")
    cuda = P.plan_step(16, arm="cuda")
    assert cuda.dense == "cuda_core" and cuda.moe == "cuda_core" and cuda.index_scores == "cuda_core"
    assert one.kernels_per_layer() < bulk.kernels_per_layer(index_layer=True, kv_source=True)


@pytest.mark.parametrize("rows,experts,segment", [(99, 64, 16), (100, 64, 64), (1365, 64, 64), (1366, 64, 96), (1024, 384, 64), (4096, 384, 64), (8191, 384, 64),
                                                  (8192, 384, 96)])
def test_segments_follow_the_pairs_per_expert_of_the_whole_layer(monkeypatch, rows, experts, segment):
    """The same sizes when one rank holds every expert and when eight hold an eighth each, and in the plan of the step."""
    from types import SimpleNamespace
    from sparkflash_b200.models.deepseek_v41 import engine as E
    cfg = SimpleNamespace(hidden_size=5120, n_routed_experts=experts, top_k=6, swiglu_limit=10.0)
    seen = []
    names = SimpleNamespace(**{f: lambda *a, seg=None, **k: seen.append(seg) for f in ("moe_plan", "moe_permute", "umma_gate_up_grouped", "umma_down_grouped", "moe_combine")})
    monkeypatch.setattr(E, "N", names)
    mat = SimpleNamespace(tmap=None, atoms=None)

    class Buffers(dict):
        def __missing__(self, key):
            return None

    class Rank(E.Engine):
        def __init__(self, local):
            self.cfg, self.w, self.il, self.status, self.xq, self.xs, self.ids, self.wts = cfg, SimpleNamespace(experts_local=local), 2304, None, None, None, None, None
            self.y_ffn = SimpleNamespace(stride=lambda i: 5120)

        def _group_buffers(self, *a):
            return Buffers(x_atom_bytes=0)

        def _k(self):
            pass
    for local in (0, experts // 8):
        seen.clear()
        Rank(local)._ffn_grouped(rows, SimpleNamespace(w13=mat, s13=mat, w2=mat, s2=mat), 6, True)
        assert set(seen) - {None} == {segment}, local
    assert E.Engine.GROUP_WIDER_PAIRS == P.GROUP_WIDER_PAIRS
    assert P.plan_step(rows, experts=experts).moe == f"seg{segment}"
    assert P.plan_step(rows, experts=experts, d=5120 + 128).moe == f"seg{min(segment, 64)}"


def test_workspaces_of_the_experts_cover_the_steps_that_use_them_and_no_more(monkeypatch):
    """4,096 rows over 128 experts: segments of 16 pairs serve up to 99 rows, of 64 up to 2,730, of 96 the rest."""
    from types import SimpleNamespace
    from sparkflash_b200.models.deepseek_v41 import engine as E
    nothing = lambda *a, **k: None
    names = ("moe_plan", "moe_permute", "umma_gate_up_grouped", "umma_down_grouped", "moe_combine")
    planned = []
    monkeypatch.setattr(E, "N", SimpleNamespace(**dict.fromkeys(names, nothing), TensorMap=lambda *a: SimpleNamespace(ptr=0)))
    E.N.moe_plan = lambda ids, wts, n, k, El, shared, S, expert, count, weight, token, pos, seg: planned.append(
        expert.numel() >= S and token.numel() >= S * seg and pos.numel() >= n * (k + 1))
    mat = SimpleNamespace(tmap=None, atoms=None)
    T = SimpleNamespace(w13=mat, s13=mat, w2=mat, s2=mat)

    class Stub(E.Engine):
        def __init__(self):
            self.cfg = SimpleNamespace(hidden_size=5120, n_routed_experts=128, top_k=6, swiglu_limit=10.0)
            self.w, self.il, self.max_rows, self.dev = SimpleNamespace(experts_local=128), 2304, 4096, "meta"
            self.status = self.xq = self.xs = self.ids = self.wts = None
            self.y_ffn = SimpleNamespace(stride=lambda i: 5120)

        def _k(self):
            pass
    eng = Stub()
    for n in (4, 42, 43, 99, 100, 777, 2730, 2731, 4096):
        eng._ffn_grouped(n, T, 6, True)
    assert all(planned)
    sets = {seg: sum(t.numel() * t.element_size() for t in g.values() if hasattr(t, "numel")) for seg, g in eng._grp.items()}
    # a pair slot: its FP8 row, its FP8 activations, the 32-bit output, the scales, weight and token
    slot = lambda seg: 5120 + 2304 + 4 * 5120 + 2 * (5120 + 2304) * (128 if seg <= 128 else seg) // seg // 32 + 64
    assert set(sets) == {16, 64, 96}
    assert sets[16] <= (128 + 99 * 6 // 16 + 7) * 16 * slot(16) and sets[64] <= (128 + 2730 * 6 // 64 + 43) * 64 * slot(64)
    assert sets[96] <= (128 + 4096 * 6 // 96 + 43) * 96 * slot(96)
    assert eng._group_rows() == {16: 99, 64: 2730, 96: 4096}
    for eng.max_rows in (3, 4, 98, 99, 100, 101, 2730, 2731, 2732):
        assert eng._group_rows() == {eng._group_size(n, 6, 128): n for n in range(4, eng.max_rows + 1)}
    eng.max_rows = 4096
    # a rule changed under a running engine: a larger workspace, the earlier one alive for what was captured with it
    first = eng._grp[16]
    eng.GROUP_WIDE_ROWS = 1000
    eng._ffn_grouped(900, T, 6, True)
    assert all(planned) and eng._grp[16]["rows"] == 999 and eng._grp[16]["before"] is first
    eng._ffn_grouped(50, T, 6, True)
    assert eng._grp[16]["before"] is first


def test_collective_plan_forms_and_bytes():
    d = 5120
    assert P.plan_collective(8, d, 1).kind is P.CollectiveKind.NONE
    a = P.plan_collective(8, d, 8)
    b = P.plan_collective(1024, d, 8)
    assert a.kind is P.CollectiveKind.ONE_SHOT and b.kind is P.CollectiveKind.TWO_SHOT
    assert P.plan_collective(1024, d, 4).kind is P.CollectiveKind.ONE_SHOT                # below 8 ranks the one-shot push measured faster
    assert P.plan_collective(1024, d, 4, two_shot_world=4).kind is P.CollectiveKind.TWO_SHOT
    assert a.bytes_sent_per_rank == 8 * d * 2 * 7
    assert b.bytes_sent_per_rank == 2 * 1024 * d * 2 * 7 // 8            # 2 (W-1)/W of the message
    assert P.plan_collective(1024, d, 8, arm="nccl").kind is P.CollectiveKind.NCCL
    o = P.plan_collective(4096, d, 4, bulk_chunks=8)
    assert o.kind is P.CollectiveKind.OVERLAPPED and o.chunks_in_flight == 3
    # rows are owned in equal blocks; every row has exactly one owner
    owned = [b.rows_owned(r) for r in range(8)]
    assert owned[0] == (0, 128) and owned[-1] == (896, 1024)
    odd = P.plan_collective(1000, d, 8)
    cover = [i for r in range(8) for i in range(*odd.rows_owned(r))]
    assert cover == list(range(1000))
    assert b.link_seconds() == pytest.approx(b.bytes_sent_per_rank / 770e9)
