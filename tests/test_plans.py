"""The launch plans of the attention parts, asked on the host: no device is needed."""
from types import SimpleNamespace

import pytest
import torch

from gophonic_b200.engine import graphs
from gophonic_b200.engine.step import build_batch
from gophonic_b200.parts.attention import Attention, choose_splits, few_splits, page_class, wave_splits
from gophonic_b200.parts.gated_attention import GatedAttention
from gophonic_b200.parts.latent_attention import LatentAttention

SIZES = [1, 2, 3, 5, 8, 13, 24, 50, 64, 128]
LENGTHS = [1, 63, 64, 65, 100, 256, 700, 1500, 4096, 12000, 40960]


def part(heads=32, kv_heads=8, head_dim=128, window=0, keep_first=0, fp32=False):
    p = SimpleNamespace(spec=SimpleNamespace(heads=heads, kv_heads=kv_heads, head_dim=head_dim, value_dim=head_dim, window=window, keep_first=keep_first),
                        rt=SimpleNamespace(is_fp32=fp32))
    p.splits_of = lambda *a: Attention.splits_of(p, *a)
    p.plan = lambda *a: Attention.plan(p, *a)
    return p


@pytest.mark.parametrize("window", [0, 100, 1024])
def test_a_prompt_is_never_cut_by_what_else_is_in_its_step(window):
    """Pieces are joined in another order than one pass over the keys adds them: a portion's rows must not depend on how many
    sequences the step has or how long the others are."""
    a = part(window=window)
    assert {a.plan(n, q, max(q, kv), 148) for n in SIZES for q in (2, 64, 65, 90, 256, 2048) for kv in LENGTHS} == {1}


def test_pieces_of_few_sequences():
    """A power of two, pieces of at least 96 keys, no more CTAs than SMs and no more than 32 pieces; and as many as may be."""
    for units in (1, 2, 7, 8, 9, 32, 64, 74, 75, 148, 149, 4000):
        for kv_len in LENGTHS + [95, 96, 191, 192, 193, 383, 384]:
            s = few_splits(units, kv_len, 148)
            ok = lambda n: n == 1 or (kv_len >= 96 * n and units * n <= 148 and n <= 32)
            assert s & (s - 1) == 0 and ok(s) and not ok(2 * s)


@pytest.mark.parametrize("window", [0, 300, 1024])
def test_single_tokens_take_the_finest_of_the_rules(window):
    a, full = part(window=window), part(window=window, fp32=True)
    for n in SIZES:
        for kv in LENGTHS:
            coarse, seen = choose_splits(8 * n, kv), min(kv, window) if window else kv
            assert a.plan(n, 1, kv, 148) == wave_splits(max(coarse, few_splits(8 * n, seen)), 8 * n, 32 * n, seen, 296)
            assert full.plan(n, 1, kv, 148) == choose_splits(8 * n, kv, 148, 65536)
            # the gated form has two of them, over the keys that a row can see
            g, seen = part(window=window, keep_first=20), min(kv, window + 20) if window else kv
            assert GatedAttention.plan(g, n, 1, kv, 148) == wave_splits(choose_splits(8 * n, seen), 8 * n, 32 * n, seen, 296)


def test_pieces_that_fill_one_wave():
    """Nothing up to 512 visible keys; else no more CTAs than one wave holds (or two, nearly full, in three pieces of eight pages), no more than 16
    pieces, partial results of no more than four heads a place, no piece empty at the largest length of a class, and no more pieces that
    save a CTA too little."""
    for places in (148, 296):
        for units in (1, 2, 7, 8, 9, 24, 32, 64, 74, 75, 96, 148, 149, 192, 197, 198, 400, 4000):
            for group in (1, 4, 16):
                for kv_len in LENGTHS + [512, 513, 1472, 1473, 8192]:
                    for had in (1, 2, 5, 12, 32):
                        s, pages = wave_splits(had, units, units * group, kv_len, places), -(-kv_len // 64)
                        if pages <= 8:
                            assert s == had
                        elif 2 * units > places:
                            three = 3 * units <= 2 * places and 3 * group * units <= 8 * places and pages >= 24
                            assert s == (max(3, had) if three else had)
                        elif s != had:
                            assert had < s <= 16 and s * units <= places and s * units * group <= 4 * places
                            size = page_class(pages)
                            assert pages <= size <= 3 * pages // 2 and (pages <= s or (s - 1) * -(-size // s) < size)
                            assert -(-pages // had) - -(-pages // s) >= (5 if had == 1 else 1 if s == had + 1 else 2)
    rule = lambda n, kv: wave_splits(max(choose_splits(8 * n, kv), few_splits(8 * n, kv)), 8 * n, 32 * n, kv, 296)
    assert [rule(n, 700) for n in (1, 2, 3, 4, 5, 8, 12, 16, 24, 32, 64)] == [16, 16, 12, 4, 6, 4, 3, 2, 1, 1, 1]      # as measured
    assert [rule(n, 1500) for n in (1, 2, 3, 5, 8, 12, 16, 24, 32, 64)] == [8, 8, 12, 6, 4, 3, 2, 3, 1, 1]
    assert [rule(n, 4096) for n in (1, 2, 3, 5, 8, 12, 16, 24, 32, 64)] == [16, 16, 11, 7, 4, 3, 2, 3, 1, 1]
    assert rule(2, 900) == 8 and rule(16, 530) == 1
    assert wave_splits(8, 16, 256, 1500, 296) == 8       # eight sequences of two key heads, 16 heads each: the merge reads them all


def test_what_the_tensor_core_kernel_does_not_take_is_cut_as_before():
    wide = part(head_dim=40)
    unequal = part()
    unequal.spec.value_dim = 64
    for p, page in ((wide, 2 * 64 * 40 * 2), (unequal, 32768)):
        for n in (1, 4, 8):
            for kv in LENGTHS:
                assert GatedAttention.plan(p, n, 1, kv, 148) == choose_splits(8 * n, kv, 148, page)


def test_the_plan_of_a_step_does_not_depend_on_the_other_lengths():
    """Neither the number of pieces nor, with it, the captured step that is replayed moves with the mean length of a batch."""
    a = part()
    plans = set()
    for others in (1, 64, 700, 2999):
        batch, _ = build_batch([(i, [5], 2999 if i == 3 else others) for i in range(8)], torch.device("cpu"))
        plans.add(batch.plan_for(a))
    assert plans == {a.plan(8, 1, 3000, 148)}


def test_a_batch_of_one_size_asks_for_few_captured_steps():
    """Every answer is a step of its own to capture: over contexts of up to 8192 keys no more of them than the coarse rule gave."""
    a = part()
    for n, most in ((1, 16), (2, 14), (4, 8), (8, 4), (12, 3), (16, 2), (24, 2), (32, 1)):
        assert len({a.plan(n, 1, kv, 148) for kv in range(1, 8193, 7)}) <= most


def captured_steps(monkeypatch, plan, nseq, contexts):
    """How many steps are captured for ``nseq`` sequences as the longest of them grows, with mixers that answer ``plan``."""
    monkeypatch.setattr(graphs, "DecodeGraph", lambda engine, size, plans, *more: object())

    class Engine:
        sm_count = 148
        model = SimpleNamespace(step_plans=lambda *a: (plan(*a),))
    engine = Engine()        # the graphs refer to it weakly
    g = graphs.DecodeGraphs(engine, max_graphs=10 ** 6)
    g.pool = object()
    return len({id(g.get(nseq, kv)) for kv in contexts})


@pytest.mark.parametrize("plan", [part().plan, part(fp32=True).plan, part(window=300).plan, lambda *a: None])
def test_steps_are_captured_once_for_every_answer_of_the_plans(monkeypatch, plan):
    contexts = range(1, 12289, 7)
    for n in (1, 2, 8, 16, 24, 64):
        answers = {plan(graphs.captured_size(n), 1, kv, 148) for kv in contexts}
        assert captured_steps(monkeypatch, plan, n, contexts) == len(answers)


# ---- latent attention: which sequences of a step go over expanded keys and values -------------------------
def latent_part(window=1024, dtype=torch.bfloat16, heads=16, kv_rank=512, dims=(128, 64, 128)):
    from gophonic_b200 import ops
    weights = torch.empty(0, dtype=dtype)
    spec = SimpleNamespace(heads=heads, head_dim=dims[0], rot_dim=dims[1], value_dim=dims[2], kv_rank=kv_rank, window=window)
    return SimpleNamespace(spec=spec, rt=SimpleNamespace(ops=ops, act_dtype=dtype), uk_kn=weights, uv_nk=weights, key_dim=kv_rank + dims[1],
                           EXPANDED_KEYS_A_ROW=LatentAttention.EXPANDED_KEYS_A_ROW, EXPANDED_BYTES=LatentAttention.EXPANDED_BYTES,
                           FEW_ROWS_PAGES=LatentAttention.FEW_ROWS_PAGES)


def runs_of(extents, **kw):
    batch, _ = build_batch([(i, [5] * rows, known) for i, (known, rows) in enumerate(extents)], torch.device("cpu"))
    return LatentAttention._runs(latent_part(**kw), batch)


STEPS = [[(0, 65)], [(0, 64)], [(700, 1)], [(0, 2048), (0, 1196)], [(0, 70), (5, 1), (0, 64), (3000, 65), (3000, 90), (3000, 100), (11, 1000)],
         [(40000, 1000), (0, 100)], [(40000, 4000)] * 5, [(i * 37 % 5000, 1 + i * 61 % 400) for i in range(40)], [(2000, 3), (0, 1000), (90, 3)]]


@pytest.mark.parametrize("window", [0, 100, 1024])
@pytest.mark.parametrize("extents", STEPS)
def test_the_runs_of_a_step(extents, window):
    """A sequence's form does not depend on the others' contexts; runs follow one another without a gap, the pages are what the
    gather kernel walks, and no run's expanded rows take more scratch memory than is allowed."""
    runs, at, row = runs_of(extents, window=window), 0, 0
    for k, (first, end, lo, hi, most, pages) in enumerate(runs):
        assert (first, lo) == (at, row) and end > first
        mine = extents[first:end]
        at, row = end, row + sum(r for _, r in mine)
        assert hi == row and most == max(r for _, r in mine)
        if pages:
            # as the kernel counts: from the page of the first key that the first row sees to the last token's
            assert pages == sum(-(-(n + r) // 64) - (max(0, n - window + 1) // 64 if window else 0) for n, r in mine)
            assert 128 * pages * (576 + 16 * 256) <= max((hi - lo) * 32 * (576 + 512), LatentAttention.EXPANDED_BYTES)
        assert k == 0 or (runs[k - 1][5] > 0) != (pages > 0) or pages > 0
    assert at == len(extents)
    forms = lambda runs: [pages > 0 for first, end, _, _, _, pages in runs for _ in range(first, end)]
    for i in range(len(extents)):                # the same rows, the others behind other contexts
        for other in (0, 10, 777, 30000):
            assert forms(runs_of([e if j == i else (other, e[1]) for j, e in enumerate(extents)], window=window))[i] == forms(runs)[i]


def test_the_rule_of_expanded_latents():
    expanded = lambda known, rows, **kw: runs_of([(known, rows)], **kw)[0][5] > 0
    for window in (0, 1024):                                    # 1024 keys ahead of the portion, eleven a row
        for known in (0, 700, 3000):
            assert expanded(known, 94, window=window) and not expanded(known, 93, window=window)
    assert expanded(0, 65, window=100) and not expanded(0, 64, window=100)     # the fewest rows the kernel is for
    assert expanded(100000, 2000) and not expanded(100000, 2000, window=0)     # scratch memory: what the window hides takes none
    assert len(runs_of([(300, 300), (300, 9), (300, 120), (300, 1)])) == 1 and runs_of([(0, 66), (0, 5)]) == [(0, 2, 0, 71, 66, 0)]
    # few rows behind many keys leave the others, where the window does not hide them
    assert [r[5] > 0 for r in runs_of([(0, 500), (2000, 3), (1200, 3)], window=0)] == [True, False, True]
    assert [r[5] > 0 for r in runs_of([(0, 500), (2000, 3), (1200, 3)])] == [True]
    assert not expanded(0, 500, dtype=torch.float32) and not expanded(0, 500, dims=(64, 64, 128)) and not expanded(0, 500, kv_rank=516)
    assert runs_of([(0, 100), (9, 3)], dtype=torch.float32) == [(0, 2, 0, 103, 100, 0)]


@pytest.mark.parametrize("heads", [8, 16, 32, 64])
def test_pieces_of_single_tokens_over_latents(heads):
    """One wave of an SM a CTA, only where the pages that a CTA is saved are worth the merge; float32, narrow latents and many sequences
    are cut as the general rule says, and the captured steps of a batch size are few."""
    p = object.__new__(LatentAttention)
    p.spec = SimpleNamespace(heads=heads, kv_rank=512, window=0, chunk=0)
    p.rt, p.key_dim = SimpleNamespace(is_fp32=False), 576
    ctas = -(-heads // 32)
    for n in SIZES + [256, 8192, 100000]:
        for kv in LENGTHS + [129, 192, 193, 250, 350]:
            rule, got, fine = choose_splits(n, kv, 74, 64 * 576 * 2), p.plan(n, 1, kv, 148), p.fine_splits(n, kv, 148)
            assert got == max(rule, fine) and p.plan(n, 2, kv, 148) == 1
            assert fine == 1 or (n * ctas * fine <= 148 and fine <= 32 and kv > 128)
            if 2 * n * ctas > 148 or kv <= 128:
                assert got == rule
        assert len({p.plan(n, 1, kv, 148) for kv in range(1, 8193, 31)}) <= len({choose_splits(n, kv, 74, 64 * 576 * 2) for kv in range(1, 8193, 31)}) + 2
    if heads == 16:      # as measured
        assert [p.plan(n, 1, kv, 148) for n, kv in ((1, 700), (8, 1024), (16, 250), (16, 350), (24, 150), (24, 1500), (32, 350), (64, 1024))] == [12, 16, 1, 6, 1, 6, 1, 2]
    p.spec.kv_rank = 256
    assert p.fine_splits(1, 700, 148) == 1
    p.spec.kv_rank, p.rt.is_fp32 = 512, True
    assert p.plan(1, 1, 700, 148) == choose_splits(1, 700, 74, 64 * 576 * 4)


class RecordingOps:
    """Stands for the kernels that latent attention calls; keeps what attention was asked for."""

    def __init__(self):
        from gophonic_b200 import ops
        self.latent_expanded_accepts, self.LATENT_TC5_MIN_ROWS = ops.latent_expanded_accepts, ops.LATENT_TC5_MIN_ROWS
        self.attention_scratch_floats = ops.attention_scratch_floats
        self.cuts = []

    def head_gemm_mma_accepts(self, *a):
        return True

    def head_gemm_mma(self, *a):
        pass

    latent_q_rot = head_gemm_mma

    def attention(self, q, out, k, v, table, slot, q_start, q_len, kv_len, nseq, max_q_len, heads, kv_heads, dim, scale, window, splits, scratch, **more):
        more.pop("value_dim"), more.pop("chunk")
        self.cuts.append((max_q_len, splits, sorted(more)))


def test_a_mixed_steps_single_rows_are_cut_alike_whatever_their_neighbours_hold():
    """A row that joins other sequences' rows in a step is attended to in one pass over its keys: nothing follows from how many of the others
    have long contexts, or from how many rows they bring."""
    prompt = [(0, 1500)]
    cuts = []
    for others in ([(1300, 1)] * 10, [(1300, 1)] * 3 + [(100, 1)] * 7, [(1300, 1)] * 9 + [(1300, 2)]):
        p = object.__new__(LatentAttention)
        p.spec = SimpleNamespace(heads=4, head_dim=128, rot_dim=64, value_dim=128, kv_rank=512, window=0, chunk=0, scale=1.0)
        p.rt = SimpleNamespace(ops=RecordingOps(), act_dtype=torch.bfloat16, is_fp32=False)
        p.key_dim, p.position = 576, SimpleNamespace(kernel_args=lambda: (None, None, 64))
        p.uk_kn = p.uv_nk = p.uk_nk = p.uv_kn = torch.empty(0, dtype=torch.bfloat16)
        batch, _ = build_batch([(i, [5] * rows, known) for i, (known, rows) in enumerate(prompt + others)], torch.device("cpu"))
        q = torch.empty((batch.rows, 4 * 192), dtype=torch.bfloat16)
        ctx = torch.empty((batch.rows, 4 * 128), dtype=torch.bfloat16)
        cache = SimpleNamespace(k=torch.empty((1, 1, 64, 576), dtype=torch.bfloat16), v=None, block_table=None)
        runs = [r for r in LatentAttention.runs(p, batch) if not r[5]]
        assert runs                          # rows behind many pages stay on the latents
        for run in runs:
            LatentAttention._absorbed(p, batch, q, ctx, cache, run)
        cuts += p.rt.ops.cuts
    assert cuts and all((splits, more) == (1, []) for _, splits, more in cuts)
