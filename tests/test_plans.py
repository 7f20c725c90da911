"""The launch plans of the attention parts, asked on the host: no device is needed."""
from types import SimpleNamespace

import pytest
import torch

from gophonic_b200.engine.step import build_batch
from gophonic_b200.parts.attention import Attention, choose_splits, few_splits
from gophonic_b200.parts.gated_attention import GatedAttention

SIZES = [1, 2, 3, 5, 8, 13, 24, 50, 64, 128]
LENGTHS = [1, 63, 64, 65, 100, 256, 700, 1500, 4096, 12000, 40960]


def part(heads=32, kv_heads=8, head_dim=128, window=0, keep_first=0, fp32=False):
    p = SimpleNamespace(spec=SimpleNamespace(heads=heads, kv_heads=kv_heads, head_dim=head_dim, window=window, keep_first=keep_first),
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


@pytest.mark.parametrize("window", [0, 300])
def test_single_tokens_take_the_finer_of_both_rules(window):
    a, full = part(window=window), part(window=window, fp32=True)
    for n in SIZES:
        for kv in LENGTHS:
            coarse = choose_splits(8 * n, kv)
            assert a.plan(n, 1, kv, 148) == max(coarse, few_splits(8 * n, min(kv, window) if window else kv))
            assert full.plan(n, 1, kv, 148) == choose_splits(8 * n, kv, 148, 65536)
            # the gated form keeps to the one rule, over the keys that a row can see
            g = part(window=window, keep_first=20)
            assert GatedAttention.plan(g, n, 1, kv, 148) == choose_splits(8 * n, min(kv, window + 20) if window else kv)


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
