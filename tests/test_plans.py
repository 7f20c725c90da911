"""The launch plans of the attention parts, asked on the host: no device is needed."""
from types import SimpleNamespace

import pytest

from gophonic_b200.parts.attention import Attention

SIZES = [1, 2, 3, 5, 8, 13, 24, 50, 64, 128]
LENGTHS = [1, 63, 64, 65, 100, 256, 700, 1500, 4096, 12000, 40960]


def part(heads=32, kv_heads=8, head_dim=128, window=0, fp32=False):
    return SimpleNamespace(spec=SimpleNamespace(heads=heads, kv_heads=kv_heads, head_dim=head_dim, window=window), rt=SimpleNamespace(is_fp32=fp32))


@pytest.mark.parametrize("window", [0, 100, 1024])
def test_a_prompt_is_never_cut_by_what_else_is_in_its_step(window):
    """Pieces are joined in another order than one pass over the keys adds them: a portion's rows must not depend on how many
    sequences the step has or how long the others are."""
    a = part(window=window)
    assert {Attention.plan(a, n, q, max(q, kv), 148) for n in SIZES for q in (2, 64, 65, 90, 256, 2048) for kv in LENGTHS} == {1}
