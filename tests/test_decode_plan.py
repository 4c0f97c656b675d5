"""How many CTAs share a sequence's keys in a decode step, worked out on the host (3 CTAs on each of 148 SMs, as on a B200)."""

import pytest

from tokensprint_b200 import ops


@pytest.fixture
def b200(monkeypatch):
    monkeypatch.setattr(ops, "_decode_slots", lambda head_dim: 444)
    monkeypatch.delenv("TS_DECODE_SPLITS", raising=False)


@pytest.mark.parametrize("seqs,heads,splits", [(1, 8, 8), (3, 8, 8), (5, 8, 8), (6, 4, 8), (1, 1, 8), (16, 2, 8)])
def test_few_pairs_merge_in_a_cluster(b200, seqs, heads, splits):
    assert ops.attention_decode_splits(seqs, heads, 2048) == splits
    assert ops.attention_decode_splits(seqs, heads, 2048, reach=4096) == splits


@pytest.mark.parametrize("seqs,heads,splits", [(1, 8, 16), (3, 8, 16), (4, 8, 11), (5, 8, 11), (1, 1, 16), (6, 4, 16)])
def test_steps_that_may_meet_long_contexts_are_split_further(b200, seqs, heads, splits):
    for reach in (8192, 40960):
        assert ops.attention_decode_splits(seqs, heads, 2048, reach=reach) == splits


@pytest.mark.parametrize("seqs,heads,context,splits", [(8, 8, 2048, 6), (19, 8, 2048, 8), (22, 8, 2048, 5), (28, 8, 2048, 3), (40, 8, 2048, 4),
                                                       (80, 4, 2048, 4), (32, 8, 1024, 3), (40, 8, 1024, 4), (64, 8, 576, 3)])
def test_larger_steps_leave_the_choice_to_the_even_share_kernel(b200, seqs, heads, context, splits):
    """Steps whose lengths differ gain from the even shares: these counts send them there where that kernel takes the layer."""
    for reach in (0, 4096):
        assert ops.attention_decode_splits(seqs, heads, context, reach=reach) == splits


def test_a_window_bounds_what_a_step_can_meet(b200):
    assert ops.attention_decode_splits(1, 8, ops.attention_decode_plan_context(40960, 512), reach=576) == 5
