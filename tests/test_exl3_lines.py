"""Which EXL3 calls sort into the wide items (no GPU: the choice is a function of the call's shape)."""

from types import SimpleNamespace

import pytest


@pytest.mark.parametrize("dims, width, count, wide_from", [
    (1024, 1536, 128, 13), (1024, 640, 128, 13), (2048, 768, 128, 7), (2048, 1536, 64, 7), (3072, 768, 160, 7),
    (4096, 1280, 64, 6), (4096, 1536, 160, 6), (4096, 1536, 20, 14), (1024, 512, 32, 14)])
def test_mixed_widths_take_the_wide_items_by_the_inputs_a_block_walks(dims, width, count, wide_from):
    """At each line and one row of pairs below it, for layers whose tensors differ in width."""

    from tensorfold_b200.exl3 import experts

    ex = SimpleNamespace(mixed=True, dims=dims, width=width, count=count, k2_gu=(4, 16), k2_d=(4, 16))
    for pairs, want in ((wide_from * count, experts.WIDE_ITEM_PAIRS), (wide_from * count - 1, experts.ITEM_PAIRS)):
        assert experts.item_pairs(pairs, count, experts.wide_from(ex, pairs)) == want
