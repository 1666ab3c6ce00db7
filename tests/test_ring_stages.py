"""Stages of the rings of decode-sized products (host arithmetic, no GPU)."""
import pytest

from nkipy_b200.ops import _lib


# from 113 or 227 KB less barriers; one CTA per SM: stages of 16 KB of weights (32 KB gated by weights) and 4 KB per 32 tokens
# (8 KB gated by tokens)
@pytest.mark.parametrize("block_n,ctas_per_sm,gated,push,stages", [
    (32, 2, 0, 0, 4), (32, 2, 1, 0, 3), (32, 2, 2, 0, 4), (32, 1, 0, 0, 10), (32, 1, 1, 0, 5), (32, 1, 2, 0, 8), (32, 2, 0, 1, 5),
    (64, 2, 0, 0, 4), (64, 1, 0, 0, 9), (64, 1, 1, 0, 5), (64, 2, 0, 1, 4), (128, 2, 0, 0, 3), (128, 1, 0, 0, 7), (128, 2, 0, 1, 3)])
def test_rings_keep_the_stages_that_fit(block_n, ctas_per_sm, gated, push, stages):
    """Only rings of 32 tokens with four stages and more stay as they were before the memory of bulk stores was theirs."""
    assert _lib.lib().nkb_gemm_ring_stages(block_n, ctas_per_sm, gated, push) == stages
