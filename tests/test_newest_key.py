"""Decode steps on one rank: the newest key's probability is not rounded on its way to the values."""
import pytest
import torch

from nkipy_b200 import ops


@pytest.mark.skipif(ops.FUSED_ROPE_ATTN != "auto", reason="NKIPY_B200_FUSED_ROPE_ATTN is set")
def test_one_rank_fuses_by_default():
    assert ops.fused_rope_attn_enabled(1) and not ops.fused_rope_attn_enabled(2)


@pytest.mark.gpu
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("ctx", [2, 33, 300])
@pytest.mark.parametrize("splits", [1, 3])
def test_newest_key_is_weighted_in_32_bits(D, ctx, splits):
    """Two keys count: an older one of probability 1 (before the division) and the newest.  Their values cancel up to what bf16
    cannot hold of the newest key's probability, so the result is nothing but that."""
    score = -0.28125                                             # of the newest key; exact in bf16, its exponential is not
    p = torch.tensor(score, dtype=torch.float64).exp()
    c = p.to(torch.bfloat16).double()
    pages = -(-ctx // 32)
    k, v = (torch.zeros((pages, 1, 32, D), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    k[..., 0] = -200.0                                           # the other keys: probabilities below 2^-200
    k[0, 0, 0, 0] = 0.0
    v[0, 0, 0] = -float(c)
    row = torch.zeros((1, 1, 3 * D), device="cuda")
    row[..., 0], row[..., D], row[..., 2 * D:] = 1.0, score, 1.0
    at = torch.tensor([ctx - 1], dtype=torch.int32, device="cuda")
    table = torch.arange(pages, dtype=torch.int32, device="cuda")[None]
    out = ops.rope_attn_decode(row, at, at, None, k, v, table, at + 1, 1.0, 1, 1, num_splits=splits).double()
    want = (p - c) / (1 + p)
    assert abs(want) > 2.0 ** -12
    # sums of a few terms of at most 1 in fp32 and the approximate exponential, then one rounding to bf16
    assert ((out - want).abs() <= 2.0 ** -20 + 2.0 ** -8 * abs(want)).all()
    ops.raise_on_device_error()
