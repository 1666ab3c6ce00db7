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


@pytest.mark.gpu
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("batch,nq,nkv", [(3, 16, 1), (5, 6, 2), (40, 32, 4), (75, 64, 8)])
@pytest.mark.parametrize("splits", [1, 4, 5, 8, 11])
@pytest.mark.parametrize("offset", [0, 1])
def test_rows_of_the_newest_token(D, batch, nq, nkv, splits, offset):
    """Rows shared out among all warps of a CTA, for every number of CTAs per SM: as many partial sums as a round holds and more, also
    where two do not lie on eight bytes, give bit by bit what their sum gives as one."""
    g = torch.Generator(device="cuda").manual_seed(batch + splits)
    W, ctx = (nq + 2 * nkv) * D, 70
    # small multiples of 1/64: their sums are exact in any order
    parts = torch.randint(-8, 9, (splits, batch, W), generator=g, device="cuda").float() / 64
    flat = torch.zeros(parts.numel() + offset, device="cuda")
    flat[offset:] = parts.flatten()
    tab = ops.rope_table(D, 128, device="cuda")
    w = torch.randn(2, D, generator=g, device="cuda").bfloat16()
    at = torch.full((batch,), ctx - 1, dtype=torch.int32, device="cuda")
    table = torch.arange(3 * batch, dtype=torch.int32, device="cuda").view(batch, 3)
    slots = table[:, 2] * 32 + (ctx - 1) % 32
    kv = torch.randn(2, 3 * batch, nkv, 32, D, generator=g, device="cuda").bfloat16()
    got = []
    for x in (flat[offset:].view(splits, batch, W), parts.sum(0, keepdim=True)):
        k, v = kv.clone().unbind()
        o = ops.rope_attn_decode(x, at, slots, tab, k, v, table, at + 1, D ** -0.5, nq, nkv, q_norm_w=w[0], k_norm_w=w[1])
        got.append((o, k, v))
    ops.raise_on_device_error()
    assert all(torch.equal(a, b) for a, b in zip(*got)) and not torch.equal(got[0][1], kv[0])
