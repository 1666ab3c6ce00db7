"""Tiles of the grouped products where a rank holds some of the experts."""
import types

import pytest
import torch

from nkipy_b200 import ops
from nkipy_b200.models import config as C
from nkipy_b200.models.moe import MoEBlock
from nkipy_b200.parallel.comm import TPGroup


@pytest.mark.parametrize("ranks,tokens,widths", [(1, 128, (32, 32)), (8, 128, (32, 32)), (4, 256, (32, 32)), (2, 512, (32, 32)),
                                                 (8, 1023, (64, 128)), (8, 1024, (256, 256)), (1, 1024, (256, 256))])
@pytest.mark.parametrize("last", [False, True])
def test_width_follows_the_rows_of_an_expert(monkeypatch, ranks, tokens, widths, last):
    """128 experts, 8 per token: 256-row tiles from 1024 tokens (64 rows per expert) on, on however many ranks."""
    cfg = C.qwen3_30b_a3b(num_layers=1, hidden_size=64, moe_intermediate_size=8)
    block = MoEBlock(cfg, TPGroup(ranks - 1 if last else 0, ranks))
    seen = {}
    dispatch = ops.moe_dispatch

    def spy(x, experts, lo, local, **kw):
        seen["widths"] = ops.moe_tile_widths(tokens, ops.rows_per_expert(experts.numel(), lo, local, kw.get("num_experts", 0)))
        return dispatch(x, experts, lo, local, **kw)

    monkeypatch.setattr(ops, "moe_dispatch", spy)
    rnd = lambda *shape: torch.randn(shape, generator=torch.Generator().manual_seed(sum(shape))).to(torch.bfloat16)
    n = block.num_local
    lw = types.SimpleNamespace(router=rnd(128, 64), router_bias=None, gate_up=rnd(n, 16, 64), down=rnd(n, 64, 8), gate_up_bias=None,
                               down_bias=None)
    block._experts(lw, rnd(tokens, 64))
    assert seen["widths"] == widths


def test_pair_tiles_refuse_arrival_counters():
    x, w = torch.zeros((4, 64), dtype=torch.bfloat16), torch.zeros((1, 256, 64), dtype=torch.bfloat16)
    offsets = torch.tensor([0, 4], dtype=torch.int32)
    with pytest.raises(ValueError):
        ops.grouped_linear(x, w, offsets, max_rows_per_group=4, tiles={256: (None, None, 1)}, arrive=1, arrive_target=1)


@pytest.mark.gpu
@pytest.mark.parametrize("lo,tokens,wide", [(0, 128, False), (12, 128, False), (0, 600, True), (8, 600, True), (12, 600, True)])
def test_some_of_the_experts(lo, tokens, wide):
    """Four of sixteen experts: the products of their rows, and the form chosen; most rows of the sorted buffer stay unused."""
    g = torch.Generator(device="cuda").manual_seed(tokens + lo)
    rnd = lambda *shape, s=1.0: (s * torch.randn(shape, generator=g, device="cuda")).to(torch.bfloat16)
    x, w = rnd(tokens, 264), rnd(4, 2 * 136, 264, s=0.1)
    pick = torch.rand((tokens, 16), generator=g, device="cuda").argsort(1)[:, :2].to(torch.int32)
    plan = ops.moe_dispatch(x, pick, lo, 4, num_experts=16)
    assert (256 in plan.tiles) == wide
    off = plan.offsets.tolist()
    assert 0 < off[-1] < tokens * 2
    plan.x_sorted[off[-1]:] = float("nan")
    out = torch.full((tokens * 2, 136), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.grouped_linear(plan.x_sorted, w, plan.offsets, max_rows_per_group=tokens, gated=True, tiles=plan.tiles, out=out)
    for e in range(4):
        z = plan.x_sorted[off[e]:off[e + 1]].double() @ w[e].double().T
        want = torch.nn.functional.silu(z[:, :136]) * z[:, 136:]
        # one rounding to bf16; sums and the approximate exponential are far below it
        assert ((out[off[e]:off[e + 1]].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-3).all()
    assert (out[off[-1]:] == 7).all()
    ops.raise_on_device_error()
