"""CTA-pair products split over k, and the plan of a packed step's projections."""
import pytest
import torch

from nkipy_b200 import ops


@pytest.mark.gpu
@pytest.mark.parametrize("m", [129, 255, 256, 257, 414])
@pytest.mark.parametrize("n,k,splits", [(256, 512, 2), (300, 4096, 3), (2880, 1032, 5), (4096, 14336, 8)])
def test_split_sums(m, n, k, splits):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x = torch.randn((m, k + 8), generator=g, device="cuda").to(torch.bfloat16)[:, :k]
    w = torch.randn((n, k), generator=g, device="cuda").to(torch.bfloat16)
    parts = ops.linear(x, w, swap=False, splits=splits)
    assert parts.dtype == torch.float32 and parts.shape[1:] == (m, n) and 1 < parts.shape[0] <= splits
    want = x.double() @ w.double().T
    # exact products summed in 32 bits, at most k roundings of values below the sum of the absolute products
    bound = k * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)
    assert ((parts.double().sum(0) - want).abs() <= bound).all()
    ops.raise_on_device_error()


@pytest.mark.gpu
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("m", [129, 200, 300, 500])
def test_whole_products_of_middle_sizes(m, gated):
    """Either kernel of the rule, with the epilogues a packed step uses."""
    g = torch.Generator(device="cuda").manual_seed(m)
    n, k = 520, 384
    x = torch.randn((m, k), generator=g, device="cuda").to(torch.bfloat16)
    w = (0.05 * torch.randn((2 * n if gated else n, k), generator=g, device="cuda")).to(torch.bfloat16)
    bias, res = None, None
    want = x.double() @ w.double().T
    if gated:
        want = torch.nn.functional.silu(want[:, :n]) * want[:, n:]
    else:
        bias = torch.randn((n,), generator=g, device="cuda").to(torch.bfloat16)
        res = torch.randn((m, n), generator=g, device="cuda").to(torch.bfloat16)
        want = want + bias.double() + res.double()
    y = ops.linear(x, w, swap=False, gated=gated, bias=bias, residual=res)
    # one rounding to bf16, and the approximate exponential of the gate
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-3).all()


def test_plan_leaves_no_split_empty():
    for rows in (1, 64, 128, 129, 257, 512, 1500, 5000):
        for cols, k in ((256, 64), (300, 128), (4096, 1032), (4096, 14336), (22016, 4096)):
            swap, splits = ops.prefill_plan(rows, cols, k)
            slabs = -(-k // 64)
            assert swap == (rows <= 128) and 1 <= splits <= 8
            assert splits == 1 or swap or -(-slabs // -(-slabs // splits)) == splits


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,experts,top,width,inner", [(300, 4, 2, 256, 136), (1500, 5, 2, 264, 384), (257, 3, 3, 512, 104)])
@pytest.mark.parametrize("limit", [0.0, 7.0])
def test_grouped_products_on_pairs(tokens, experts, top, width, inner, limit):
    """Experts with at least 64 rows on average: unequal groups, one of them empty, sizes off the tiles, biases and clamped gates."""
    g = torch.Generator(device="cuda").manual_seed(tokens)
    rnd = lambda *shape, s=1.0: (s * torch.randn(shape, generator=g, device="cuda")).to(torch.bfloat16)
    x, w1, w2 = rnd(tokens, width), rnd(experts, 2 * inner, width, s=0.1), rnd(experts, width, inner, s=0.1)
    b1, b2 = rnd(experts, 2 * inner), rnd(experts, width)
    pick = torch.rand((tokens, experts), generator=g, device="cuda").argsort(1)[:, :top].to(torch.int32)
    if experts > top:
        pick[pick == experts - 1] = 0                 # an empty group, and a token that names one expert twice
    plan = ops.moe_dispatch(x, pick, 0, experts)
    assert 256 in plan.tiles
    off = plan.offsets.tolist()
    h = ops.grouped_linear(plan.x_sorted, w1, plan.offsets, max_rows_per_group=tokens, gated=True, bias=b1, act_limit=limit,
                           tiles=plan.tiles)
    y = ops.grouped_linear(h, w2, plan.offsets, max_rows_per_group=tokens, bias=b2, tiles=plan.tiles)
    for e in range(experts):
        rows = slice(off[e], off[e + 1])
        z = plan.x_sorted[rows].double() @ w1[e].double().T + b1[e].double()
        a, u = z[:, :inner], z[:, inner:]
        if limit:
            a, u = a.clamp(max=limit), u.clamp(-limit, limit) + 1
            want = u * a * torch.sigmoid(1.702 * a)
        else:
            want = torch.nn.functional.silu(a) * u
        # one rounding to bf16; sums and the approximate exponential are far below it
        assert ((h[rows].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-3).all()
        want = h[rows].double() @ w2[e].double().T + b2[e].double()
        assert ((y[rows].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-3).all()
    ops.raise_on_device_error()


@pytest.mark.gpu
def test_one_partial_of_a_requested_split():
    """Splits of a contraction of one slab are one partial, in fp32."""
    x, w = torch.randn((130, 64), device="cuda").to(torch.bfloat16), torch.randn((256, 64), device="cuda").to(torch.bfloat16)
    y = ops.linear(x, w, swap=False, splits=4)
    assert y.shape == (1, 130, 256) and y.dtype == torch.float32
    assert ((y[0] - x.double() @ w.double().T).abs() <= 64 * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)).all()
    ops.raise_on_device_error()


@pytest.mark.gpu
@pytest.mark.parametrize("width", [32, 64, 96, 128, 160, 192, 224])
@pytest.mark.parametrize("m,n,k", [(257, 256, 192), (130, 1000, 264), (600, 4104, 64)])
def test_tile_widths(width, m, n, k):
    """The width of a tile only says which CTA computes a value: every form gives the bits of the widest tile."""
    from nkipy_b200.ops import _lib

    g = torch.Generator(device="cuda").manual_seed(m + width)
    bf = lambda *shape: torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
    x, w, bias, res = bf(m, k), bf(2 * n, k), bf(n), bf(m, n)

    def run(tile_n, gated, act, splits, b=None, r=None):
        pad = 8                                        # a row pitch: columns behind the result stay as they are
        out = torch.full((splits, m, n + pad), 7.0, dtype=torch.float32 if splits > 1 else torch.bfloat16, device="cuda")
        rc = _lib.lib().nkb_gemm_bf16_2cta(x.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, k, k, n + pad,
                                           b.data_ptr() if b is not None else None, r.data_ptr() if r is not None else None, int(gated),
                                           n if gated else 0, act, 0.0, 0.0, splits, m * (n + pad) if splits > 1 else 0, 1, tile_n,
                                           torch.cuda.current_stream().cuda_stream)
        assert rc == 0 and (out[..., n:] == 7).all()
        return out

    res = torch.nn.functional.pad(res, (0, 8))         # rows of the residual lie as those of the output
    forms = [(False, 0, 1), (False, 2, 1), (True, 0, 1), (True, 1, 1)] + ([(False, 0, 2)] if k > 64 else [])
    for form in forms:
        assert torch.equal(run(width, *form), run(256, *form)), form
    assert torch.equal(run(width, False, 0, 1, bias, res), run(256, False, 0, 1, bias, res))
    ops.raise_on_device_error()
