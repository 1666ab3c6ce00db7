"""Row-per-warp norms, RoPE in sixteen-byte pieces and argmax with several accesses ahead, against the CPU statement of the same
operators, around the sizes where the kernels change."""
import pytest
import torch

from nkipy_b200 import ops

pytestmark = pytest.mark.gpu


def rnd(*shape, seed=0, s=1.0):
    return (s * torch.randn(shape, generator=torch.Generator().manual_seed(seed + sum(shape)))).to(torch.bfloat16)


def close(got, want):
    # both round once to bf16; the fp32 value before that may differ by the order of a sum and an approximate square root
    got, want = got.float().cpu(), want.float()
    assert ((got - want).abs() <= 2.0 ** -7 * want.abs() + 1e-6).all()


@pytest.mark.parametrize("rows", [1023, 1024, 1027, 2500])
@pytest.mark.parametrize("hidden", [8, 264, 1024, 2048, 2056, 2880, 4096, 4104])
@pytest.mark.parametrize("residual", [False, True])
def test_norms(rows, hidden, residual):
    x, r, w = rnd(rows, hidden), rnd(rows, hidden, seed=1), rnd(hidden, seed=2)
    want = ops.add_rmsnorm(x, w, residual_in=r if residual else None)
    got = ops.add_rmsnorm(x.cuda(), w.cuda(), residual_in=r.cuda() if residual else None)
    if residual:
        assert torch.equal(got[0].cpu(), want[0])
    close(got[1], want[1])


@pytest.mark.parametrize("hidden,splits", [(4096, 8), (4096, 3), (2880, 5), (8200, 2)])
def test_norm_of_partials(hidden, splits):
    p = torch.randn((splits, 9, hidden), generator=torch.Generator().manual_seed(4))
    r, w, b = rnd(9, hidden), rnd(hidden, seed=2), rnd(hidden, seed=3)
    want = ops.add_rmsnorm(None, w, residual_in=r, partials=p, bias=b)
    got = ops.add_rmsnorm(None, w.cuda(), residual_in=r.cuda(), partials=p.cuda(), bias=b.cuda())
    # sums in another order may round the stream differently
    assert ((got[0].float().cpu() - want[0].float()).abs() <= 2.0 ** -7 * want[0].float().abs() + 1e-5).all()
    assert (got[1].float().cpu() - want[1].float()).norm() <= 2.0 ** -8 * want[1].float().norm()


@pytest.mark.parametrize("tokens", [255, 256, 301])
@pytest.mark.parametrize("dim,nq,nkv", [(64, 6, 2), (128, 4, 1), (128, 5, 2), (256, 2, 1)])
@pytest.mark.parametrize("splits", [0, 3])
@pytest.mark.parametrize("norm,bias,shift", [(True, True, 0), (False, False, 0), (False, True, 1)])
def test_rope_append(tokens, dim, nq, nkv, splits, norm, bias, shift):
    """shift 1: a bias that does not start on sixteen bytes (the general kernel)."""
    width, bs, blocks = (nq + 2 * nkv) * dim, 32, 12
    qkv = (torch.randn((splits, tokens, width), generator=torch.Generator().manual_seed(dim)) if splits
           else rnd(tokens, width, seed=dim))
    pos = torch.randint(0, 700, (tokens,), generator=torch.Generator().manual_seed(1)).to(torch.int32)
    slots = torch.randperm(blocks * bs, generator=torch.Generator().manual_seed(2))[:tokens].to(torch.int32)
    slots[5] = -1
    table = ops.rope_table(dim, 700)
    qw, kw = (rnd(dim, seed=5), rnd(dim, seed=6)) if norm else (None, None)
    b = rnd(width + 1, seed=7)[shift:shift + width] if bias else None
    outs = []
    for dev in ("cpu", "cuda"):
        k = torch.zeros((blocks, nkv, bs, dim), dtype=torch.bfloat16, device=dev)
        v = torch.zeros_like(k)
        to = lambda t: None if t is None else t.to(dev)
        bd = None if b is None else rnd(width + 1, seed=7).to(dev)[shift:shift + width]
        q = ops.rope_kv_append(qkv.to(dev), pos.to(dev), slots.to(dev), table.to(dev), k, v, nq, nkv, dim, bias=bd, q_norm_w=to(qw),
                               k_norm_w=to(kw), norm_eps=1e-6)
        outs.append((q, k, v))
    for got, want in zip(outs[1], outs[0]):
        got, want = got.float().cpu(), want.float()
        # the norm is rounded to bf16 before the rotation: a rounding that falls the other way is a unit of either operand
        assert ((got - want).abs() <= 2.0 ** -6 * want.abs() + 2.0 ** -6).all()
        assert (got - want).norm() <= 2.0 ** -8 * want.norm()


@pytest.mark.parametrize("rows,vocab", [(1, 128256), (3, 4099), (2, 8), (5, 1003), (1, 201088)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_argmax(rows, vocab, dtype):
    z = torch.randn((rows, vocab), generator=torch.Generator().manual_seed(vocab)).to(dtype)
    z[0, vocab - 1] = z[0, vocab // 2] = 50.0         # a tie: the first wins
    assert torch.equal(ops.argmax(z.cuda()).cpu().long(), z.float().argmax(-1))
    z[0, vocab // 2 - 1] = float("nan")               # loses against any number
    z[rows - 1, :] = -0.0
    z[rows - 1, vocab // 3:] = 0.0                    # zeros of either sign are a tie
    got = ops.argmax(z.cuda()).cpu().tolist()
    assert got[rows - 1] == 0 and (rows == 1 or got[0] == vocab // 2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_argmax_of_rows_masked_with_the_lowest_value(dtype):
    low = torch.finfo(dtype).min
    z = torch.full((3, 4096), low, dtype=dtype)
    z[1, 4093], z[2, 5], z[2, 6:] = low / 2, 0.0, float("-inf")
    assert ops.argmax(z.cuda()).cpu().tolist() == [0, 4093, 5]


@pytest.mark.parametrize("hidden", [8, 72, 256, 260, 2048])
@pytest.mark.parametrize("tokens,experts,k", [(1, 4, 1), (37, 8, 3), (130, 12, 9), (1501, 16, 7)])
def test_expert_rows_and_their_sums(tokens, experts, k, hidden):
    """Pairs around whole blocks of four, more pairs per token than are on their way at a time, rows with and without whole pieces."""
    g = torch.Generator().manual_seed(tokens + hidden)
    ids = torch.stack([torch.randperm(experts, generator=g)[:k] for _ in range(tokens)]).to(torch.int32)
    x, w = rnd(tokens, hidden), torch.rand((tokens, k), generator=g)
    lo, local = 1, experts - 1                         # the first expert is another rank's
    here = (ids >= lo).flatten()
    for scale in (None, w):
        rows, offsets, pos = ops.moe_dispatch(x.cuda(), ids.cuda(), lo, local, weights=None if scale is None else scale.cuda())
        at, n = pos.cpu().long().flatten(), int(here.sum())
        assert offsets[-1] == n and (at[~here] == -1).all() and at[here].sort().values.tolist() == list(range(n))
        want = x.repeat_interleave(k, 0)[here]
        if scale is not None:
            want = (scale.flatten()[here, None] * want.float()).to(torch.bfloat16)
        assert torch.equal(rows.cpu()[at[here]], want)
        by_row = torch.empty(n, dtype=torch.int32)
        by_row[at[here]] = ids.flatten()[here]
        assert torch.equal(by_row, by_row.sort().values)
    if hidden % 8 == 0:
        rows, _, pos = ops.moe_dispatch(x.cuda(), ids.cuda(), lo, local)
        got = ops.moe_combine(rows, pos, w.cuda(), tokens).double().cpu()
        terms = (w * here.view(tokens, k)).double()[:, :, None] * x.double()[:, None]
        # k products summed in 32 bits, then one rounding to bf16
        assert ((got - terms.sum(1)).abs() <= (2.0 ** -8 + k * 2.0 ** -23) * terms.abs().sum(1)).all()


@pytest.mark.parametrize("experts,k,splits", [(8, 2, 1), (32, 4, 3), (60, 5, 20), (128, 8, 8), (128, 32, 17), (200, 6, 2), (1000, 8, 4)])
@pytest.mark.parametrize("mode", ["softmax_topk", "topk_softmax", "sigmoid_topk"])
def test_router_picks(experts, k, splits, mode):
    """Partial sums around what is loaded ahead, experts per lane of every instance, ties, infinities and a NaN."""
    g = torch.Generator().manual_seed(experts + splits)
    z = torch.randn((splits, 37, experts), generator=g)
    z[:, 3] = 0.0
    z[0, 3, 1::2] = -0.0                              # zeros of either sign are a tie: the first experts
    z[0, 5, experts // 2], z[0, 6, 1] = float("-inf"), float("nan")
    w, e = ops.router_topk(z.cuda(), k, mode)
    total = z[0].clone()
    for s in range(1, splits):
        total += z[s]                                 # in the kernel's order
    order = total.nan_to_num(nan=-3e38, neginf=-3.3e38).sort(dim=-1, descending=True, stable=True).indices[:, :k]
    rows = [i for i in range(37) if not (experts == k and i in (5, 6))]
    assert torch.equal(e.cpu().long()[rows], order[rows])
    top = total.double().gather(1, order)
    keep = total.double().masked_fill(total.isnan(), float("-inf"))
    want = top.sigmoid() if mode == "sigmoid_topk" else (top - keep.amax(-1, keepdim=True)).exp()
    if mode != "sigmoid_topk":
        want = want / want.sum(-1, keepdim=True)
    # exponentials of 32-bit differences of a few units, a sum of k and a division
    assert ((w.cpu().double() - want).abs() <= 64 * 2.0 ** -24 * want + 1e-12)[rows].all()
