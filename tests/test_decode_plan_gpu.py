"""Decode attention divides the pages of ragged batches evenly among its CTAs: against one CTA per sequence, at the edges of the plan."""
import pytest
import torch

from nkipy_b200 import ops

pytestmark = pytest.mark.gpu


def case(lens, nq, nkv, D, q_len=1, seed=3):
    g = torch.Generator(device="cuda").manual_seed(seed)
    pages = [-(-n // 32) for n in lens]
    k, v = (torch.randn((sum(pages) + 1, nkv, 32, D), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    table = torch.zeros((len(lens), max(max(pages), 1)), dtype=torch.int32)
    order, at = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(seed)), 0
    for b, n in enumerate(pages):
        table[b, :n] = order[at:at + n]
        at += n
    q = torch.randn((len(lens) * q_len, nq * D), generator=g, device="cuda").to(torch.bfloat16)
    return q, k, v, table.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")


LENS = [[1], [31, 32, 33], [0, 70, 0, 1, 2000], [5000, 1, 1, 1, 1, 1, 1, 1], [640] * 6, [33 * i + 1 for i in range(40)], [4096, 4064, 2047]]


@pytest.mark.parametrize("lens", LENS, ids=lambda l: str(len(l)) + "x" + str(max(l)))
@pytest.mark.parametrize("nq,nkv,D", [(8, 2, 128), (2, 2, 64), (32, 8, 128), (6, 1, 64)])
@pytest.mark.parametrize("window,chunk", [(0, 0), (100, 0), (0, 256)])
def test_any_number_of_splits(lens, nq, nkv, D, window, chunk):
    q, k, v, table, ctx = case(lens, nq, nkv, D)
    sinks = torch.linspace(-1, 1, nq, device="cuda")
    run = lambda s: ops.paged_attn_decode(q, k, v, table, ctx, D ** -0.5, window=window, chunk=chunk, sinks=sinks, num_splits=s).float()
    want = run(1)
    for s in (0, 2, 3, 7, 16):
        # the same probabilities rounded to bf16 against another running maximum, then one rounding of the result
        assert ((run(s) - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -7).all(), s
        assert torch.equal(run(s), run(s))
    ops.raise_on_device_error()


@pytest.mark.parametrize("q_len", [2, 4])
def test_several_new_tokens(q_len):
    lens = [q_len, 900, 37, 3000]
    q, k, v, table, ctx = case(lens, 8, 2, 128, q_len)
    want = ops.paged_attn_decode(q, k, v, table, ctx, 0.1, q_len=q_len, num_splits=1).float()
    for s in (2, 5):
        got = ops.paged_attn_decode(q, k, v, table, ctx, 0.1, q_len=q_len, num_splits=s).float()
        assert ((got - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -7).all()


def test_lengths_change_under_a_captured_graph():
    """The plan is made from the lengths that a replay finds."""
    q, k, v, table, ctx = case([4000, 4000, 4000], 8, 2, 128)
    out = torch.empty_like(q)
    attend = lambda: ops.paged_attn_decode(q, k, v, table, ctx, 0.1, num_splits=3, out=out)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        attend()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            attend()
    torch.cuda.current_stream().wait_stream(side)
    for lens in ([4000, 4000, 4000], [1, 4000, 30], [0, 0, 77], [3, 2, 1]):
        ctx.copy_(torch.tensor(lens, dtype=torch.int32))
        graph.replay()
        want = ops.paged_attn_decode(q, k, v, table, ctx, 0.1, num_splits=1).float()
        assert ((out.float() - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -7).all(), lens
    ops.raise_on_device_error()
