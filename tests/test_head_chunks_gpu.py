"""Recurrences with one decay per head by chunks of sixteen tokens: against the same recurrence in 64 bits, and against the kernel that
goes token by token, at the edges of chunks, columns and channels."""
import pytest
import torch

from nkipy_b200.ops import HeadRecurrence, Proj, ShortConv, head_recurrence

pytestmark = pytest.mark.gpu
DEV = "cuda"


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


class Problem:
    def __init__(self, dtype, delta, heads, groups, dim, vdim, lens, done, decay=-2.0, seed=0, pad=0):
        g = torch.Generator(device=DEV).manual_seed(seed)
        r = lambda *s, std=1.0, mean=0.0: torch.randn(s, generator=g, device=DEV) * std + mean
        self.dtype, self.delta, self.lens, self.done, T = dtype, delta, lens, done, sum(lens)
        C, H = 2 * groups * dim + heads * vdim, heads
        self.rec = HeadRecurrence(H, groups, dim, vdim, 0, groups * dim, 2 * groups * dim, torch.exp(r(H, std=0.1, mean=decay)),
                                  r(H, std=0.1, mean=-2.0), delta=delta, q_scale=dim ** -0.5, skip=None if delta else r(H))
        self.x = r(T, C).to(dtype)
        self.a, self.b = r(T, H).to(dtype), r(T, H).to(dtype) if delta else None
        self.conv = ShortConv(torch.ones(1, C, device=DEV))
        self.state = r(len(lens) + 1, *self.rec.state_shape, std=0.3)
        self.pad = pad

    def run(self, chunks, parts=1):
        """(results, each of `parts` parts of a row brought to size 1, and state); chunks False: token by token."""
        rec, T = self.rec, sum(self.lens)
        wide = torch.zeros(T, self.x.shape[1] + self.pad, dtype=self.dtype, device=DEV)
        wide[:, :self.x.shape[1]] = self.x
        x = Proj(wide, 0, self.x.shape[1])
        P = lambda t: None if t is None else Proj(t, 0, t.shape[1])
        state, ring = self.state.clone(), torch.zeros(len(self.lens) + 1, 1, self.x.shape[1], device=DEV)
        gate = Proj(torch.ones(T, rec.heads * rec.vdim, dtype=self.dtype, device=DEV), 0, rec.heads * rec.vdim)
        starts = [sum(self.lens[:i]) for i in range(len(self.lens))]
        # parts equal to the row's elements would lose the size: the norm over whole rows keeps what is compared here
        out = head_recurrence(rec, x, self.conv, P(self.a), P(self.b), gate, torch.ones(rec.heads * rec.vdim, device=DEV), state, ring,
                              i32([n + d for n, d in zip(self.lens, self.done)]), parts=parts, gate_act="none", q_start=i32(starts),
                              q_lens=i32(self.lens), rows=i32([i + 1 for i in range(len(self.lens))]), dtype=self.dtype,
                              max_q_len=0 if chunks else 1)
        torch.cuda.synchronize()
        assert torch.equal(state[0], self.state[0])
        return out, state

    def exact(self):
        rec, per = self.rec, self.rec.heads // self.rec.groups
        y = torch.nn.functional.silu(self.x.float()).to(self.dtype).double()
        G, d, H, n = rec.groups, rec.dim, rec.heads, rec.vdim
        q, k, v = y.split([G * d, G * d, H * n], -1)
        q, k, v = q.reshape(-1, G, d), k.reshape(-1, G, d), v.reshape(-1, H, n)
        if self.delta:
            q, k = (t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = ((t * s).repeat_interleave(per, 1) for t, s in ((q, rec.q_scale), (k, 1.0)))
        dt = torch.nn.functional.softplus(self.a.double() + rec.dt_bias.double(), threshold=100.0)
        g, outs, states, t = torch.exp(-rec.rate.double() * dt), [], [], 0
        for i, m in enumerate(self.lens):
            S = self.state[i + 1, :, :, :d].double() if self.done[i] else torch.zeros(H, n, d, dtype=torch.float64, device=DEV)
            for t in range(t, t + m):
                S = g[t][:, None, None] * S
                u = torch.sigmoid(self.b[t].double())[:, None] * (v[t] - torch.einsum("hnd,hd->hn", S, k[t])) if self.delta else \
                    dt[t][:, None] * v[t]
                S = S + u[:, :, None] * k[t][:, None, :]
                o = torch.einsum("hnd,hd->hn", S, q[t])
                outs.append(o if rec.skip is None else o + rec.skip.double()[:, None] * v[t])
            states.append(S)
            t += 1
        o = torch.stack(outs).flatten(1)
        return o / torch.sqrt(o.square().mean(-1, keepdim=True) + rec.eps), torch.stack(states)


def err(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "f32"])
@pytest.mark.parametrize("delta", [True, False], ids=["delta", "space"])
@pytest.mark.parametrize("heads,groups,dim,vdim,pad", [(2, 2, 128, 128, 0), (4, 2, 64, 64, 16), (3, 1, 40, 24, 8), (2, 1, 72, 136, 0),
                                                       (40, 40, 64, 96, 0)])
@pytest.mark.parametrize("decay", [-6.0, -2.0, 2.0])
def test_chunks(dtype, delta, heads, groups, dim, vdim, pad, decay):
    """Lengths around sixteen and its multiples, new and continued sequences; decays from almost none to almost all."""
    p = Problem(dtype, delta, heads, groups, dim, vdim, [1, 15, 16, 17, 96, 130], [0, 3, 0, 40, 7, 0], decay, pad=pad)
    (o, s), (o1, s1), (want, states) = p.run(True), p.run(False), p.exact()
    # sums of up to 130 tokens and 128 channels in 24 bits, decays of up to e^-7 from exponentials of two bits' error a token: 130 * 2^-24
    assert err(s[1:], states) < 8e-6 and err(s1[1:], states) < 8e-6
    assert err(o, want) < (4e-3 if dtype == torch.bfloat16 else 1.6e-5)          # two roundings to eight bits
    assert err(s, s1) < 8e-6 and err(o, o1) < (4e-3 if dtype == torch.bfloat16 else 1.6e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "f32"])
@pytest.mark.parametrize("delta", [True, False], ids=["delta", "space"])
def test_numbers_that_are_not_finite_stay_where_they_are(dtype, delta):
    """An infinite value and a NaN in the middle of a chunk reach what the recurrence token by token lets them reach."""
    p = Problem(dtype, delta, 2, 2, 128, 128, [100], [5])
    p.x[37, 2 * 2 * 128 + 9] = float("inf")                  # a value column of head 0
    p.x[70, 2 * 2 * 128 + 128 + 40] = float("nan")           # one of head 1
    (_, s), (_, s1) = p.run(True), p.run(False)
    assert torch.equal(torch.isfinite(s), torch.isfinite(s1)) and not torch.isfinite(s[1, 0, 9]).any()
    bad = ~torch.isfinite(s[1]).all(-1)
    assert bad.sum() == 2 and bad[0, 9] and bad[1, 40]
    keep = torch.isfinite(s)
    assert err(s[keep], s1[keep]) < 8e-6


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "f32"])
@pytest.mark.parametrize("heads,vdim", [(80, 16), (80, 128)])
@pytest.mark.parametrize("chunks", [True, False])
def test_products_of_two_32_bit_numbers(dtype, heads, vdim, chunks):
    """Errors of the two products that take numbers of 24 bits on both sides, (1 + A)^-1 b and P u, do not add up: their mean over the
    heads.  Two write strengths w just below 129/256, whose second parts are as large as they come, and powers of two otherwise."""
    d, n = 128, 96
    p = Problem(dtype, True, heads, 1, d, vdim, [n], [0])
    p.rec.rate.zero_()
    p.x.zero_()
    g = torch.Generator(device=DEV).manual_seed(7)
    p.b[:2] = (torch.rand(2, heads, generator=g, device=DEV) * 0.0077 + 0.0079).to(dtype)
    w = torch.sigmoid(p.b[:2].double())
    p.x[0, d] = 1024.0                                   # k_0 = (1, 0, ...)
    p.x[1, d:d + 4] = 1024.0                             # k_1 = (1, 1, 1, 1) / 2
    p.x[0, 2 * d:] = 64.0                                # v_0; the other tokens are zeros
    u = 64.0 * w[0]
    state = p.run(chunks)[1][1].double()                 # [heads, vdim, d]: second channel u_1 / 2 = -w_1 u_0 / 4
    off = (state[:, :, 1] / (-0.25 * w[1] * u)[:, None] - 1).mean()
    # a few roundings of 2^-25 each that average out, and the exponential's own bias within a ulp; six part products: -1.7e-7
    assert off.abs() < 2.0 ** -23.5
    if dtype == torch.float32:
        p.x[1, d:2 * d] = 0.0
        p.x[1, 0] = 1024.0                               # q_1 = (1, 0, ...): o_1 = q_scale u_0
        p.rec.q_scale = 129 / 128 - 2.0 ** -23           # its parts as large as they come
        p.b[0, :4] = 40.0                                # w = 1 where the row's norm is read from
        o = p.run(chunks)[0][1].double().view(heads, vdim)
        off = (o[4:] / (o[:4].mean() * w[0, 4:, None]) - 1).mean()
        # as above, and the norm's rounding of one number, 2^-24; six part products: -3e-7
        assert off.abs() < 2.0 ** -23 + 2.0 ** -24


# the rules that go by chunks (the state-space form of 32-bit models goes token by token), with four and with eight warps that hold states
forms = pytest.mark.parametrize("dtype,delta,heads", [(torch.bfloat16, True, 2), (torch.bfloat16, True, 40), (torch.bfloat16, False, 2),
                                                      (torch.bfloat16, False, 40), (torch.float32, True, 2)])


@forms
def test_tiny_states_and_values_keep_their_bits(dtype, delta, heads):
    """Numbers whose third bf16 parts would lie under bf16's smallest: states of some 2^-120 and values of the same size."""
    p = Problem(dtype, delta, heads, 1, 128, 128, [100, 40], [5, 0])
    p.state *= 2.0 ** -118
    p.x[:, 2 * 128:] *= 2.0 ** -118
    (_, s), (_, s1), (_, states) = p.run(True), p.run(False), p.exact()
    assert err(s[1:] * 2.0 ** 100, states * 2.0 ** 100) < 8e-6 and err(s1[1:] * 2.0 ** 100, states * 2.0 ** 100) < 8e-6


def alike(a, b):
    """Infinities and NaN in the same places, and the rest as close as sums in another order are."""
    keep = torch.isfinite(b)
    assert keep.any()
    return torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a[torch.isinf(b)], b[torch.isinf(b)]) and err(a[keep], b[keep]) < 5e-3


@forms
def test_infinite_states_stay_where_they_are(dtype, delta, heads):
    p = Problem(dtype, delta, heads, 1, 128, 128, [100, 40], [5, 7])
    p.state[1, 0, 9, 40] = float("inf")
    p.state[2, 1, 70, 3] = -float("inf")
    (o, s), (o1, s1) = p.run(True, heads), p.run(False, heads)     # rows of a head that are not affected stay numbers
    assert alike(s, s1) and alike(o, o1) and not torch.isfinite(s[1, 0, 9, 40]) and torch.isfinite(s[1, 0, 10]).all()


@forms
def test_infinite_keys_and_queries_reach_what_they_reach(dtype, delta, heads):
    p = Problem(dtype, delta, heads, heads, 128, 128, [100, 40], [5, 0])
    p.x[37, heads * 128 + 5] = float("inf")                  # a key of head 0
    p.x[70, 128 + 7] = float("inf")                          # a query of head 1
    p.x[120, heads * 128 + 128 + 3] = float("nan")           # a key of head 1
    p.x[131, heads * 128 + 9] = float("inf")                 # a key of head 0, whose first value is 0
    p.x[131, 2 * heads * 128] = 0.0
    (o, s), (o1, s1) = p.run(True, heads), p.run(False, heads)
    assert alike(s, s1) and alike(o, o1) and not torch.isfinite(s[1, 0, :, 5]).any() and torch.isfinite(s[1, 1]).all()


def test_tiny_32_bit_keys_keep_their_bits():
    p = Problem(torch.float32, True, 2, 1, 128, 128, [100, 40], [0, 0])
    p.x[:, :2 * 128] *= 2.0 ** -118
    (_, s), (_, s1), (_, states) = p.run(True), p.run(False), p.exact()
    assert err(s[1:] * 2.0 ** 100, states * 2.0 ** 100) < 8e-6 and err(s1[1:] * 2.0 ** 100, states * 2.0 ** 100) < 8e-6
