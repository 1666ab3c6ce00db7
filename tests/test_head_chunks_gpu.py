"""Recurrences with one decay per head over prompts: against the same recurrence in 64 bits at the edges of sixteen tokens, of columns and
of channels, and whatever the caller says of the lengths."""
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

    def run(self, chunks):
        """(results before norm and gate, state); chunks False: token by token."""
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
                              i32([n + d for n, d in zip(self.lens, self.done)]), parts=1, gate_act="none", q_start=i32(starts),
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
@pytest.mark.parametrize("delta", [True, False], ids=["delta", "space"])
@pytest.mark.parametrize("heads,dim,lens", [(16, 128, [1, 15, 16, 17, 96, 130]), (4, 64, [100, 300])])
def test_what_is_known_of_the_lengths_changes_no_bit(dtype, delta, heads, dim, lens):
    p = Problem(dtype, delta, heads, heads, dim, dim, lens, [3] * len(lens))
    (o, s), (o1, s1) = p.run(True), p.run(False)
    assert torch.equal(o, o1) and torch.equal(s, s1)
