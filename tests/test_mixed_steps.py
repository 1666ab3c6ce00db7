"""Steps of an external scheduler: single tokens and portions in any order give what they give alone."""
import numpy as np
import pytest
import torch

from nkipy_b200 import ops
from nkipy_b200.models import config as C
from nkipy_b200.models.engine import GenerationEngine, StepEntry
from nkipy_b200.models.kv_cache import BLOCK_SIZE, OutOfBlocks
from nkipy_b200.models.transformer import TransformerLM
from nkipy_b200.models.weights import random_weights

DEVICES = ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)]


def engine(device, **kw):
    cfg = C.tiny(hidden_size=256, head_dim=64, num_heads=8, num_kv_heads=2, intermediate_size=512, vocab_size=512, num_layers=2)
    model = TransformerLM(cfg, random_weights(cfg, device=device, seed=1, std=0.05), device=device)
    return GenerationEngine(model, max_batch=6, max_seq_len=256, enable_prefix_sharing=False, **kw)


def ids(n, seed):
    return torch.randint(0, 512, (n,), generator=torch.Generator().manual_seed(seed)).tolist()


@pytest.mark.parametrize("device", DEVICES)
def test_any_order_of_singles_and_portions(device):
    prompts, news = [ids(n, n) for n in (70, 1, 33, 64, 5)], [ids(1, 90), ids(40, 91), ids(1, 92), ids(2, 93), ids(1, 94)]
    want = [[0], [39, 0], [0], [-1], [0]]
    alone = []
    for p, n, w in zip(prompts, news, want):
        e = engine(device)
        s = e.open_request()
        e.run_step([StepEntry(s, p)])
        # -1 counts from the end of the step's tokens
        alone.append(e.run_step([StepEntry(s, n + [7], [x % len(n) for x in w])]).float().cpu())
    e = engine(device)
    seqs = [e.open_request() for _ in prompts]
    for s, p in zip(seqs, prompts):
        e.run_step([StepEntry(s, p)])
    entries = [StepEntry(s, n, [x for x in w]) for s, n, w in zip(seqs, news, want)]
    entries[3].want = [1]
    got = e.run_step(entries).float().cpu()
    ref = torch.cat(alone)
    assert got.shape == ref.shape
    # bf16 activations in batches of other sizes
    assert (got - ref).norm() <= (2e-2 if device == "cuda" else 1e-2) * ref.norm()
    assert ((got - ref).norm(dim=1) <= 4e-2 * ref.norm(dim=1)).all()


@pytest.mark.parametrize("device", DEVICES)
def test_places_outside_a_step_are_refused(device):
    e = engine(device)
    s = e.open_request()
    with pytest.raises(IndexError):
        e.run_step([StepEntry(s, ids(4, 1), [4])])
    with pytest.raises(IndexError):
        e.run_step([StepEntry(s, ids(4, 1), [-5])])
    with pytest.raises(ValueError):
        e.run_step([StepEntry(s, [2 ** 40], [0])])
    assert s.num_computed == 0 and e.run_step([StepEntry(s, ids(4, 1), [-1])]).shape[0] == 1


@pytest.mark.parametrize("device", DEVICES)
def test_tables_and_lengths_follow_growth_and_release(device):
    """The device's block table and context lengths after steps that cross blocks, leave sequences out and give rows back."""
    e = engine(device)
    seqs = [e.open_request() for _ in range(4)]
    e.run_step([StepEntry(s, ids(BLOCK_SIZE - 2 + i, i)) for i, s in enumerate(seqs)])
    for step in range(5):
        out = [s for i, s in enumerate(seqs) if (i + step) % 3]
        before = {s.seq_id: s.num_computed for s in seqs}
        assert e.run_step([StepEntry(s, ids(1, step), [0]) for s in out]).shape[0] == len(out)
        for s in seqs:
            assert s.num_computed == before[s.seq_id] + (s in out) == len(s.tokens)
            assert int(e.context_lens[s.slot]) == s.num_computed
            assert e.cache.block_table[s.slot, :len(s.blocks)].tolist() == s.blocks
    e.release([seqs[0], seqs[2], seqs[3]])
    assert [int(e.context_lens[s.slot]) for s in seqs] == [-1, seqs[1].num_computed, -1, -1]
    free = e.cache.allocator.num_free()
    with pytest.raises((OutOfBlocks, RuntimeError)):
        e.run_step([StepEntry(seqs[1], ids(300, 1))])
    assert e.cache.allocator.num_free() == free


@pytest.mark.parametrize("device", DEVICES)
def test_places_are_those_of_their_entry(device):
    """In packed and in decode steps: negative places count from the entry's own end, a place wanted twice comes twice, and one
    outside the entry is refused before anything has changed."""
    e = engine(device)
    a, b = e.open_request(), e.open_request()
    p, q = ids(40, 1), ids(9, 2)
    both = e.run_step([StepEntry(a, p, [-1, 3, 39]), StepEntry(b, q, [-9, -1])]).float()
    assert both.shape[0] == 5
    a.num_computed = b.num_computed = 0
    same = e.run_step([StepEntry(a, p, [39, 3, 39]), StepEntry(b, q, [0, 8])]).float()
    assert torch.equal(both, same)
    free, tokens = e.cache.allocator.num_free(), (list(a.tokens), list(b.tokens))
    for entries in ([StepEntry(a, ids(100, 3), [0]), StepEntry(b, ids(2, 4), [2])], [StepEntry(a, [5], [0]), StepEntry(b, [6], [1])],
                    [StepEntry(a, [5], [-2])]):
        with pytest.raises(IndexError):
            e.run_step(entries)
        assert (a.tokens, b.tokens) == tokens and e.cache.allocator.num_free() == free
    once = e.run_step([StepEntry(a, [5], [0]), StepEntry(b, [6], [-1])])
    a.num_computed, b.num_computed = 40, 9
    many = e.run_step([StepEntry(a, [5], [0] * 70), StepEntry(b, [6], [0, 0])])
    assert once.shape[0] == 2 and torch.equal(many, once[[0] * 70 + [1] * 2])


@pytest.mark.parametrize("device", DEVICES)
def test_a_sequence_takes_the_tokens_of_another(device):
    """The tokens of an entry may be another sequence's list, which the step itself makes longer."""
    p = ids(12, 1)
    got = []
    for own in (False, True):
        e = engine(device)
        a, b, c = (e.open_request() for _ in range(3))
        e.run_step([StepEntry(a, p)])
        got.append(e.run_step([StepEntry(a, [7], [0]), StepEntry(b, a.tokens if own else list(p), [11]),
                               StepEntry(c, ids(20, 5), [0, 4])]).float())
        assert a.tokens == p + [7] and b.tokens == p and b.num_computed == 12
    assert torch.equal(*got)


@pytest.mark.parametrize("device", DEVICES)
def test_release_takes_any_iterable(device):
    e = engine(device)
    seqs = [e.open_request() for _ in range(4)]
    e.run_step([StepEntry(s, ids(40, i)) for i, s in enumerate(seqs)])
    e.release(s for s in seqs[:2])
    assert set(e.active) == {s.slot for s in seqs[2:]} and len(e.cache.sequences) == 2
    e.release(e.active.values())
    e.release(iter(()))
    assert not e.active and e.context_lens.tolist() == [-1] * 6


@pytest.mark.parametrize("device", DEVICES)
def test_release_after_a_failed_step(device, monkeypatch):
    """Rows whose lengths a decode step has brought over are inactive after their release, also where the step itself failed."""
    e = engine(device)
    seqs = [e.open_request() for _ in range(3)]
    e.run_step([StepEntry(s, ids(5, i), [4]) for i, s in enumerate(seqs)])

    def fails():
        raise RuntimeError("no memory")
    with monkeypatch.context() as m:
        m.setattr(e, "decode_step_device", fails)
        with pytest.raises(RuntimeError, match="no memory"):
            e.run_step([StepEntry(s, [9], [0]) for s in seqs[:2]])
    e.release(seqs)
    assert e.context_lens.tolist() == [-1] * 6


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("lens", [[1], [129], [1, 1, 1], [31, 33, 1, 64, 5], [1] * 70 + [300]])
def test_positions_of_packed_tokens(device, lens):
    """Positions and slots as counted out one by one, for new sequences and continued ones."""
    done = [(37 * i) % 90 for i in range(len(lens))]
    ends = [d + n for d, n in zip(done, lens)]
    table = torch.randperm(len(lens) * 13, generator=torch.Generator().manual_seed(1)).reshape(len(lens), 13)
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).to(device)
    pos, slots = ops.packed_positions(i32([sum(lens[:i]) for i in range(len(lens))]), i32(lens), i32(ends), i32(table), sum(lens))
    want = [(b, p) for b, (d, e) in enumerate(zip(done, ends)) for p in range(d, e)]
    assert pos.tolist() == [p for _, p in want]
    assert slots.tolist() == [int(table[b, p // BLOCK_SIZE]) * BLOCK_SIZE + p % BLOCK_SIZE for b, p in want]


@pytest.mark.parametrize("device", DEVICES)
def test_positions_refuse_what_does_not_fit(device):
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=device)
    good = dict(q_start=i32([0, 2]), q_lens=i32([2, 3]), context_lens=i32([2, 40]), block_table=i32([[1, 2], [3, 4]]), tokens=5)
    assert ops.packed_positions(**good)[0].tolist() == [0, 1, 37, 38, 39]
    for bad in (dict(q_lens=i32([2])), dict(context_lens=i32([2, 40, 1])), dict(block_table=i32([[1, 2]])), dict(tokens=-1), dict(block_size=0),
                dict(block_table=i32([[], []]))):
        with pytest.raises(ValueError):
            ops.packed_positions(**{**good, **bad})
    slots = ops.packed_positions(**good)[1].tolist()
    for part in (i32([[1, 2, 9], [3, 4, 9]])[:, :2], i32([[9, 1, 2], [9, 3, 4]])[:, 1:], i32([[1, 3], [2, 4]]).T):
        assert ops.packed_positions(**{**good, "block_table": part})[1].tolist() == slots
    for bad in (dict(q_lens=good["q_lens"].long()), dict(q_start=i32([0, 9, 2, 9])[::2])):
        with pytest.raises(TypeError):
            ops.packed_positions(**{**good, **bad})


def test_token_ids_of_all_kinds():
    """Lists, tuples, arrays and tensors, of whole numbers and of what stands for them, alone and beside one another."""
    e = engine("cpu")
    p = ids(5, 3)
    kinds = [p, tuple(p), np.array(p), np.array(p, dtype=np.uint8) if max(p) < 256 else np.array(p, dtype=np.int64), torch.tensor(p),
             [float(t) for t in p], [np.int64(t) for t in p], [torch.tensor(t) for t in p]]
    got = []
    for k in kinds:
        s = e.open_request()
        got.append(e.run_step([StepEntry(s, k, [4])]))
        assert s.tokens == p and all(type(t) is int for t in s.tokens)
        e.release([s])
    assert all(torch.equal(g, got[0]) for g in got)
    a, b = e.open_request(), e.open_request()
    assert torch.equal(e.run_step([StepEntry(a, kinds[0], [4]), StepEntry(b, kinds[4], [4])]), torch.cat([got[0]] * 2))
    for bad in ([2 ** 31], [-2 ** 31 - 1], [1, 2 ** 40]):
        with pytest.raises(ValueError):
            e.run_step([StepEntry(a, bad, [0])])
    assert a.num_computed == 5 and e.run_step([StepEntry(a, [np.int32(3)], [0])]).shape[0] == 1
