"""Filtering and sampling of wide rows against float64: thresholds by rank and by mass in every combination, ties, masked entries,
penalties with repeats, rows to skip, vocabularies that leave blocks of a row without entries or a last slice short."""
import math

import numpy as np
import pytest
import torch

from test_gpu_kernels import DEV, _ops

pytestmark = pytest.mark.gpu


def _filtered(x, inv_t, k, top_p, min_p, pen, history):
    """(float64 row, kept entries, entries whose fate float32 rounding may decide)."""
    x = x.astype(np.float64).copy()
    for t in history:
        if 0 <= t < len(x):
            x[t] = x[t] * pen if x[t] <= 0 else x[t] / pen
    keep, near = np.isfinite(x), np.zeros(len(x), dtype=bool)
    v = x.astype(np.float32).astype(np.float64) * inv_t
    order = np.lexsort((np.arange(len(x)), -v))
    if 0 < k < len(x):
        keep[order[k:]] = False
    if top_p < 1 or min_p > 0:
        p = np.where(keep, np.exp(v - v[keep].max()), 0.0)
        total = p.sum()
        if min_p > 0:
            near |= np.abs(p - min_p) < 1e-5 * min_p
            keep &= p >= min_p
        if top_p < 1:
            before = np.zeros(len(x))
            before[order] = np.cumsum(np.where(keep, p, 0.0)[order]) - np.where(keep, p, 0.0)[order]
            # a chain of float32 sums over up to 120,818 terms: their order's rounding, at most vocab * 2^-24 of the mass, in practice its root
            near |= np.abs(before - top_p * total) < 1e-5 * total
            keep &= before < top_p * total
    return x, keep, near


@pytest.mark.parametrize("vocab", [7, 300, 8193, 120818])
@pytest.mark.parametrize("k, top_p, min_p", [(1, 1.0, 0.0), (20, 0.6, 0.0), (50, 0.9, 0.05), (1000, 0.95, 0.0), (1500, 0.9, 0.0), (0, 0.8, 0.0), (0, 1.0, 0.02),
                                             (5000, 1.0, 0.0), (3, 1.0, 0.3)])
def test_filters_of_wide_rows(vocab, k, top_p, min_p):
    ops = _ops()
    rng = np.random.default_rng(vocab + k)
    rows = 4
    x = (rng.standard_normal((rows, vocab)) * 2.5).astype(np.float32)
    x[1] = np.round(x[1] * 2) / 2                       # many ties, at the threshold too
    x[2, rng.random(vocab) < 0.4] = -np.inf             # entries that are masked from the start
    x[3, : vocab // 2] = 0.25                            # half of the row one value
    history = rng.integers(0, vocab, (rows, 16)).astype(np.int32)
    history[:, 3:6] = history[:, :1]                     # a token that was said four times
    history[:, 10] = -1
    f32 = lambda v: torch.full((rows,), v, dtype=torch.float32, device=DEV)
    inv_t = np.float32(1.0) / np.float32(0.7)
    wide = torch.empty((rows + 1, vocab + 3), device=DEV)       # rows with a stride, one of them to skip
    logits = wide[:, :vocab]
    logits.copy_(torch.from_numpy(np.concatenate([x, x[:1]])).to(DEV))
    skipped = logits[4].clone()
    row_map = torch.tensor([0, 1, 2, 3, -1], dtype=torch.int32, device=DEV)
    ops.filter_logits(logits, f32(float(inv_t)), torch.full((rows,), k, dtype=torch.int32, device=DEV), f32(top_p), f32(min_p), f32(1.1),
                      torch.from_numpy(history).to(DEV), row_map)
    got = logits.cpu().numpy()
    for r in range(rows):
        want, keep, near = _filtered(x[r], float(inv_t), k, top_p, min_p, float(np.float32(1.1)), history[r])
        kept = np.isfinite(got[r])
        if top_p == 1.0 and min_p == 0.0:
            assert (kept == keep).all()
        elif r == 1 or r == 3:    # entries of one value are kept in index order: only their number may hang on rounding
            assert abs(int(kept.sum()) - int(keep.sum())) <= int(near.sum())
            differ = np.nonzero(kept != keep)[0]
            assert len(np.unique(want[differ])) <= 1
            for value in np.unique(want[differ]):
                flags = kept[(want == value) & np.isfinite(x[r])]
                assert (flags[:-1] >= flags[1:]).all()
        else:
            assert ((kept == keep) | near).all()
        both = kept & keep
        assert np.allclose(got[r][both], want[both], rtol=1e-6, atol=0)      # four float32 divisions at most
    assert torch.equal(logits[4], skipped)


@pytest.mark.parametrize("vocab", [5, 1025, 65536, 120818])
def test_draws_from_wide_rows_fall_into_their_interval(vocab):
    from plain.hunyuan_plain import Xoshiro256StarStar
    ops = _ops()
    torch.manual_seed(vocab)
    logits = torch.randn(2, vocab, device=DEV) * 3
    logits[1, torch.rand(vocab, device=DEV) < 0.9] = -math.inf
    logits[1, vocab - 1] = 1.0
    cdf = torch.softmax(logits.double() / 0.7, dim=1).cumsum(1).cpu().numpy()
    states = torch.zeros(2, 4, dtype=torch.int64, device=DEV)
    ops.seed_rng(states, torch.arange(2, dtype=torch.int32, device=DEV), torch.tensor([5, 6], dtype=torch.int64, device=DEV))
    refs = [Xoshiro256StarStar(5), Xoshiro256StarStar(6)]
    out = torch.empty(2, dtype=torch.int32, device=DEV)
    inv_t = torch.full((2,), 1 / 0.7, device=DEV)
    for _ in range(200):
        ops.sample(out, logits, inv_t, states)
        for r, tok in enumerate(out.tolist()):
            u = float(refs[r].next_single())
            assert np.isfinite(logits[r, tok].item())
            assert (cdf[r][tok - 1] if tok else 0.0) - 1e-5 <= u <= cdf[r][tok] + 1e-5


@pytest.mark.parametrize("vocab, many", [(20000, 40), (120818, 104), (16999, 300)])
def test_draws_are_the_same_with_one_block_a_row_and_with_eight(vocab, many):
    ops = _ops()
    assert ops.sample_blocks(many, vocab) == 1 and ops.sample_blocks(8, vocab) == 8
    torch.manual_seed(vocab)
    logits = torch.randn(many, vocab, device=DEV) * 4
    logits[1, torch.rand(vocab, device=DEV) < 0.9] = -math.inf
    logits[2] = -math.inf
    logits[3, 5:] = -math.inf
    inv_t = torch.rand(many, device=DEV) + 0.5
    inv_t[4] = 0.0                                      # a greedy row is left alone
    rows = torch.arange(many, dtype=torch.int32, device=DEV)
    states = torch.zeros(many, 4, dtype=torch.int64, device=DEV)
    ops.seed_rng(states, rows, torch.arange(many, dtype=torch.int64, device=DEV) * 7 + 1)
    other = states.clone()
    for _ in range(40):
        one, eight = torch.full((many,), -9, dtype=torch.int32, device=DEV), torch.full((many,), -9, dtype=torch.int32, device=DEV)
        ops.sample(one, logits, inv_t, states)
        for at in range(0, many, 8):
            n = min(8, many - at)
            ops.sample(eight[at:at + n], logits[at:at + n], inv_t, other, rows[at:at + n].contiguous())
        assert torch.equal(one, eight) and torch.equal(states, other)
        assert one[4] == -9 and one[2] == 0


def test_draws_from_rows_too_wide_for_a_cluster_fall_into_their_interval():
    from plain.hunyuan_plain import Xoshiro256StarStar
    ops = _ops()
    vocab = 410000
    assert ops.sample_blocks(1, vocab) == 1
    torch.manual_seed(1)
    logits = torch.randn(1, vocab, device=DEV) * 3
    cdf = torch.softmax(logits.double() / 0.7, dim=1).cumsum(1).cpu().numpy()[0]
    states = torch.zeros(1, 4, dtype=torch.int64, device=DEV)
    ops.seed_rng(states, torch.zeros(1, dtype=torch.int32, device=DEV), torch.tensor([5], dtype=torch.int64, device=DEV))
    ref, out, inv_t = Xoshiro256StarStar(5), torch.empty(1, dtype=torch.int32, device=DEV), torch.full((1,), 1 / 0.7, device=DEV)
    for _ in range(50):
        ops.sample(out, logits, inv_t, states)
        tok, u = int(out[0]), float(ref.next_single())
        assert (cdf[tok - 1] if tok else 0.0) - 1e-5 <= u <= cdf[tok] + 1e-5


@pytest.mark.parametrize("vocab, many", [(9001, 24), (20000, 72)])
@pytest.mark.parametrize("k, top_p, min_p", [(1, 1.0, 0.0), (20, 0.6, 0.0), (50, 0.9, 0.05), (1500, 1.0, 0.02), (1500, 0.9, 0.0), (0, 0.8, 0.0), (0, 1.0, 0.02), (0, 1.0, 0.0)])
def test_filters_are_the_same_with_one_block_a_row_and_with_eight(vocab, many, k, top_p, min_p):
    ops = _ops()
    assert ops.filter_blocks(many, vocab) == 1 and ops.filter_blocks(4, vocab) == 8
    rng = np.random.default_rng(vocab + k)
    x = (rng.standard_normal((many, vocab)) * 2.5).astype(np.float32)
    x[1::4] = np.round(x[1::4] * 2) / 2                                  # ties, at the threshold too
    x[2, rng.random(vocab) < 0.4] = -np.inf
    history = rng.integers(0, vocab, (many, 16)).astype(np.int32)
    history[:, 3:6] = history[:, :1]
    f32 = lambda v: torch.full((many,), v, dtype=torch.float32, device=DEV)
    arguments = (f32(1 / 0.7), torch.full((many,), k, dtype=torch.int32, device=DEV), f32(top_p), f32(min_p), f32(1.1), torch.from_numpy(history).to(DEV))
    one, eight = torch.from_numpy(x).to(DEV), torch.from_numpy(x).to(DEV)
    ops.filter_logits(one, *arguments)
    rows = torch.arange(many, dtype=torch.int32, device=DEV)
    for at in range(0, many, 4):
        ops.filter_logits(eight[at:at + 4], *arguments, rows[at:at + 4].contiguous())
    if top_p == 1.0 or 0 < k <= 1024:        # nothing but counts, ranks and sums in one order
        assert torch.equal(one, eight)
        return
    one, eight = one.cpu().numpy(), eight.cpu().numpy()
    for r in range(many):                    # the mass per bin is added up in the order of the atomics
        want, keep, near = _filtered(x[r], float(np.float32(1 / 0.7)), k, top_p, min_p, float(np.float32(1.1)), history[r])
        differ = np.isfinite(one[r]) != np.isfinite(eight[r])
        assert (~differ | near).all()
        both = ~differ & np.isfinite(one[r])
        assert (one[r][both] == eight[r][both]).all()
