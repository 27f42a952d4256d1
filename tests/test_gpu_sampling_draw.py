"""Rows whose token the filters draw on the way: the logits they leave, the token and the random stream's state are those of filter, argmax and
sample one after the other, bit for bit; rows that do not qualify are passed on."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, _ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [300, 5000, 40000, 120818])
@pytest.mark.parametrize("k, top_p, min_p", [(20, 0.6, 0.0), (1, 0.9, 0.0), (100, 1.0, 0.05), (1000, 0.95, 0.01), (1024, 0.5, 0.0), (1500, 0.9, 0.0), (0, 0.9, 0.0), (5, 1.0, 0.0)])
def test_a_draw_on_the_way_is_the_draw_behind(vocab, k, top_p, min_p):
    ops = _ops()
    torch.manual_seed(vocab + k)
    R = 9
    x = torch.randn(R, vocab, device=DEV) * 3
    x[1] = x[1].round()                              # ties, many of them beyond the k-th
    x[2] = 1.0                                       # more than 1,024 reach any edge
    x[3, 7:] = -math.inf                             # fewer than k that are finite
    x[4, 11], x[4, 200] = math.nan, math.inf         # what the draw leaves to the kernel behind
    x[5] = -math.inf
    f32 = lambda v: torch.full((R,), v, device=DEV)
    inv_t, top_k = f32(1 / 0.7), torch.full((R,), k, dtype=torch.int32, device=DEV)
    inv_t[6] = 0.0                                   # a greedy row
    row_map = torch.arange(R, dtype=torch.int32, device=DEV)
    row_map[7] = -1                                  # a row that is skipped
    history = torch.randint(0, vocab, (R, 16), dtype=torch.int32, device=DEV)
    seeds, outs = torch.arange(R, dtype=torch.int64, device=DEV) + 5, []
    for way in ("behind", "on the way"):
        logits, states = x.clone(), torch.zeros(R, 4, dtype=torch.int64, device=DEV)
        ops.seed_rng(states, torch.arange(R, dtype=torch.int32, device=DEV), seeds)
        tokens = []
        for step in range(3):
            y, out, drawn = logits.clone(), torch.full((R,), -5, dtype=torch.int32, device=DEV), torch.full((R,), 9, dtype=torch.int32, device=DEV)
            draw = None if way == "behind" else (out, states, drawn)
            ops.filter_logits(y, inv_t, top_k, f32(top_p), f32(min_p), f32(1.1), history, row_map, draw)
            flags = None if draw is None else drawn
            ops.argmax(out, y, row_map, None, flags)
            ops.sample(out, y, inv_t, states, row_map, flags)
            tokens.append(out)
        outs.append((y, torch.stack(tokens), states, None if draw is None else drawn))
    same = (outs[0][0] == outs[1][0]) | (outs[0][0].isnan() & outs[1][0].isnan())
    assert same.all() and torch.equal(outs[0][1], outs[1][1]) and torch.equal(outs[0][2], outs[1][2])
    drawn = outs[1][3].tolist()
    assert drawn[6] == 0 and drawn[7] == 0 and set(drawn) <= {0, 1}
    if 0 < k <= 1024 and k < vocab and (top_p < 1 or min_p > 0):
        assert drawn[0] == 1 and drawn[1] == 1 and drawn[4] == 0
    else:
        assert not any(drawn)


@pytest.mark.parametrize("rows, vocab", [(3, 9000), (20, 9000), (3, 3000), (160, 3000)])
@pytest.mark.parametrize("k", [1, 50, 512, 513, 1024])
@pytest.mark.parametrize("form", ["around zero", "far from zero", "on a grid", "flat", "few finite"])
def test_a_top_k_keeps_the_k_largest_whichever_way_it_goes(rows, vocab, k, form):
    """One block a row and eight, one block an SM and two; with the threads' largest spread over their bins, crowding one of them, and equal."""
    ops = _ops()
    torch.manual_seed(rows + k)
    x = torch.randn(rows, vocab, device=DEV)
    if form == "far from zero":
        x = x + 40
    elif form == "on a grid":
        x = (x * 8).round() / 8 + 40
    elif form == "flat":
        x = torch.full_like(x, -3.0)
    elif form == "few finite":
        x[:, 700:] = -math.inf
    f32 = lambda v: torch.full((rows,), v, device=DEV)
    y, top_k = x.clone(), torch.full((rows,), k, dtype=torch.int32, device=DEV)
    ops.filter_logits(y, f32(1.0), top_k, f32(1.0), f32(1e-38), None, None)      # (a min-p that drops nothing here)
    order = torch.sort(x, dim=1, descending=True, stable=True).indices[:, :k]    # ties in index order
    want = torch.full_like(x, -math.inf).scatter(1, order, x.gather(1, order))
    assert torch.equal(y, want)
