"""The gated delta rule in steps of several tokens: against the recurrence in float64 token by token (sequences that end anywhere in a
group of eight, channels and columns that fill their blocks and ones that do not, a state that was there, decays down to zero), and
bit for bit the same however the tokens are brought: together, alone, in portions, one at a time."""
import numpy as np
import pytest
import torch

from test_gpu_kernels import DEV, _ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads, kv_heads, dk, dv", [(2, 1, 128, 128), (3, 3, 8, 5), (2, 2, 33, 20), (4, 2, 64, 16), (1, 1, 200, 24)])
@pytest.mark.parametrize("news, start", [([2, 9, 1], 0), ([3, 16, 8], 5), ([4, 17, 7], 0), ([5, 40, 6], 9)])
def test_chunks_of_tokens(heads, kv_heads, dk, dv, news, start):
    ops = _ops()
    g = torch.Generator(device=DEV)
    g.manual_seed(dk * 100 + news[1])
    T, B = sum(news), len(news)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    q, k = rnd(T, kv_heads, dk), rnd(T, kv_heads, dk)
    q, k = q / q.norm(dim=-1, keepdim=True), k / k.norm(dim=-1, keepdim=True)
    v, beta = rnd(T, heads, dv), torch.sigmoid(rnd(T, heads))
    decay = torch.exp(-torch.exp(rnd(T, heads, dk) * 3 - 2))            # from 1 down to nothing
    decay[0, 0, 0] = 0.0
    state = rnd(B, heads, dk, dv) if start else torch.full((B, heads, dk, dv), float("nan"), device=DEV)
    want, left = torch.empty(T, heads, dv, dtype=torch.float64), []
    t = 0
    for b, n in enumerate(news):
        S = state[b].double().cpu() if start else torch.zeros(heads, dk, dv, dtype=torch.float64)
        for _ in range(n):
            kt = k[t].double().cpu().repeat_interleave(heads // kv_heads, 0)
            qt = q[t].double().cpu().repeat_interleave(heads // kv_heads, 0)
            S = S * decay[t].double().cpu()[:, :, None]
            u = beta[t].double().cpu()[:, None] * (v[t].double().cpu() - torch.einsum("hkd,hk->hd", S, kt))
            S = S + kt[:, :, None] * u[:, None]
            want[t] = torch.einsum("hkd,hk->hd", S, qt)
            t += 1
        left.append(S)
    out = torch.empty(T, heads * dv, device=DEV)
    rows = state.clone().view(B, -1).view(torch.uint8)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(news)]), dtype=torch.int32, device=DEV)
    ops.delta_scan(out, q.reshape(T, -1).contiguous(), k.reshape(T, -1).contiguous(), decay.reshape(T, -1).contiguous(), beta, v.reshape(T, -1).contiguous(), rows, 0,
                   cu, torch.arange(B, dtype=torch.int32, device=DEV), torch.tensor([start + n for n in news], dtype=torch.int32, device=DEV), B,
                   heads, kv_heads, dk, dv, max(news))
    # every token adds sums of dk products of entries of at most about 4, rounded at 2^-24 each, to what the ones before left
    bound = 4.0 * 2.0 ** -24 * (dk + 16) * max(news)
    assert (out.view(T, heads, dv).double().cpu() - want).abs().max() <= bound
    got = rows.view(torch.float32).view(B, heads, dk, dv).double().cpu()
    assert (got - torch.stack(left)).abs().max() <= bound


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads, kv_heads, dk, dv", [(16, 8, 128, 128), (16, 8, 100, 84), (3, 3, 24, 20), (4, 2, 64, 40), (2, 1, 200, 24)])
def test_a_token_does_not_depend_on_what_its_step_brings(heads, kv_heads, dk, dv, dtype):
    ops = _ops()
    g = torch.Generator(device=DEV)
    g.manual_seed(dk + dv)
    news, start = [13, 1, 34], 5
    T, B = sum(news), len(news)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    q, k = rnd(T, kv_heads, dk), rnd(T, kv_heads, dk)
    q, k = q / q.norm(dim=-1, keepdim=True), k / k.norm(dim=-1, keepdim=True)
    q, k, v, beta = q.reshape(T, -1).contiguous(), k.reshape(T, -1).contiguous(), rnd(T, heads * dv).to(dtype), torch.sigmoid(rnd(T, heads))
    decay = torch.exp(-torch.exp(rnd(T, heads * dk) - 3))
    first = rnd(B, heads * dk * dv)

    def steps(portions):
        """Outputs and states when the step after step brings, of every sequence, the tokens [from, to) that `portions` says."""
        out, rows, there = torch.empty(T, heads * dv, device=DEV), first.clone().view(torch.uint8), [start] * B
        for step in portions:
            ids = [b for b, (lo, hi) in step.items() if hi > lo]
            index = torch.cat([torch.arange(sum(news[:b]) + step[b][0], sum(news[:b]) + step[b][1], device=DEV) for b in ids])
            counts = [step[b][1] - step[b][0] for b in ids]
            for b, n in zip(ids, counts):
                there[b] += n
            part = torch.empty(len(index), heads * dv, device=DEV)
            i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
            ops.delta_scan(part, q[index], k[index], decay[index], beta[index], v[index], rows, 0, i32([0, *np.cumsum(counts)]), i32(ids),
                           i32([there[b] for b in ids]), len(ids), heads, kv_heads, dk, dv, max(counts))
            out[index] = part
        return out, rows.view(torch.float32)

    together = steps([{b: (0, news[b]) for b in range(B)}])
    ways = {"alone": [{b: (0, news[b])} for b in range(B)],
            "in portions": [{0: (0, 3), 2: (0, 10)}, {0: (3, 4), 1: (0, 1), 2: (10, 29)}, {0: (4, 13), 2: (29, 34)}],
            "one at a time": [{b: (i, i + 1) for b in range(B) if i < news[b]} for i in range(max(news))]}
    for way, portions in ways.items():
        out, left = steps(portions)
        assert torch.equal(out, together[0]) and torch.equal(left, together[1]), way
