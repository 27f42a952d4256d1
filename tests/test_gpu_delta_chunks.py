"""The gated delta rule four tokens at a time, against the recurrence in float64 token by token: sequences that end anywhere in a
group of eight, channels and columns that fill their blocks and ones that do not, a state that was there, decays down to zero."""
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
