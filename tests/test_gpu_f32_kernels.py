"""The kernels of the 32-bit path: the products of few rows and in every tile (bfloat16 operands too) at the sizes where their tiles end,
and the attention of its plain form in every instance that a rule picks.  Every sum keeps one order whichever kernel runs, so the
kernels are compared with each other bit for bit, and with 64-bit sums within the bound of a chain of K float32 FMAs,
K * 2^-24 * sum |a| |w| (twice that, for the add into the output)."""
import math

import numpy as np
import pytest
import torch

from test_gpu_kernels import DEV, _ops, _paged

pytestmark = pytest.mark.gpu


def _shifted(t):
    """The same matrix at an address that is no multiple of 16 bytes: what refuses whole pieces takes another kernel."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:]
    return flat.view(t.shape).copy_(t)


@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 33, 64, 65, 129, 200])
@pytest.mark.parametrize("N, K", [(16, 128), (17, 132), (130, 516), (300, 2052)])
def test_products_of_few_rows_and_in_tiles_agree_bit_for_bit(M, N, K):
    ops = _ops()
    torch.manual_seed(M + N + K)
    a, w = torch.randn(M, K, device=DEV), torch.randn(2 * N, K, device=DEV) / math.sqrt(K)
    bound = 2 * K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T) + 1e-12
    ref = a.double() @ w.double().T
    for epilogue, rows in ((ops.EPILOGUE_STORE, N), (ops.EPILOGUE_ACCUMULATE, N), (ops.EPILOGUE_SWIGLU, 2 * N)):
        base = torch.randn(M, N, device=DEV)
        outs = []
        for x in (a, _shifted(a)):
            out = base.clone()
            ops.gemm_simt(out, x, w[:rows], epilogue)
            outs.append(out)
        # one row alone, and the whole in one go
        one = base[M - 1:].clone()
        ops.gemm_simt(one, a[M - 1:].contiguous(), w[:rows], epilogue)
        assert torch.equal(outs[0], outs[1]) and torch.equal(one, outs[0][M - 1:])
        if epilogue == ops.EPILOGUE_STORE:
            assert ((outs[0].double() - ref[:, :N]).abs() <= bound[:, :N]).all()
        elif epilogue == ops.EPILOGUE_ACCUMULATE:
            assert ((outs[0].double() - base.double() - ref[:, :N]).abs() <= bound[:, :N] + 2.0 ** -23 * (base.double().abs() + ref[:, :N].abs())).all()


@pytest.mark.parametrize("M, N, epilogue", [(16, 20480, 0), (16, 20481, 0), (17, 9472, 1), (32, 9473, 1), (32, 9473, 2), (64, 4736, 0), (64, 4737, 0), (33, 2369, 2)])
def test_products_at_the_line_between_streamed_rows_and_tiles(M, N, epilogue):
    ops = _ops()
    torch.manual_seed(M + N)
    K = 260
    a, w = torch.randn(M, K, device=DEV), torch.randn(2 * N if epilogue == ops.EPILOGUE_SWIGLU else N, K, device=DEV) / math.sqrt(K)
    base = torch.randn(M, N, device=DEV)
    outs = [base.clone(), base.clone()]
    ops.gemm_simt(outs[0], a, w, epilogue)
    for m in range(0, M, 8):                                                     # streamed, whatever the width
        assert ops.gemm_simt_route(min(8, M - m), N, epilogue) == "rows"
        ops.gemm_simt(outs[1][m:m + 8], a[m:m + 8], w, epilogue)
    assert torch.equal(*outs)


# sizes whose last tile is ragged in both directions, with the tiles that the rule picks for them
_TILES = [(100, 5003, 0, False, "64x128"), (65, 4099, 2, False, "64x128"), (65, 4099, 0, False, "64x64"), (130, 1001, 2, False, "64x64"),
          (65, 131, 1, False, "32x64"), (67, 130, 2, False, "32x64"), (100, 5003, 1, True, "64x128"), (65, 4099, 2, True, "64x128"),
          (130, 8001, 1, True, "64x64"), (100, 5003, 2, True, "64x64"), (65, 5003, 0, True, "32x64"), (65, 3001, 2, True, "32x64"),
          (65, 131, 0, True, "64x64 short"), (129, 1001, 1, True, "64x64 short"), (129, 70, 2, True, "64x64 short")]


@pytest.mark.parametrize("M, N, epilogue, narrow, tile", _TILES)
@pytest.mark.parametrize("K", [131, 132, 16, 3])
def test_products_in_every_tile(M, N, epilogue, narrow, tile, K):
    ops = _ops()
    assert ops.gemm_simt_route(M, N, epilogue, narrow=narrow, aligned=False) == tile
    torch.manual_seed(M + N + K)
    bf = torch.bfloat16
    for ta, tw, to in ([(bf, bf, bf), (torch.float32, bf, torch.float32), (bf, torch.float32, torch.float32)] if narrow else [(torch.float32,) * 3]):
        a = torch.randn(M, K, device=DEV).to(ta)
        w = (torch.randn(2 * N if epilogue == ops.EPILOGUE_SWIGLU else N, K, device=DEV) / math.sqrt(K)).to(tw)
        base = torch.randn(M, N, device=DEV).to(to)
        outs = []
        wide = torch.zeros(M, K + 4, device=DEV, dtype=ta)                       # rows a piece of 16 bytes further apart
        wide[:, :K] = a
        for x in (a, _shifted(a), wide[:, :K]):
            out = base.clone()
            ops.gemm_simt(out, x, w, epilogue)
            outs.append(out)
        assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
        for m in (0, 63, M - 1):                                                 # one row alone
            one = base[m:m + 1].clone()
            ops.gemm_simt(one, a[m:m + 1].contiguous(), w, epilogue)
            assert torch.equal(one, outs[0][m:m + 1])
        ref, sums = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
        error = K * 2.0 ** -24 * sums                                            # a chain of K float32 FMAs
        store = 2.0 ** -8 if to == bf else 2.0 ** -23                            # and the rounding of what is stored
        if epilogue == ops.EPILOGUE_SWIGLU:
            g, u = ref[:, :N], ref[:, N:]
            silu = g / (1 + torch.exp(-g))
            want = silu * u
            # |silu'| <= 1.1; the exponential and the division are within a few units of 2^-24
            bound = 1.1 * error[:, :N] * (u.abs() + error[:, N:]) + silu.abs() * error[:, N:] + (store + 2.0 ** -20) * want.abs() + 1e-12
        else:
            want = ref + base.double() if epilogue == ops.EPILOGUE_ACCUMULATE else ref
            bound = error + store * (want.abs() + ref.abs()) + 1e-12
        assert ((outs[0].double() - want).abs() <= bound).all()


@pytest.mark.parametrize("nh, nkv, d, window", [(4, 4, 128, 0), (16, 2, 128, 0), (6, 2, 40, 0), (20, 1, 64, 50), (5, 1, 256, 100), (8, 2, 8, 0), (64, 1, 128, 0)])
@pytest.mark.parametrize("news", [[1, 1, 1, 1], [70, 1, 45, 300]])
def test_attention_of_the_plain_form_is_the_general_kernels_bit_for_bit(nh, nkv, d, window, news):
    ops = _ops()
    torch.manual_seed(nh * 100 + d)
    lens = [700, 1, 257, 320]
    keys = [torch.randn(L, nkv, d, device=DEV) for L in lens]
    vals = [torch.randn(L, nkv, d, device=DEV) for L in lens]
    kp, vp, table = _paged(keys, vals, 64, torch.float32)
    T = sum(news)
    q = torch.randn(T, nh * d, device=DEV)
    cu = torch.tensor(np.concatenate([[0], np.cumsum(news)]), dtype=torch.int32, device=DEV)
    slots, kv = torch.tensor([0, 1, -1, 3], dtype=torch.int32, device=DEV), torch.tensor(lens, dtype=torch.int32, device=DEV)
    for split in ((0, 256) if max(news) == 1 else (0,)):
        splits = -(-max(lens) // 256) if split else 0
        scratch = (None, None)
        if split:
            scratch = tuple(torch.full((n,), float("nan"), device=DEV) for n in ops.attention_simt_scratch(T, nh, d, splits))
        outs = []
        for x in (q, _shifted(q)):       # (the second takes the general kernel)
            out = torch.full((T, nh * d), 5.0, device=DEV)
            ops.attention_simt(out, x, kp, vp, table, cu, slots, kv, 4, max(news), nh, nkv, d, 1 / math.sqrt(d), window, split, splits, *scratch)
            outs.append(out)
        assert torch.equal(outs[0], outs[1])
        assert (outs[0][sum(news[:2]):sum(news[:3])] == 5.0).all()      # a padding row is left alone


@pytest.mark.parametrize("nh, nkv, d", [(4, 4, 128), (6, 2, 40), (16, 2, 64), (3, 1, 256)])
@pytest.mark.parametrize("window", [0, 20])
def test_a_row_does_not_know_values_of_tiles_it_cannot_see(nh, nkv, d, window):
    """Keys and values that are not finite reach no row but those that see their tile of 32 keys."""
    ops = _ops()
    torch.manual_seed(nh + d)
    T = 200
    keys, vals, q = torch.randn(T, nkv, d, device=DEV), torch.randn(T, nkv, d, device=DEV), torch.randn(T, nh * d, device=DEV)
    bad_k, bad_v = keys.clone(), vals.clone()
    for at, value in ((40, math.nan), (150, math.inf), (199, -math.inf)):
        bad_v[at], bad_k[at] = value, value
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
    outs = []
    for k, v in ((keys, vals), (bad_k, bad_v)):
        kp, vp, table = _paged([k], [v], 64, torch.float32)
        out = torch.empty(T, nh * d, device=DEV)
        ops.attention_simt(out, q, kp, vp, table, i32(0, T), i32(0), i32(T), 1, T, nh, nkv, d, 1 / math.sqrt(d), window)
        outs.append(out)
    tile = lambda p: p // 32
    for p in range(T):
        low = max(0, p - window + 1) if window else 0
        if not any(tile(low) <= tile(at) <= tile(p) for at in (40, 150, 199)):
            assert torch.equal(outs[0][p], outs[1][p]), p
        if any(low <= at <= p for at in (40, 150, 199)):
            assert not outs[1][p].isfinite().any(), p


@pytest.mark.parametrize("nh, nkv, d, rows", [(16, 4, 128, 64), (12, 4, 104, 64), (16, 16, 96, 64), (16, 16, 72, 32), (40, 1, 128, 64), (16, 4, 64, 32), (16, 4, 24, 32), (16, 8, 136, 32)])
@pytest.mark.parametrize("window", [0, 70])
def test_long_prompts_are_the_general_kernels_bit_for_bit(nh, nkv, d, rows, window):
    """The blocks of 64 rows, several tokens each, with windows and parts of prompts; heads and tokens that do not fill a block."""
    ops = _ops()
    torch.manual_seed(nh * 100 + d)
    news, lens = [1001, 3, 613], [1001, 90, 900]
    T = sum(news)
    assert ops.attention_prompt_rows(T, nh, d) == rows
    kp, vp, table = _paged([torch.randn(L, nkv, d, device=DEV) for L in lens], [torch.randn(L, nkv, d, device=DEV) for L in lens], 64, torch.float32)
    q = torch.randn(T, nh * d, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    outs = []
    for x in (q, _shifted(q)):       # (the second takes the general kernel)
        out = torch.full((T, nh * d), 5.0, device=DEV)
        ops.attention_simt(out, x, kp, vp, table, i32([0, 1001, 1004, 1617]), i32([0, 1, 2]), i32(lens), 3, 1001, nh, nkv, d, 1 / math.sqrt(d), window)
        outs.append(out)
    assert torch.equal(*outs)
