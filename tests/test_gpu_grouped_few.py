"""The grouped product of a few sorted rows on tensor cores: against 64-bit sums and the CUDA-core kernel's accuracy, rows and tiles that are not
in use left alone, and a row's result the same bit for bit whatever other rows there are.  The bound, times sum |a| |w|: 16 products of an MMA cut
off at 2^-22, then float32 additions, (K / 64 + 6) of them rounded at 2^-24."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, _ops

pytestmark = pytest.mark.gpu


def _sorted(ops, chosen, experts):
    T, top = chosen.shape
    tiles = ops.moe_tiles(T, top, experts, 8)
    i32 = lambda *s: torch.empty(s, dtype=torch.int32, device=DEV)
    pair_row, row_token, tile_group, counts = i32(T, top), i32(tiles * 8), i32(tiles + 1), i32(experts)
    ops.moe_place(pair_row, row_token, tile_group, counts, chosen, experts, 8)
    return pair_row, row_token, tile_group


@pytest.mark.parametrize("T, experts, top", [(1, 4, 2), (3, 16, 4), (12, 3, 2), (16, 32, 4)])
@pytest.mark.parametrize("N, K", [(512, 256), (520, 512), (200, 1024), (128, 4096)])
def test_grouped_products_of_few_rows(T, experts, top, N, K):
    ops = _ops()
    torch.manual_seed(T + N + K)
    bf = torch.bfloat16
    x = torch.randn(T, K, device=DEV).to(bf)
    w = (torch.randn(experts, 2 * N, K, device=DEV) / math.sqrt(K)).to(bf)
    chosen = torch.stack([torch.randperm(experts, device=DEV)[:top] for _ in range(T)]).int()
    pair_row, row_token, tile_group = _sorted(ops, chosen, experts)
    rows = row_token.numel()
    for epilogue in (ops.EPILOGUE_STORE, ops.EPILOGUE_RELU_SQUARED, ops.EPILOGUE_SWIGLU):
        weight = w if epilogue == ops.EPILOGUE_SWIGLU else w[:, :N].contiguous()
        for dtype in (torch.float32, bf):
            out = torch.full((rows, N), 7.0, dtype=dtype, device=DEV)
            ops.gemm_grouped_few(out, x, weight, tile_group, row_token, True, epilogue)
            assert (out[row_token < 0] == 7.0).all()
            for t in range(T):
                for c in range(top):
                    m = weight[int(chosen[t, c])].double()
                    s = m @ x[t].double()
                    error = (16 + K // 64 + 6) * 2.0 ** -24 * (m.abs() @ x[t].double().abs())
                    if epilogue == ops.EPILOGUE_STORE:
                        want = s
                    elif epilogue == ops.EPILOGUE_RELU_SQUARED:
                        want, error = s.clamp(min=0) ** 2, error * (2 * s.abs() + error)
                    else:
                        g, u = s[:N], s[N:]
                        silu = g / (1 + torch.exp(-g))
                        want, error = silu * u, 1.1 * error[:N] * (u.abs() + error[N:]) + silu.abs() * error[N:] + 2.0 ** -20 * (silu * u).abs()
                    store = 2.0 ** -8 if dtype == bf else 2.0 ** -23
                    got = out[int(pair_row[t, c])].double()
                    assert ((got - want).abs() <= error + store * want.abs() + 1e-12).all()
    # one token alone: the same bits
    full = torch.empty(rows, N, device=DEV)
    ops.gemm_grouped_few(full, x, w[:, :N].contiguous(), tile_group, row_token, True)
    p1, r1, g1 = _sorted(ops, chosen[T - 1:].contiguous(), experts)
    alone = torch.empty(r1.numel(), N, device=DEV)
    ops.gemm_grouped_few(alone, x[T - 1:].contiguous(), w[:, :N].contiguous(), g1, r1, True)
    for c in range(top):
        assert torch.equal(alone[int(p1[0, c])], full[int(pair_row[T - 1, c])])
    # sorted rows instead of gathered ones
    lined = torch.zeros(rows, K, dtype=bf, device=DEV)
    used = row_token >= 0
    lined[used] = x[row_token[used].long()]
    again = torch.empty(rows, N, device=DEV)
    ops.gemm_grouped_few(again, lined, w[:, :N].contiguous(), tile_group, row_token, False)
    assert torch.equal(again[used], full[used])
    assert ops.device_status(torch.device(DEV))[0].item() == 0


def test_what_the_kernel_of_few_rows_does_not_take_goes_to_the_cuda_cores():
    ops = _ops()
    bf = torch.bfloat16
    a, w = torch.randn(8, 512, device=DEV).to(bf), torch.randn(32, 1024, 512, device=DEV).to(bf)
    assert ops.gemm_grouped_few_supported(a, w, 64)
    assert not ops.gemm_grouped_few_supported(a.float(), w.float(), 64)
    assert not ops.gemm_grouped_few_supported(a[:, :500], w[:, :, :500].contiguous(), 64)
    assert not ops.gemm_grouped_few_supported(a, w, 8)                       # too little to read


@pytest.mark.parametrize("hidden, ff, experts, top", [(2048, 1024, 8, 2), (1024, 512, 16, 2), (512, 256, 8, 2)])
def test_a_token_of_a_mixture_does_not_depend_on_the_size_of_its_step(hidden, ff, experts, top):
    """Steps of up to 64 (token, choice) pairs: the rule that picks their kernel hangs on the weights alone."""
    from hymt2sharp_b200.parts import PartSpec, build_part
    ops = _ops()
    torch.manual_seed(hidden)
    bf = torch.bfloat16
    part = build_part("feed_forward", PartSpec("routed_experts", dict(hidden=hidden, experts=experts, identity=0, top=top, intermediate=ff, activation="silu",
                                                                      router="r", gate_proj="{}.g", up_proj="{}.u", down_proj="{}.d")))
    m = lambda r, c: (torch.randn(r, c, device=DEV) / math.sqrt(c)).to(bf)
    weights = {"r": m(experts, hidden)}
    for e in range(experts):
        weights.update({f"{e}.g": m(ff, hidden), f"{e}.u": m(ff, hidden), f"{e}.d": m(hidden, ff)})
    part.load(weights, DEV, bf)
    x = torch.randn(32, hidden, device=DEV).to(bf)

    def rows(n):
        y, pair_row, _, _ = part._experts(x[:n].contiguous(), None)
        return y[pair_row.long()]

    whole = rows(32)
    for n in (1, 2, 5, 6, 11, 31):
        assert torch.equal(rows(n), whole[:n]), n
    assert ops.device_status(torch.device(DEV))[0].item() == 0
