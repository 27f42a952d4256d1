"""The float32 product on tensor cores (three bfloat16 pieces an operand): against 64-bit sums, at the sizes where its tiles, chunks and
parts of K end, and bit for bit the same for a row whatever other rows there are.

The bound, times sum |a| |w|: the dropped pieces of a product 2^-24; in a chunk of 64 entries four additions of the sum's own size, each
cut off at 2^-22 of what it has reached at most; an addition of float32 a chunk and a part, rounded at 2^-24."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, _ops

pytestmark = pytest.mark.gpu


def _bound(a, w, K):
    return (1 + 16 + -(-K // 64) + 8) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T) + 1e-12


@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 97, 200])
@pytest.mark.parametrize("N, K", [(512, 512), (520, 516), (131, 64), (900, 1100), (2000, 132)])
@pytest.mark.parametrize("narrow", [False, True])
def test_products_in_every_form(M, N, K, narrow):
    ops = _ops()
    torch.manual_seed(M + N + K)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    a, w = torch.randn(M, K, device=DEV), torch.randn(2 * N, K, device=DEV) / math.sqrt(K)
    if narrow:                      # a bfloat16 checkpoint's weights: only their first pieces are multiplied
        w = w.bfloat16().float()
    shifted = torch.empty(M * K + 1, device=DEV)[1:].view(M, K).copy_(a)      # rows that do not start on 16 bytes: the form with planes
    for epilogue, rows in ((ops.EPILOGUE_STORE, N), (ops.EPILOGUE_ACCUMULATE, N), (ops.EPILOGUE_SWIGLU, 2 * N)):
        base, outs = torch.randn(M, N, device=DEV), []
        for x in (a, shifted):
            out = base.clone()
            ops.gemm_f32_tc(out, x, w[:rows], epilogue, status)
            outs.append(out)
        assert torch.equal(*outs)
        one = base[M - 1:].clone()
        ops.gemm_f32_tc(one, a[M - 1:].contiguous(), w[:rows], epilogue, status)
        assert torch.equal(one, outs[0][M - 1:])
        ref, bound = a.double() @ w[:rows].double().T, _bound(a, w[:rows], K)
        if epilogue == ops.EPILOGUE_SWIGLU:
            g, u = ref[:, :N], ref[:, N:]
            silu = g / (1 + torch.exp(-g))
            want = silu * u
            # |silu'| <= 1.1; the exponential and the division are within a few units of 2^-24
            bound = 1.1 * bound[:, :N] * (u.abs() + bound[:, N:]) + silu.abs() * bound[:, N:] + 2.0 ** -20 * want.abs()
        else:
            want = ref + base.double() if epilogue == ops.EPILOGUE_ACCUMULATE else ref
            bound = bound + 2.0 ** -23 * (want.abs() + ref.abs())
        assert ((outs[0].double() - want).abs() <= bound + 1e-12).all()
    assert status.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("N, K, epilogue", [(1024, 2048, 0), (2048, 6144, 1), (3072, 2048, 2), (640, 8192, 0)])
def test_a_row_does_not_depend_on_the_others_and_is_nearer_than_a_chain(N, K, epilogue):
    """Long sums over several parts of K, in tiles of every width; and further from the exact product than a chain of FMAs it must not be."""
    ops = _ops()
    torch.manual_seed(N)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    M = 531
    a, w = torch.randn(M, K, device=DEV), torch.randn(2 * N if epilogue == 2 else N, K, device=DEV) / math.sqrt(K)
    base = torch.randn(M, N, device=DEV)
    whole = base.clone()
    ops.gemm_f32_tc(whole, a, w, epilogue, status)
    for m in (1, 16, 32, 64, 129, 300):
        part = base[M - m:].clone()
        ops.gemm_f32_tc(part, a[M - m:], w, epilogue, status)
        assert torch.equal(part, whole[M - m:]), m
    if epilogue == 0:
        chain = torch.empty_like(base)
        ops.gemm_simt(chain, a, w, epilogue)
        ref = a.double() @ w.double().T
        assert (whole.double() - ref).norm() <= (chain.double() - ref).norm()
    assert status.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("M", [8, 150])
def test_entries_at_the_ends_of_the_range(M):
    """Infinities, NaN and entries whose first piece rounds to infinity give what the chain of FMAs gives, beside rows and columns of small ones
    (how exact those are is asked below)."""
    ops = _ops()
    torch.manual_seed(M)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    N, K = 512, 1024
    for epilogue in (ops.EPILOGUE_STORE, ops.EPILOGUE_SWIGLU):
        a, w = torch.randn(M, K, device=DEV), torch.randn(2 * N if epilogue == ops.EPILOGUE_SWIGLU else N, K, device=DEV) / math.sqrt(K)
        a[3, 5], a[5, 9], w[11, 17], a[M - 1, 0], w[len(w) - 1, 3] = math.inf, math.nan, -math.inf, 3.4e38, 1e30
        a[6] *= 1e-30
        w[100] *= 1e-20
        bound = _bound(a.nan_to_num(0, 0, 0), w.nan_to_num(0, 0, 0), K)[:, :N] + K * 2.0 ** -24 * (a.nan_to_num(0, 0, 0).double().abs() @ w.nan_to_num(0, 0, 0).double().abs().T)[:, :N]
        got, want = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
        ops.gemm_f32_tc(got, a, w, epilogue, status)
        ops.gemm_simt(want, a, w, epilogue)
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
        assert (got[got.isinf()] == want[want.isinf()]).all()
        ok = want.isfinite()
        if epilogue == ops.EPILOGUE_STORE:          # (the chain's own error is K * 2^-24 * sum |a| |w|)
            assert ((got.double() - want.double()).abs() <= bound + 1e-44)[ok].all()
    assert status.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("M, epilogue", [(8, 0), (64, 0), (150, 1), (531, 2)])
def test_rows_of_nan_cost_no_more_than_some_finite_ones(M, epilogue):
    """Rows of NaN are what a step gone wrong leaves; their outputs are computed again as chains of FMAs, which end at the first NaN.  (To their ends they
    took 50 to 450 times as long as finite rows.)  A lone infinity has its chain to the end, and no wait gives up meanwhile."""
    ops = _ops()
    torch.manual_seed(M)
    N, K = 1024, 14336
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    w = torch.randn(2 * N if epilogue == ops.EPILOGUE_SWIGLU else N, K, device=DEV) / math.sqrt(K)
    out, took = torch.zeros(M, N, device=DEV), []

    def best(a):
        times = []
        for _ in range(6):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            out.zero_()
            begin.record()
            ops.gemm_f32_tc(out, a, w, epilogue, status)
            end.record()
            torch.cuda.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times)

    finite = torch.randn(M, K, device=DEV)
    took.append(best(finite))
    took.append(best(torch.full_like(finite, math.nan)))
    assert out.isnan().all()
    one = finite.clone()
    one[M // 2] = math.nan
    took.append(best(one))
    assert out[M // 2].isnan().all() and out.isnan().sum() == N
    assert max(took[1:]) <= 5 * took[0], took
    one[M // 2] = finite[M // 2]
    one[M // 2, K // 2] = math.inf
    ops.gemm_f32_tc(out, one, w, epilogue, status)
    assert not out[torch.arange(M, device=DEV) != M // 2].isinf().any() and not out[M // 2].isfinite().all()
    assert status.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("M", [8, 40, 300])
def test_small_and_large_entries_lose_nothing_down_to_2_to_the_minus_110(M):
    """A power of two on either side comes out as that power of two, bit for bit, as long as no entry falls below 2^-110 (2^-70 here, and none of these
    normal entries is below 2^-40).  Below, the third piece is lost: an entry is off by half of bfloat16's smallest number, 2^-134, at most."""
    ops = _ops()
    torch.manual_seed(M)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    N, K = 640, 2048
    a, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV) / math.sqrt(K)
    a, w = (torch.where(t.abs() < 2.0 ** -40, 2.0 ** -40, t) for t in (a, w))
    product = lambda x, y: (out := torch.empty(M, N, device=DEV), ops.gemm_f32_tc(out, x, y, ops.EPILOGUE_STORE, status))[0]
    base = product(a, w)
    for e in (60, -60, -70):
        assert torch.equal(product(a * 2.0 ** e, w), base * 2.0 ** e) and torch.equal(product(a, w * 2.0 ** e), base * 2.0 ** e), e
    for e, f in ((-116, 0), (-116, 20), (-125, 30), (-130, 40)):       # (the last rows are no normal numbers themselves; the products are)
        x, y = a * 2.0 ** e, w * 2.0 ** f
        ref, sums = x.double() @ y.double().T, x.double().abs() @ y.double().abs().T
        bound = (1 + 16 + K // 64 + 8) * 2.0 ** -24 * sums + 2.0 ** -134 * y.double().abs().sum(1)
        assert ((product(x, y).double() - ref).abs() <= bound).all(), (e, f)
    assert status.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("M", [8, 32, 48, 300])
@pytest.mark.parametrize("entries", [1, 2, 8])
def test_rows_with_few_entries(M, entries):
    """Where a chain of FMAs rounds once a term, this is off by the dropped pieces (2^-24 of a term) and a cut-off at 2^-22 and a rounding a term; the
    small products' cut-offs are some 2^-24 together."""
    ops = _ops()
    torch.manual_seed(M + entries)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    N, K = 1024, 2048
    a, w, out = torch.zeros(M, K, device=DEV), torch.randn(N, K, device=DEV), torch.empty(M, N, device=DEV)
    for m in range(M):
        a[m, torch.randperm(K, device=DEV)[:entries]] = torch.randn(entries, device=DEV)
    ops.gemm_f32_tc(out, a, w, ops.EPILOGUE_STORE, status)
    ref, sums = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert ((out.double() - ref).abs() <= (2 + 5 * entries) * 2.0 ** -24 * sums).all()
    assert status.tolist() == [0, 0, 0, 0]
