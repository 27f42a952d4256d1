"""The kernels of the 32-bit path at the sizes where their tiles end: the products for few rows and in tiles.  Every sum keeps one
order whichever kernel runs, so the kernels are compared with each other bit for bit, and with 64-bit sums within the bound of a
chain of K float32 FMAs, K * 2^-24 * sum |a| |w| (twice that, for the add into the output)."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, _ops

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
