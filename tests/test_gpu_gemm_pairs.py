"""Products that pairs of CTAs run (tiles of 256 tokens): the same bits as the kernel of single CTAs gives for the rows a few at a time, at sizes
whose last tiles are ragged in both directions, with every epilogue."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, _ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T, N, K, epilogue", [(8192, 3072, 2048, 0), (8000, 2504, 3080, 0), (10001, 4096, 4096, 1), (8200, 4104, 3072, 2), (16001, 1000, 4104, 0),
                                               (1025, 4104, 3080, 0), (1700, 2048, 4104, 1), (1000, 8192, 1024, 2)])
def test_pairs_give_the_bits_of_single_ctas(T, N, K, epilogue):
    ops = _ops()
    assert ops.gemm_tc_pairs(T, N, K, epilogue)["pairs"] > 0
    torch.manual_seed(T)
    bf, status = torch.bfloat16, torch.zeros(4, dtype=torch.int32, device=DEV)
    x = torch.randn(T, K, device=DEV).to(bf)
    w = (torch.randn(2 * N if epilogue == ops.EPILOGUE_SWIGLU else N, K, device=DEV) / math.sqrt(K)).to(bf)
    base = torch.randn(T, N, device=DEV) if epilogue == ops.EPILOGUE_ACCUMULATE else torch.zeros(T, N, device=DEV, dtype=bf)
    tiles = -(-N // 16)
    sums = lambda t: (torch.empty(t, N, dtype=bf, device=DEV), torch.ones(N, device=DEV), torch.empty(t, tiles, device=DEV)) if epilogue == ops.EPILOGUE_ACCUMULATE else None
    scale = torch.rand(T, 7, device=DEV) * K if epilogue != ops.EPILOGUE_ACCUMULATE else None
    out, after = base.clone(), sums(T)
    ops.gemm_tc(out, x, w, epilogue, status, row_scale=None if scale is None else (scale, K, 1e-5), norm_after=after)
    step = 400
    for at in list(range(0, T, step))[:3] + [T - 300]:        # (parts of more than 128 rows: fewer run on another kernel, whose sums are split)
        part = base[at:at + step].clone()
        n = part.shape[0]
        assert ops.gemm_tc_pairs(n, N, K, epilogue)["pairs"] == 0
        left = sums(n)
        ops.gemm_tc(part, x[at:at + n].contiguous(), w, epilogue, status, row_scale=None if scale is None else (scale[at:at + n].contiguous(), K, 1e-5), norm_after=left)
        assert torch.equal(part, out[at:at + n])
        if left is not None:
            assert torch.equal(left[0], after[0][at:at + n]) and torch.equal(left[2], after[2][at:at + n])
    ref = x[T - 300:].double() @ w.double().T
    if epilogue == ops.EPILOGUE_STORE:
        ref = ref / torch.sqrt(scale[T - 300:].double().sum(1, keepdim=True) / K + 1e-5)
        assert (out[T - 300:].double() - ref).norm() <= 4e-3 * ref.norm()
    assert status.tolist() == [0, 0, 0, 0]
