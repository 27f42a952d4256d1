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


@pytest.mark.parametrize("T, N, K, dtype, rule", [(3000, 2504, 3080, torch.float32, None), (3000, 2504, 3080, torch.bfloat16, "clamped"), (2100, 4000, 2048, torch.bfloat16, "biases")])
def test_pairs_give_the_bits_of_single_ctas_in_the_other_epilogues(T, N, K, dtype, rule):
    """The float32 store, and the gates of other rules: the clamped one, and biases in front of silu(gate) * up."""
    ops = _ops()
    epilogue = ops.EPILOGUE_SWIGLU if rule else ops.EPILOGUE_STORE
    assert ops.gemm_tc_pairs(T, N, K, epilogue)["pairs"] > 0
    torch.manual_seed(N)
    bf, status = torch.bfloat16, torch.zeros(4, dtype=torch.int32, device=DEV)
    x = torch.randn(T, K, device=DEV).to(bf)
    w = (torch.randn(2 * N if rule else N, K, device=DEV) / math.sqrt(K)).to(bf)
    glu = ops.GluRule("clamped", 0.8, 1.702) if rule == "clamped" else None
    bias = torch.randn(2 * N, device=DEV) if rule else None
    out = torch.empty(T, N, dtype=dtype, device=DEV)
    ops.gemm_tc(out, x, w, epilogue, status, glu=glu, glu_bias=bias)
    for at in (0, 800, T - 300):
        part = torch.empty_like(out[at:at + 300])
        assert ops.gemm_tc_pairs(300, N, K, epilogue)["pairs"] == 0
        ops.gemm_tc(part, x[at:at + 300].contiguous(), w, epilogue, status, glu=glu, glu_bias=bias)
        assert torch.equal(part, out[at:at + 300])
    ref = x[T - 300:].double() @ w.double().T
    if rule:
        g, u = ref[:, :N] + bias[:N].double(), ref[:, N:] + bias[N:].double()
        if rule == "clamped":
            g, u = g.clamp(max=0.8), u.clamp(-0.8, 0.8)
            ref = g * torch.sigmoid(1.702 * g) * (u + 1)
        else:
            ref = g * torch.sigmoid(g) * u
    # (a bfloat16 result is rounded at 2^-9, a sum of K products in float32 is off by some 2^-24 * sqrt(K) of it)
    assert (out[T - 300:].double() - ref).norm() <= (1e-5 if dtype == torch.float32 else 4e-3) * ref.norm()
    assert status.tolist() == [0, 0, 0, 0]


@pytest.mark.parametrize("T, nh, nkv, K, rope_dim, norm, scaled, width", [
    (2001, 16, 4, 2048, 128, True, True, 128), (3001, 16, 4, 2048, 128, False, False, 256), (2300, 15, 3, 2048, 0, True, True, 128),
    (2300, 9, 1, 4104, 128, True, False, 256), (1301, 16, 8, 2048, 128, True, True, 128)])
def test_paired_projection_rotates_and_appends_like_single_ctas(T, nh, nkv, K, rope_dim, norm, scaled, width):
    """The q/k/v projection of a prompt with rotation, norm and cache append: q and both planes have the bits that single CTAs give for some hundred
    of its tokens.  Tiles of one head and of two (an odd number of heads: the last holds one), ragged last tiles of 256 tokens, a padding row."""
    ops = _ops()
    d, bt, bf = 128, 64, torch.bfloat16
    plan = ops.gemm_tc_pairs(T, (nh + 2 * nkv) * d, K, 3)
    assert plan["pairs"] > 0 and plan["tile_width"] == width
    torch.manual_seed(T + nh)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    # a long prompt that starts inside a block, a padding row, a second prompt
    first, padding = T // 2, 37
    pos = torch.cat([torch.arange(first) + 100, torch.arange(padding), torch.arange(T - first - padding)]).int().to(DEV)
    seq = torch.cat([torch.zeros(first), torch.ones(padding), torch.full((T - first - padding,), 2.0)]).int().to(DEV)
    slots = torch.tensor([1, -1, 0], dtype=torch.int32, device=DEV)
    per_slot = -(-(T + 100) // bt)
    table = torch.randperm(2 * per_slot, device=DEV).int().view(2, per_slot)
    x = torch.randn(T, K, device=DEV).to(bf)
    w = (torch.randn((nh + 2 * nkv) * d, K, device=DEV) / math.sqrt(K)).to(bf)
    inv = (1.0 / (10000.0 ** (torch.arange(rope_dim // 2, dtype=torch.float32) / max(1, rope_dim // 2)))).to(DEV) if rope_dim else None
    gains = [(1 + 0.1 * torch.randn(d, device=DEV)).to(bf) if norm else None for _ in range(2)]
    scale = torch.rand(T, 7, device=DEV) * K if scaled else None

    def project(rows):
        n = len(pos[rows])
        planes = [torch.zeros(2 * per_slot, nkv, bt, d, dtype=bf, device=DEV) for _ in range(2)]
        q = torch.full((n, nh * d), 9.0, dtype=bf, device=DEV)
        at = pos[rows].contiguous()
        angles = ops.rope_angles(at, inv) if ops.gemm_tc_rope_kv_wants_angles(n, rope_dim) else None
        ops.gemm_tc_rope_kv(x[rows].contiguous(), w, q, *planes, table, bt, seq[rows].contiguous(), at, slots, inv, rope_dim, *gains, 1e-5, nh, nkv,
                            status, angles=angles, row_scale=(scale[rows].contiguous(), K, 1e-5) if scaled else None)
        return q, planes

    q, planes = project(slice(0, T))
    slot = slots[seq.long()].long()
    real = slot >= 0
    block, offset = table[slot.clamp(min=0), pos.long() // bt].long(), pos.long() % bt
    for plane in planes:        # what no token names is left alone
        untouched = torch.ones(2 * per_slot, bt, dtype=torch.bool, device=DEV)
        untouched[block[real], offset[real]] = False
        assert (plane.permute(0, 2, 1, 3)[untouched] == 0).all()
    for at in (0, 256, first - 150, T - 300):
        rows = slice(at, at + 300)
        assert ops.gemm_tc_pairs(300, (nh + 2 * nkv) * d, K, 3)["pairs"] == 0
        part_q, part_planes = project(rows)
        assert torch.equal(part_q, q[rows])
        mine = real[rows]
        b, o = block[rows][mine], offset[rows][mine]
        for whole, part in zip(planes, part_planes):
            assert torch.equal(whole[b, :, o], part[b, :, o]) and (part[b, :, o] != 0).any()
    assert status.tolist() == [0, 0, 0, 0]
