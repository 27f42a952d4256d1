"""What enters the delta rule: four channels an access and one at a time give the same bits."""
import pytest
import torch

from test_gpu_kernels import DEV, _ops

pytestmark = pytest.mark.gpu


# fewer quads than threads, as many, one pass and a rest of the two in flight; several blocks a token (64 tokens) and one (600)
@pytest.mark.parametrize("T, H, G, d", [(1, 1, 1, 4), (3, 2, 1, 36), (5, 4, 2, 128), (64, 9, 3, 100), (600, 16, 8, 128), (513, 3, 3, 12)])
def test_decays_by_fours_and_one_at_a_time(T, H, G, d):
    ops = _ops()
    torch.manual_seed(T + d)
    qk = torch.randn(T, 2 * G * d, device=DEV).bfloat16()
    x, bias, a_log, b = 3 * torch.randn(T, H * d, device=DEV), torch.randn(H * d, device=DEV), torch.randn(H, device=DEV), torch.randn(T, H, device=DEV)
    outs = []
    for off in (0, 1):                # rows on 16 bytes, and not
        decay = torch.empty(T * H * d + off, device=DEV)[off:].view(T, H * d).copy_(x)
        qn, kn, beta = torch.empty(T, G * d, device=DEV), torch.empty(T, G * d, device=DEV), b.clone()
        ops.delta_prep(qk, qn, kn, decay, beta, bias, a_log, H, G, d, 0.25, 1e-6)
        outs.append((qn, kn, decay, beta))
    assert all(torch.equal(p, q) for p, q in zip(*outs))
    step = torch.nn.functional.softplus(x.double() + bias.double())
    want = torch.exp(-(a_log.double().exp().repeat_interleave(d) * step))
    # the exponent, up to 100 here, carries a few roundings of 2^-24
    assert ((outs[0][2].double() - want).abs() <= 2.0 ** -24 * want * (8 + 8 * (a_log.double().exp().repeat_interleave(d) * step)) + 1e-37).all()
