"""A dense block's prompt step launched by one call is the step of its parts one by one, bit for bit: residual, cache, and the next norm's input."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, _ops

pytestmark = pytest.mark.gpu


def _weights(h, nh, nkv, f, gen):
    bf = torch.bfloat16
    m = lambda r, c: (torch.randn(r, c, generator=gen, device=DEV) / math.sqrt(c)).to(bf)
    g = lambda n: (1 + 0.1 * torch.randn(n, generator=gen, device=DEV)).to(bf)
    return {"q": m(nh * 128, h), "k": m(nkv * 128, h), "v": m(nkv * 128, h), "o": m(h, nh * 128), "qn": g(128), "kn": g(128), "g": m(f, h), "u": m(f, h),
            "d": m(h, f), "n1": g(h), "n2": g(h)}


def _compare(monkeypatch, news, past, h, nh, nkv, f, window, rope, qk_norm, taken):
    """A block's step twice over (the second takes what the first has prepared), by its parts and as `dense` allows it; `taken`: whether the one
    call is to launch it.  Launches of the two ways."""
    from hymt2sharp_b200.cache import PagedCache
    from hymt2sharp_b200.engine.engine import StepEntry, make_context
    from hymt2sharp_b200.parts import MixerSlot, PartSpec, build_part
    ops = _ops()
    gen = torch.Generator(device=DEV)
    gen.manual_seed(h + sum(news))
    block = build_part("block", PartSpec("pre_norm", dict(
        norm1=PartSpec("rmsnorm", dict(dim=h, eps=1e-5, weight="n1")), norm2=PartSpec("rmsnorm", dict(dim=h, eps=1e-5, weight="n2")),
        mixer=PartSpec("gqa_attention", dict(hidden=h, heads=nh, kv_heads=nkv, head_dim=128, eps=1e-5, qk_norm=qk_norm, q_proj="q", k_proj="k", v_proj="v",
                                             o_proj="o", q_norm="qn", k_norm="kn", window=window,
                                             position=PartSpec("neox_rope", dict(head_dim=128, rope_dim=rope, base=10000.0)) if rope else None)),
        feed_forward=PartSpec("swiglu", dict(hidden=h, intermediate=f, gate_proj="g", up_proj="u", down_proj="d")))))
    block.load(_weights(h, nh, nkv, f, gen), DEV, torch.bfloat16)
    assert block.dense
    need = block.cache_needs()[0]
    need = type(need)(need.kind, need.kv_heads, need.head_dim, planes=1, window=need.window)
    T = sum(news)
    start = torch.randn(T, h, generator=gen, device=DEV)
    filling = torch.randn(1, generator=gen, device=DEV)
    results, launches, calls = [], [], []
    launch = ops.dense_block
    monkeypatch.setattr(ops, "dense_block", lambda *args: (calls.append(1), launch(*args)))
    for whole in (False, True):
        cache = PagedCache([need], torch.bfloat16, DEV, 4096, max_slots=len(news), max_sequence_tokens=2048)
        slots = cache.alloc_slots(len(news))
        earlier = [(s, p) for s, p in zip(slots, past) if p]
        if earlier:
            cache.begin_step(earlier)
            cache.end_step(earlier)
        for store in cache.storage:
            store.fill_(float(filling))
        entries = [StepEntry(s, [1] * n, []) for s, n in zip(slots, news)]
        ctx, _, _, _ = make_context(cache, entries, 8, torch.bfloat16, torch.device(DEV), ops.device_status(torch.device(DEV)))
        ctx.next_first_norm = block.norm1
        block.dense = whole
        residual = start.clone()
        before = ops.launches
        for last in (False, True):                   # twice, so that the second one takes what the first has prepared
            if last:
                ctx.next_first_norm = None
            block.forward(residual, ctx, [MixerSlot(group=0, plane=0)])
            if not last:
                left = (ctx.prenormed.normed.clone(), ctx.prenormed.ss.clone()) if ctx.prenormed is not None else ()
        assert ctx.prenormed is None
        launches.append(ops.launches - before)
        assert len(calls) == (2 if whole and taken else 0)
        results.append((residual, *left, *[s.clone() for s in cache.storage]))
    assert len(results[0]) == len(results[1])
    for a, b in zip(*results):
        assert torch.equal(a, b)
    assert ops.device_status(torch.device(DEV))[0].item() == 0
    return launches


@pytest.mark.parametrize("news, past", [([61], [0]), ([129], [0]), ([300, 7, 64], [0, 33, 100]), ([1000], [70])])
@pytest.mark.parametrize("h, nh, nkv, f, window, rope, qk_norm", [(1024, 8, 2, 2816, 0, 128, True), (512, 4, 4, 1000, 50, 0, False), (512, 4, 1, 520, 0, 128, True)])
def test_one_call_is_the_parts_one_by_one(monkeypatch, news, past, h, nh, nkv, f, window, rope, qk_norm):
    parts, whole = _compare(monkeypatch, news, past, h, nh, nkv, f, window, rope, qk_norm, taken=True)
    assert parts == whole


@pytest.mark.parametrize("news, f, rope", [([61], 1002, 128), ([300], 1002, 128), ([300], 1000, 48)])
def test_what_the_one_call_does_not_take_goes_through_the_parts(monkeypatch, news, f, rope):
    """An inner width that is no multiple of 8; heads rotated in part beyond 128 tokens."""
    parts, whole = _compare(monkeypatch, news, [0], 512, 4, 2, f, 0, rope, True, taken=False)
    assert parts == whole
