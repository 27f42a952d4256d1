"""A prompt's step of a pre-norm block of the dense form, launched by one call: grouped-query attention with heads of 128 and a SwiGLU
feed-forward without biases, bfloat16, both norms folded into the products.  The kernels, their arguments and their order are those of
the parts (parts.attention, parts.swiglu); what is saved is the host's way through them, which is what a short prompt waits for."""
from __future__ import annotations

import torch

from ..kernels import ops
from . import linear
from .base import Prenormed

HEAD = 128


def _foldable(norm, width: int) -> bool:
    return norm is not None and getattr(norm, "foldable", False) and getattr(norm, "gain", None) is not None and norm.dim == width \
        and norm.gain.dtype in (torch.bfloat16, torch.float32)


def _weight(t: torch.Tensor, rows: int, cols: int) -> bool:
    return t.dtype == torch.bfloat16 and t.shape == (rows, cols) and t.is_contiguous() and t.data_ptr() % 16 == 0


def takes(block) -> bool:
    """Whether a block's parts are of this form."""
    from .attention import GQAAttention
    from .swiglu import SwiGLU
    mixer, ff = block.mixer, block.feed_forward
    return type(mixer) is GQAAttention and mixer.classic and mixer.head_dim == HEAD and mixer.qk_norm in (None, "head") and type(ff) is SwiGLU \
        and ff.activation == "silu"


def try_block(block, x, residual: torch.Tensor, ctx, slot) -> bool:
    """The block's step behind its first norm's output x; False: nothing ran, and the parts do it one by one."""
    mixer, ff = block.mixer, block.feed_forward
    T, width = residual.shape
    if ctx.decode or ctx.dtype != torch.bfloat16 or not linear.fold_norms or ops.profile_active() or not residual.is_contiguous():
        return False
    nh, nkv, inner = mixer.heads, mixer.kv_heads, ff.intermediate
    if ff.output_bias is not None or ff.gate_up.glu is not None or ff.gate_up.glu_bias is not None or mixer.hidden != width or ff.hidden != width \
            or T != ctx.num_tokens or not _foldable(block.norm2, width):
        return False
    turn = mixer.position.kernel_epilogue(ctx) if mixer.position is not None else None
    if mixer.position is not None and (turn is None or (turn.rope_dim and turn.pairing != "half") or turn.amplitude != 1.0):
        return False
    rope_dim = turn.rope_dim if turn is not None else 0
    tiles = ops.dense_block_tiles(T, width, nh, nkv, inner, rope_dim)
    w_qkv, w_o, w_in, w_down = mixer.qkv.weight, mixer.out.weight, ff.gate_up.weight, ff.down.weight
    k_plane, v_plane = ctx.cache.plane(slot.group, slot.plane)
    pre = x if isinstance(x, Prenormed) else None
    rows = pre.normed if pre else x
    if tiles == 0 or k_plane.dtype != torch.bfloat16 or k_plane.shape[2] != 64 or rows.dtype != torch.bfloat16 or rows.shape != (T, width) \
            or rows.stride(1) != 1 or rows.stride(0) % 8 or rows.data_ptr() % 16 or not _weight(w_qkv, (nh + 2 * nkv) * HEAD, width) \
            or not _weight(w_o, width, nh * HEAD) or not _weight(w_in, 2 * inner, width) or not _weight(w_down, width, inner):
        return False
    following = ctx.next_first_norm if _foldable(ctx.next_first_norm, width) else None
    key = ("dense block", nh, inner, width)
    space = ctx.shared.get(key)
    if space is None:       # what the blocks of a step hand from kernel to kernel; a block's is free again when the next one starts
        new = lambda n: torch.empty((T, n), dtype=torch.bfloat16, device=residual.device)
        space = ctx.shared[key] = (new(nh * HEAD), new(nh * HEAD), new(inner), new(width),
                                   torch.empty((T, tiles), dtype=torch.float32, device=residual.device))
    q, att, act, normed, ss = space
    angles = None
    if rope_dim and ops.gemm_tc_rope_kv_wants_angles(T, rope_dim):
        at = ("rotary angles", turn.inv_freq.data_ptr())
        angles = ctx.shared.get(at)
        if angles is None:
            angles = ctx.shared[at] = ops.rope_angles(ctx.token_pos[:T], turn.inv_freq)
    ops.dense_block(rows, pre, residual, w_qkv, w_o, w_in, w_down, mixer.q_gain, mixer.k_gain, block.norm2, following, q, att, act, normed, ss,
                    k_plane, v_plane, ctx.cache.tables[slot.group], ctx, turn.inv_freq if rope_dim else None, angles, rope_dim, nh, nkv, inner,
                    slot.writes, mixer.window, mixer.eps, mixer.scale)
    ctx.prenormed = Prenormed(normed, ss, width, following.eps, residual, following) if following is not None else None
    return True
