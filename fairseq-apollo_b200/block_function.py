"""Training pass of the Mega block between its moving average and its output, as one autograd Function (native,
host/host.cpp): projections, gates, query / key affine, attention and the output gate (moving_average_gated_attention.py:317-414 of the
reference's fairseq/modules).

The products are library GEMMs, forward and backward; everything around them runs on this library's kernels.  The
gradients of the four slices of the mx_proj output are written side by side into one matrix, and the bias gradients
are column sums taken while those matrices are written, so autograd has no slices to zero, copy and add."""
import torch

from . import _lib
from .functions import plain

CAUSAL, _BIAS = 0, 1


def _own(module, name):
    """A plain one of the package's classes (by name: their module imports this one)."""
    return type(module).__name__ == name and plain(module, type(module))


def projections_plain(blk):
    return all(plain(m, torch.nn.Linear) for m in (blk.v_proj, blk.mx_proj, blk.h_proj))


def mode_of(blk, x, padding_mask, attn_mask, need_weights, before_attn_fn):
    """CAUSAL (chunked causal softmax with rotary positions), _BIAS (softmax with the learned relative bias, with or
    without a padding mask), or None when the block's own sequence of operations has to run."""
    if (attn_mask is not None or need_weights or before_attn_fn or not x.is_cuda
            or (blk.training and (blk.dropout_p or blk.hidden_dropout_p or blk.attention_dropout_p))
            or x.dtype not in (torch.float32, torch.bfloat16, torch.float16) or torch.is_autocast_enabled()):
        return None
    n = 16 // x.element_size()
    if blk.embed_dim % n or blk.zdim % n or blk.hdim % n or blk.zdim > 512:
        return None
    if not projections_plain(blk):
        return None
    if any(w.dtype != x.dtype for w in (blk.v_proj.weight, blk.mx_proj.weight, blk.h_proj.weight)):
        return None
    seq = x.size(1)
    period = blk.chunk_size if 1 < blk.chunk_size < seq else seq
    if seq % period:
        return None
    if blk.efficient_attn is not None:
        ok = _own(blk.rel_pos_bias, "RotaryEmbedding") and _own(blk.efficient_attn, "EfficientAttention") and period <= 8192
        return CAUSAL if ok else None
    if (blk.attention_activation == 'softmax' and blk.attn_softmax is None and period <= 8192
            and _own(blk.rel_pos_bias, "SimpleRelativePositionalBias") and period <= blk.rel_pos_bias.max_positions
            and x.size(0) * (seq // period) <= 65535):   # (chunks that the softmax takes in a launch)
        return _BIAS
    return None


def run(blk, mode, x, xn, mx, padding_mask):
    seq = x.size(1)
    period = blk.chunk_size if 1 < blk.chunk_size < seq else seq
    rot = bias = None
    if mode == CAUSAL:
        rot = torch.view_as_real(blk.rel_pos_bias._angles(0, period))
        padding_mask = None      # (as EfficientAttention: the causal kernel takes none)
    else:
        bias = blk.rel_pos_bias.rel_pos_bias
    return _lib.host().block_train(x, xn, mx, blk.v_proj.weight, blk.v_proj.bias, blk.mx_proj.weight, blk.mx_proj.bias,
                                   blk.h_proj.weight, blk.gamma, blk.beta, bias, rot, padding_mask, period)


def infer(blk, x, xn, mx, cache):
    """The same in inference, causal mode: the output, and with ``cache`` the keys (not rotated) and values."""
    seq = x.size(1)
    period = blk.chunk_size if 1 < blk.chunk_size < seq else seq
    rot = torch.view_as_real(blk.rel_pos_bias._angles(0, period))
    return _lib.host().block_infer(x, xn, mx, blk.v_proj.weight, blk.v_proj.bias, blk.mx_proj.weight, blk.mx_proj.bias,
                                   blk.h_proj.weight, blk.gamma, blk.beta, rot, period, cache)
