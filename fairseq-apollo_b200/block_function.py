"""Training pass of the Mega block between its moving average and its output, as one autograd Function: projections,
gates, query / key affine, attention and the output gate (moving_average_gated_attention.py:317-414 of the
reference's fairseq/modules).

The products are library GEMMs, forward and backward; everything around them runs on this library's kernels.  The
gradients of the four slices of the mx_proj output are written side by side into one matrix, and the bias gradients
are column sums taken while those matrices are written, so autograd has no slices to zero, copy and add."""
import torch

from . import _lib, ops

_CAUSAL, _BIAS = 0, 1


def mode_of(blk, x, padding_mask, attn_mask, need_weights, before_attn_fn):
    """_CAUSAL (chunked causal softmax with rotary positions), _BIAS (softmax with the learned relative bias, with or
    without a padding mask), or None when the block's own sequence of operations has to run."""
    from .modules.moving_average_gated_attention import RotaryEmbedding, SimpleRelativePositionalBias
    if (attn_mask is not None or need_weights or before_attn_fn or not x.is_cuda
            or (blk.training and (blk.dropout_p or blk.hidden_dropout_p or blk.attention_dropout_p))
            or x.dtype not in (torch.float32, torch.bfloat16, torch.float16) or torch.is_autocast_enabled()):
        return None
    n = 16 // x.element_size()
    if blk.embed_dim % n or blk.zdim % n or blk.hdim % n or blk.zdim > 512:
        return None
    if any(w.dtype != x.dtype for w in (blk.v_proj.weight, blk.mx_proj.weight, blk.h_proj.weight)):
        return None
    seq = x.size(1)
    period = blk.chunk_size if 1 < blk.chunk_size < seq else seq
    if seq % period:
        return None
    if blk.efficient_attn is not None:
        ok = isinstance(blk.rel_pos_bias, RotaryEmbedding) and period <= 8192
        return _CAUSAL if ok else None
    if (blk.attention_activation == 'softmax' and blk.attn_softmax is None and period <= 8192
            and isinstance(blk.rel_pos_bias, SimpleRelativePositionalBias) and period <= blk.rel_pos_bias.max_positions):
        return _BIAS
    return None


def run(blk, mode, x, xn, mx, padding_mask):
    seq = x.size(1)
    period = blk.chunk_size if 1 < blk.chunk_size < seq else seq
    rot = bias = None
    if mode == _CAUSAL:
        rot = torch.view_as_real(blk.rel_pos_bias._angles(0, period))
        padding_mask = None      # (as EfficientAttention: the causal kernel takes none)
    else:
        bias = blk.rel_pos_bias.rel_pos_bias
    return BlockFunction.apply(x, xn, mx, blk.v_proj.weight, blk.v_proj.bias, blk.mx_proj.weight, blk.mx_proj.bias,
                               blk.h_proj.weight, blk.gamma, blk.beta, bias, rot, padding_mask, period)


def _slices(base, d, s, e):
    return base[:, :d], base[:, d:d + s], base[:, d + s:d + s + e], base[:, d + s + e:]


class BlockFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, xn, mx, wv, bv, wm, bm, wh, gamma, beta, bias, rot, padding_mask, period):
        bsz, seq, d = x.shape
        rows, s, e = bsz * seq, gamma.shape[1], wv.shape[0]
        x, xn, mx = x.contiguous(), xn.contiguous().view(rows, d), mx.contiguous().view(rows, d)
        v_lin = torch.addmm(bv, xn, wv.t())
        base = torch.addmm(bm, mx, wm.t())
        u, z, r, hx = _slices(base, d, s, e)
        v = ops.gate_silu(v_lin)
        if rot is not None:
            q, k = ops.gate_qk_rotary(z, gamma, beta, rot, period)
        else:
            q, k = ops.gate_qk(z, gamma, beta, eps=1e-5)
        nb = rows // period
        q, k, v3 = q.view(nb, period, s), k.view(nb, period, s), v.view(nb, period, e)
        scores = torch.bmm(q, k.transpose(1, 2))
        if rot is not None:
            w = ops.attention_softmax_fwd(scores, True)
        else:
            mask = None if padding_mask is None else ops._mask_u8(padding_mask, bsz, seq).view(nb, period)
            w = ops.attention_bias_softmax_fwd(scores, bias.detach(), mask)
        del scores
        attn = torch.bmm(w, v3).view(rows, e)
        gated = ops.gate_mul_silu(attn, r)
        h_lin = torch.mm(gated, wh.t())
        out = ops.gate_output(x.view(rows, d), u, hx, h_lin)
        ctx.save_for_backward(x, xn, mx, wv, wm, wh, gamma, bias, rot, v_lin, base, q, k, v3, w, attn, gated, h_lin)
        ctx.period = period
        ctx.dtypes = (bv.dtype, bm.dtype, gamma.dtype, beta.dtype)
        return out.view(bsz, seq, d)

    @staticmethod
    def backward(ctx, dout):
        x, xn, mx, wv, wm, wh, gamma, bias, rot, v_lin, base, q, k, v3, w, attn, gated, h_lin = ctx.saved_tensors
        bsz, seq, d = x.shape
        rows, s, e = bsz * seq, gamma.shape[1], wv.shape[0]
        f = base.shape[1]
        need = ctx.needs_input_grad
        u, z, r, hx = _slices(base, d, s, e)
        dout = dout.to(x.dtype).contiguous().view(rows, d)
        # one zeroed array for every sum: bias gradients, (2, s) affine, relative bias
        nbias = 0 if bias is None else bias.shape[0]
        sums = torch.zeros(e + f + 4 * s + nbias, device=x.device, dtype=torch.float32)
        dbv, dbm, dgamma, dbeta, dbias = torch.split(sums, (e, f, 2 * s, 2 * s, nbias))
        dbase = torch.empty_like(base)
        du, dz, dr, dhx = _slices(dbase, d, s, e)
        dx = torch.empty_like(dout)
        ops.gate_output_bwd(dout, x.view(rows, d), u, hx, h_lin, dx, du, dhx, dbm[:d], dbm[d + s + e:])
        dgated = torch.mm(dhx, wh)
        dwh = torch.mm(dhx.t(), gated) if need[7] else None
        ops.gate_mul_silu_bwd(dgated, attn, r, dgated, dr, dbm[d + s:d + s + e])
        dattn = dgated.view(v3.shape)
        dv = torch.bmm(w.transpose(1, 2), dattn).view(rows, e)
        dw = torch.bmm(dattn, v3.transpose(1, 2))
        ds = ops.attention_softmax_bwd(dw, w, rot is not None)
        if bias is not None:
            ops.attention_bias_grad(ds, dbias)
        dq = torch.bmm(ds, k).view(rows, s)
        dk = torch.bmm(ds.transpose(1, 2), q).view(rows, s)
        ops.gate_qk_bwd(z, gamma, rot, ctx.period, dq, dk, dz, dgamma, dbeta, dbm[d:d + s])
        ops.gate_silu_bwd(dv, v_lin, dv, dbv)
        dxn = torch.mm(dv, wv).view(bsz, seq, d) if need[1] else None
        dwv = torch.mm(dv.t(), xn) if need[3] else None
        dmx = torch.mm(dbase, wm).view(bsz, seq, d) if need[2] else None
        dwm = torch.mm(dbase.t(), mx) if need[5] else None
        dbv, dbm, dgamma, dbeta, dbias = torch.split(sums.to(wv.dtype), (e, f, 2 * s, 2 * s, nbias))
        t = ctx.dtypes
        return (dx.view(bsz, seq, d), dxn, dmx, dwv, dbv.to(t[0]), dwm, dbm.to(t[1]), dwh, dgamma.view(2, s).to(t[2]),
                dbeta.view(2, s).to(t[3]), None if bias is None else dbias.to(bias.dtype), None, None, None)
