"""Fused TimestepNorm -> EMA, the drop-in for the three statements
``x = self.norm(x, ...); mx = self.move(x.transpose(1, 2), ...); mx = move_act(mx.transpose(1, 2))``
of MovingAverageGatedAttention.forward (fairseq/modules/moving_average_gated_attention.py:306-316).
"""
from typing import Dict, Optional

import torch
from torch import Tensor

from .. import _lib, ops
from ..functions import needs_grad, plain
from ..ops import _raw_stream
from .complex_exponential_moving_average import MultiHeadComplexEMA
from .exponential_moving_average import MultiHeadEMA
from .sequence_norm import SequenceNorm
from .timestep_norm import TimestepNorm


def timestep_norm_ema(norm: TimestepNorm, move: MultiHeadEMA, x: Tensor,
                      padding_mask: Optional[Tensor] = None,
                      incremental_state: Optional[Dict[str, Dict[str, Optional[Tensor]]]] = None,
                      activation: Optional[str] = None, return_normed: bool = False):
    """x (B, L, D) -> mx (B, L, D) [, normed x (B, L, D)].

    One pass over x when the norm keeps per-feature statistics and the EMA is causal;
    otherwise the two modules run back to back.  Both modules' incremental buffers are read
    and updated exactly as their own ``forward`` would.
    """
    if incremental_state is not None and padding_mask is None:   # a step like the one before it
        out = _lib.host().norm_ema_step(norm, move, x, incremental_state, activation, return_normed)
        if out is not None:
            return out
    assert activation in (None, 'silu')
    per_feature = norm.num_groups is None or norm.num_groups == norm.num_features
    # the decode fast path first: one token, an incremental state, inference
    if (incremental_state is not None and x.size(1) == 1 and padding_mask is None and per_feature
            and not move.bidirectional and not torch.is_grad_enabled() and x.is_contiguous()
            and (not move.complex or move.ndim in (2, 4, 8, 16, 32))):
        return _decode_step(norm, move, x, incremental_state, activation, return_normed)
    train = torch.is_grad_enabled() and needs_grad(x, *norm.parameters(), *move.parameters())
    if train or not per_feature or move.bidirectional:
        # training, grouped statistics or a bidirectional layer: the two modules in turn
        xn = norm(x, padding_mask, incremental_state)
        mx = ema_channels_last(move, xn, padding_mask, incremental_state, activation)
        return (mx, xn) if return_normed else mx
    if (incremental_state is not None and x.size(1) == 1 and padding_mask is None and x.is_contiguous()
            and (not move.complex or move.ndim in (2, 4, 8, 16, 32))):
        with torch.no_grad():
            return _decode_step(norm, move, x, incremental_state, activation, return_normed)
    p, q, g, omega = _ema_params(move)
    gamma_eff, beta, prev_count, prev_mean, prev_var, nstate = norm.operands(x.size(0), incremental_state)
    h_in = None
    estate = None
    if incremental_state is not None:
        estate = move._get_input_buffer(incremental_state)
        h_in = estate.get('prev_state')
    res = ops.tsn_ema_forward(x, prev_count, prev_mean, prev_var, gamma_eff, beta,
                              norm.eps, p, q, g, omega, padding_mask, h_in,
                              want_state=incremental_state is not None, silu=activation == 'silu',
                              want_normed=return_normed, complex_poles=move.complex)
    norm.store_statistics(incremental_state, nstate, res["count"], res["mean"], res["var"])
    if incremental_state is not None:
        estate['prev_state'] = res["h"]
        move._set_input_buffer(incremental_state, estate)
    return (res["y"], res["xn"]) if return_normed else res["y"]


def ema_channels_last(move, x, padding_mask, incremental_state, activation):
    """move(x) for x (B, L, D).  In training without transposes around it, which cost the backward a node each (a module
    with hooks or a forward of its own is called as one)."""
    if needs_grad(x, *move.parameters()) and plain(move, MultiHeadEMA, MultiHeadComplexEMA):
        return move._forward_train(x, padding_mask, incremental_state, activation, channels_last=True)
    return move(x.transpose(1, 2), padding_mask, incremental_state, activation).transpose(1, 2)


def sequence_norm_ema(norm: SequenceNorm, move: MultiHeadEMA, x: Tensor, padding_mask: Optional[Tensor] = None,
                      activation: Optional[str] = None):
    """x (B, D, L) -> EMA(SequenceNorm(x)) (B, D, L): the bidirectional branch of the Mega block
    (moving_average_gated_attention.py:298-303, 313).  One kernel, one pass over x, when the norm
    is per channel and the rows fit the row-resident kernel; otherwise the two modules in turn."""
    assert activation in (None, 'silu')
    train = torch.is_grad_enabled() and needs_grad(x, *norm.parameters(), *move.parameters())
    if not train and not move.complex and norm.num_groups is None and move.truncation is None:
        p, q, g = move.coeffs()
        gamma, beta = norm.operands()
        y = ops.sqn_ema_forward(x, gamma, beta, norm.eps, p, q, g, move.omega, padding_mask, move.bidirectional, move.shift,
                                silu=activation == 'silu')
        if y is not None:
            return y
    return move(norm(x, padding_mask), padding_mask, None, activation)


def _ema_params(move: MultiHeadEMA):
    """(p, q, gamma, omega) of the layer, fp32 and contiguous.  Outside of training they are kept until a parameter
    changes (identity, version counter, storage), the layer is moved or its mode is set; never across streams, nor in a
    graph that is being captured: it has its own, which stay as long as it does."""
    third = move.theta if move.complex else move.beta
    tensors = (move.alpha, move.delta, third, move.gamma, move.omega)
    key = None
    if not move.training and not torch.cuda.is_current_stream_capturing():
        key = [_raw_stream(move.alpha.get_device())] + [t._version for t in tensors] + [t.data_ptr() for t in tensors]
        cache = move.__dict__.get("_decode_cache")
        if cache is not None and cache[0] == key and all(a is b for a, b in zip(cache[2], tensors)):
            return cache[1]
    if move.complex:   # q, g complex64 (K, N): the kernel reads them as interleaved (re, im) floats
        p, q, g = ops.cema_coeffs(move.alpha, move.delta, move.theta, move.gamma)
        p, q, g = p.reshape(p.shape[0], -1).contiguous(), q.reshape(q.shape[0], -1).contiguous(), g.contiguous()
    else:
        p, q, g = ops.ema_coeffs(move.alpha, move.delta, move.beta, move.gamma)
    prm = (p, q, g, move.omega.detach().float().reshape(-1).contiguous())
    if key is not None:
        move._decode_cache = (key, prm, tensors)
    return prm


def _param_names(move):
    return ('weight', 'bias', 'alpha', 'delta', 'theta' if move.complex else 'beta', 'gamma', 'omega')


def _param_tensors(norm, move):
    """The seven parameter tensors the step depends on, fetched from the modules' parameter dicts
    (several times cheaper than attribute access through nn.Module.__getattr__)."""
    np_, mp_ = norm._parameters, move._parameters
    n = _param_names(move)
    return np_[n[0]], np_[n[1]], mp_[n[2]], mp_[n[3]], mp_[n[4]], mp_[n[5]], mp_[n[6]]


def _decode_step(norm, move, x, incremental_state, activation, return_normed):
    """Single-token step (x: (B, 1, D)): one fused kernel, one launch, running state updated in place."""
    _decode_step_plan(norm, move, x, incremental_state, activation, return_normed)
    out = _lib.host().norm_ema_step(norm, move, x, incremental_state, activation, return_normed)
    if out is None:
        raise RuntimeError("single-token step: a freshly built plan does not match its own inputs")
    return out


def _decode_step_plan(norm, move, x, incremental_state, activation, return_normed):
    """Builds (or rebuilds) the plan of the single-token step."""
    bsz, _, dim = x.shape
    nkey = norm._get_full_incremental_state_key("norm_state")
    ekey = move._get_full_incremental_state_key("ema_state")
    nstate = incremental_state.get(nkey)
    estate = incremental_state.get(ekey)
    if nstate is None or estate is None or 'prev_mean' not in nstate or estate.get('prev_state') is None:
        nstate, estate = _seed_decode_state(norm, move, bsz, dim, x.device, incremental_state)
    count, mean, var, h = nstate['prev_count'], nstate['prev_mean'], nstate['prev_var'], estate['prev_state']
    sdtype = torch.complex64 if move.complex else torch.float32
    if (mean.dtype != torch.float32 or not mean.is_contiguous() or var.dtype != torch.float32
            or not var.is_contiguous() or h.dtype != sdtype or not h.is_contiguous()
            or count.dtype != torch.int64 or not count.is_contiguous()):
        nstate['prev_mean'], nstate['prev_var'] = mean.float().contiguous(), var.float().contiguous()
        nstate['prev_count'] = count.long().contiguous()
        estate['prev_state'] = h.to(sdtype).contiguous()
        count, mean, var, h = nstate['prev_count'], nstate['prev_mean'], nstate['prev_var'], estate['prev_state']
    gamma, beta = ops.norm_prepare(norm.weight, norm.bias)
    p, q, g, omega = _ema_params(move)
    move._step_plan = _lib.host().StepPlan(
        _param_names(move), _param_tensors(norm, move), nkey, ekey, norm.num_groups, activation,
        [count, torch.empty_like(count), mean, var, h], [gamma, beta, p, q, g, omega], x, move.complex, return_normed, norm.eps)


def _seed_decode_state(norm, move, bsz, dim, device, incremental_state):
    """First single-token call of a generation: running statistics from the priors (fresh tensors,
    never views of the parameters: the step updates them in place) and zero pole states."""
    nstate = norm._get_input_buffer(incremental_state)
    if 'prev_mean' not in nstate:
        count, mean, var, nstate = norm.initial_statistics(bsz, incremental_state)
        nstate['prev_count'], nstate['prev_mean'], nstate['prev_var'] = count.clone(), mean.clone(), var.clone()
        norm._set_input_buffer(incremental_state, nstate)
    estate = move._get_input_buffer(incremental_state)
    if estate.get('prev_state') is None:
        sdtype = torch.complex64 if move.complex else torch.float32
        estate['prev_state'] = torch.zeros(bsz, dim, move.ndim, device=device, dtype=sdtype)
    move._set_input_buffer(incremental_state, estate)
    return nstate, estate
