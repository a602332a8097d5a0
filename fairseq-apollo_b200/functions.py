"""The training path's differentiable operators.  The autograd Functions are native (host/host.cpp): forward and
backward run on the library's kernels, and the backward without the interpreter; what is saved between them follows
the reference's Functions (fairseq/modules/norm_layer/timestep_norm.py:14-66, sequence_norm.py:12-52,
fairseq/modules/fused_ops/{fftconv,ema_parameters,ema_hidden}.py)."""
import torch
from torch.nn.modules.module import _has_any_global_hook

from . import _lib, ops


def needs_grad(*tensors):
    return torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)


def plain(module, *types):
    """Whether calling the module is its class's forward and nothing else: one of these classes itself (an adapter, a
    quantised or a sharded layer is another), no forward of its own, no hooks.  Only then may a path take the module's
    parameters instead of calling it."""
    d = module.__dict__
    return (type(module) in types and "forward" not in d
            and not (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"])
            and not _has_any_global_hook())


def ema(x, alpha, delta, third, gamma, omega, padding_mask, bidirectional, shift, truncation=None, complex_poles=False,
        silu=False, channels_last=False):
    """y = EMA(x) [then SiLU] for x (B, D, L), with ``channels_last`` (B, L, D), from the layer's raw parameters; ``third`` is beta (real poles) or
    theta (complex ones)."""
    return _lib.host().ema_train(x, alpha, delta, third, gamma, omega, padding_mask, ops._flags(bidirectional, shift, False),
                                 ops._trunc(truncation), complex_poles, silu, channels_last)


def timestep_norm(x, prior_count, prior_mean, prior_logv, weight, bias, padding_mask, num_groups, eps):
    """y = TimestepNorm(x (B, L, D)) from the module's parameters.  Per-feature statistics (channels contiguous) are
    taken again in the backward, so only the arguments are kept; otherwise the statistics of every step are."""
    return _lib.host().timestep_norm_train(x, prior_count, prior_mean, prior_logv, weight, bias, padding_mask,
                                           0 if num_groups is None else num_groups, eps)


def sequence_norm(x, weight, bias, padding_mask, eps, length_last, num_groups=None):
    """y = SequenceNorm(x), per channel or per channel group, from the module's parameters."""
    return _lib.host().sequence_norm_train(x, weight, bias, padding_mask, eps, length_last,
                                           0 if num_groups is None else num_groups)
