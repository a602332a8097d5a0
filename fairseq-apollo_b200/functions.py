"""autograd Functions of the training path: forward and backward both run on the library's
kernels; what is saved between them follows the reference's Functions
(fairseq/modules/norm_layer/timestep_norm.py:14-66, sequence_norm.py:12-52,
fairseq/modules/fused_ops/{fftconv,ema_parameters,ema_hidden}.py)."""
import torch

from . import ops


def needs_grad(*tensors):
    return torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)


class EMAFunction(torch.autograd.Function):
    """y = EMA(x) for x (B, D, L): coefficients, convolution, mask and omega residual in one
    forward kernel; one backward kernel for (dx, dp, dq, dgamma_hat, domega) and a small one for
    the chain rule to (alpha, delta, beta, gamma)."""

    @staticmethod
    def forward(ctx, x, alpha, delta, beta, gamma, omega, padding_mask, bidirectional, shift, truncation=None):
        p, q, g = ops.ema_coeffs(alpha, delta, beta, gamma)
        y = ops.ema_forward(x, p, q, g, omega, padding_mask, None, False, bidirectional=bidirectional,
                            shift=shift, truncation=truncation)
        ctx.save_for_backward(x, alpha, delta, beta, omega, padding_mask, p, q, g)
        ctx.bidirectional, ctx.shift, ctx.truncation = bidirectional, shift, truncation
        return y

    @staticmethod
    def backward(ctx, dy):
        x, alpha, delta, beta, omega, padding_mask, p, q, g = ctx.saved_tensors
        dx, dp, dq, dg, dom, _ = ops.ema_backward(dy, x, p, q, g, omega, padding_mask,
                                                  bidirectional=ctx.bidirectional, shift=ctx.shift,
                                                  truncation=ctx.truncation)
        da, dd, db, dgm = ops.ema_coeffs_bwd(alpha, delta, beta, dp, dq, dg, alpha.dtype)
        return (dx, da, dd.to(delta.dtype), db.to(beta.dtype), dgm, dom.to(omega.dtype), None, None, None, None)


class ComplexEMAFunction(torch.autograd.Function):
    """y = complex EMA(x) for x (B, D, L); parameters alpha, delta (K, N, 1), theta (K, 1, 1),
    gamma (K, N, 2), omega (D, 1) as in MultiHeadComplexEMA."""

    @staticmethod
    def forward(ctx, x, alpha, delta, theta, gamma, omega, padding_mask, bidirectional, shift, truncation=None):
        p, q, g = ops.cema_coeffs(alpha, delta, theta, gamma)
        y = ops.cema_forward(x, p, q, g, omega, padding_mask, None, False, bidirectional=bidirectional, shift=shift,
                             truncation=truncation)
        ctx.save_for_backward(x, alpha, delta, theta, omega, padding_mask, p, q, g)
        ctx.bidirectional, ctx.shift, ctx.truncation = bidirectional, shift, truncation
        ctx.gamma_dtype = gamma.dtype
        return y

    @staticmethod
    def backward(ctx, dy):
        x, alpha, delta, theta, omega, padding_mask, p, q, g = ctx.saved_tensors
        dx, dp, dq, dg, dom = ops.cema_backward(dy, x, p, q, g, omega, padding_mask,
                                                bidirectional=ctx.bidirectional, shift=ctx.shift,
                                                truncation=ctx.truncation)
        da, dd, dt, dgm = ops.cema_coeffs_bwd(alpha, delta, theta, q, dp, dq, dg, alpha.dtype)
        return (dx, da, dd.to(delta.dtype), dt.to(theta.dtype), dgm.to(ctx.gamma_dtype),
                dom.view_as(omega).to(omega.dtype), None, None, None, None)


class TimestepNormFunction(torch.autograd.Function):
    """y = TimestepNorm(x (B, L, D)) from the module's own parameters.  Per-feature statistics (channels contiguous)
    are taken again in the backward, so only the arguments are kept; otherwise the statistics of every step are."""

    @staticmethod
    def forward(ctx, x, prior_count, prior_mean, prior_logv, weight, bias, padding_mask, num_groups, eps):
        gamma, beta, prev_count, prev_mean, prev_var = ops.norm_prepare(weight, bias, (prior_count, prior_mean, prior_logv),
                                                                        x.shape[0])
        ctx.recompute = num_groups is None and ops.timestep_norm_keeps_nothing(x)
        if ctx.recompute:
            y, _, _, _ = ops.timestep_norm_fwd(x, prev_count, prev_mean, prev_var, gamma, beta, padding_mask, eps)
            ctx.save_for_backward(x, prior_logv, prev_count, prev_mean, prev_var, gamma, padding_mask)
        else:
            y, count, _, _, cummean, cumrstd, group_mean = ops.timestep_norm_fwd_train(
                x, prev_count, prev_mean, prev_var, gamma, beta, padding_mask, eps, num_groups)
            ctx.save_for_backward(x, prior_logv, prev_mean, count, cummean, cumrstd, group_mean, gamma, padding_mask)
        ctx.num_groups, ctx.eps = num_groups, eps
        return y

    @staticmethod
    def backward(ctx, dy):
        if ctx.recompute:
            x, prior_logv, prev_count, prev_mean, prev_var, gamma, padding_mask = ctx.saved_tensors
            dx, dpm, dpv, dgamma, dbeta = ops.timestep_norm_bwd_stats(dy, None, None, x, prev_count, prev_mean, prev_var,
                                                                      gamma, padding_mask, ctx.eps)
        else:
            x, prior_logv, prev_mean, count, cummean, cumrstd, group_mean, gamma, padding_mask = ctx.saved_tensors
            dx, dpm, dpv, dgamma, dbeta = ops.timestep_norm_bwd(dy, None, None, x, prev_mean, count, cummean, cumrstd,
                                                                group_mean, gamma, padding_mask, ctx.num_groups)
        need = ctx.needs_input_grad
        dw, db, dm, dl = ops.norm_finish(prior_logv, dgamma, dbeta, dpm, dpv, prior_logv)
        return dx, None, dm if need[2] else None, dl if need[3] else None, dw, db, None, None, None


class SequenceNormFunction(torch.autograd.Function):
    """y = SequenceNorm(x), per channel or per channel group, from the module's own parameters."""

    @staticmethod
    def forward(ctx, x, weight, bias, padding_mask, eps, length_last, num_groups=None):
        gamma, beta = ops.norm_prepare(weight, bias)
        y, count, mean, rstd = ops.sequence_norm_fwd(x, gamma, beta, padding_mask, eps, length_last, num_groups)
        ctx.save_for_backward(x, weight, count, mean, rstd, gamma, padding_mask)
        ctx.length_last = length_last
        ctx.num_groups = num_groups
        return y

    @staticmethod
    def backward(ctx, dy):
        x, weight, count, mean, rstd, gamma, padding_mask = ctx.saved_tensors
        dx, dgamma, dbeta = ops.sequence_norm_bwd(dy, x, count, mean, rstd, gamma, padding_mask, ctx.length_last,
                                                  ctx.num_groups)
        dw, db = ops.norm_finish(weight, dgamma, dbeta)
        return dx, dw, db, None, None, None, None
