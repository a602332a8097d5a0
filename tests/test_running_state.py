"""What a call leaves behind for the next one: exported pole states, running statistics updated in place, counts.

The forms that run in fp32 throughout keep a state to 1e-5 of its norm (sums of L rounded terms); a form with bf16 operands
would be 1e-3 off."""
import pytest
import torch

from _util import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture
def option():
    from fairseq_apollo_b200 import _lib
    yield _lib.set_option
    for key in (1, 5):
        _lib.set_option(key, 0)


@pytest.mark.parametrize("split", [1, 0])
@pytest.mark.parametrize("normed", [False, True])
def test_ragged_complex_prefill_state(split, normed, option):
    """bf16, a length that 32 does not divide: the exported state is that of an fp32 recurrence."""
    import fairseq_apollo_b200 as M
    from oracle import mega_oracle as O
    torch.manual_seed(7)
    bsz, length, dim = 6, 333, 64
    norm, move = M.TimestepNorm(dim, prior_count=2).cuda().eval(), M.MultiHeadComplexEMA(dim, ndim=16).cuda().eval()
    x = torch.randn(bsz, length, dim, device="cuda").bfloat16()
    inc = {}
    option(5, split)
    with torch.no_grad():
        M.timestep_norm_ema(norm, move, x, None, inc, "silu" if normed else None, normed)
    state = {n: t for d in inc.values() for n, t in d.items()}
    one = torch.ones(dim, dtype=torch.float64)
    xn, _, mean, var = O.timestep_norm(x.cpu().double(), torch.full((bsz,), 2), torch.zeros(bsz, dim).double(),
                                       torch.ones(bsz, dim).double(), one, 0 * one, acc_dtype=torch.float64)
    prm = [t.detach().cpu() for t in (move.alpha, move.delta, move.theta, move.gamma, move.omega)]
    _, h = O.cema_forward_recurrence(xn.transpose(1, 2), *prm, return_state=True)
    got = state["prev_state"].cpu().to(torch.complex128)
    assert float((got - h).norm() / h.norm()) < 1e-5
    assert rel_l2(state["prev_mean"], mean) < 1e-5 and rel_l2(state["prev_var"], var) < 1e-5


def _taps(q, c, length, lag=0):
    """sum_n c q^(t + lag) for t < length, (D, length) float64"""
    t = torch.arange(lag, length + lag, dtype=torch.float64)
    out = 0
    for n in range(q.size(1)):
        v = torch.exp(t * torch.log(q[:, n:n + 1])) * c[:, n:n + 1]
        out = out + (v.real if v.is_complex() else v)
    return out


@pytest.mark.parametrize("cplx", [False, True])
def test_bidirectional_beyond_a_quarter_million(cplx):
    """More segments of 64 positions than 4096; forward and input gradient against a convolution in float64."""
    import math
    from fairseq_apollo_b200 import functions, ops
    gen = torch.Generator().manual_seed(3)
    dim, ndim, length = 8, 4, 4096 * 64 + 1
    alpha, delta = torch.randn(2 * dim, ndim, 1, generator=gen), torch.randn(2 * dim, ndim, 1, generator=gen)
    third = torch.randn(2 * dim, 1 if cplx else ndim, 1, generator=gen)
    gamma = torch.randn(2 * dim, ndim, 2, generator=gen) if cplx else torch.randn(2 * dim, ndim, generator=gen)
    omega = torch.randn(dim, generator=gen)
    from oracle import mega_oracle as O
    p, q, g = (O.cema_coeffs if cplx else O.ema_coeffs)(alpha, delta, third, gamma, dtype=torch.float64)
    x, dy = torch.randn(1, length, dim, generator=gen), torch.randn(1, length, dim, generator=gen)
    xg = x.cuda().requires_grad_(True)
    y = functions.ema(xg, *(t.cuda() for t in (alpha, delta, third, gamma, omega)), None, True, True, None, cplx, False, True)
    y.backward(dy.cuda())
    n = 2 * length
    right, left = _taps(q[:dim], p[:dim] * g[:dim], length), _taps(q[dim:], p[dim:] * g[dim:], length)
    kernel = torch.zeros(dim, n, dtype=torch.float64)
    kernel[:, :length] = right
    kernel[:, n - length + 1:] += left[:, :length - 1].flip(-1)    # lag -1 - k
    kernel[:, 0] += omega.double()
    kf = torch.fft.rfft(kernel)
    conv = lambda t, k: torch.fft.irfft(torch.fft.rfft(t[0].t().double(), n=n) * k, n=n)[:, :length].t()
    assert rel_l2(y[0], conv(x, kf)) < 5e-6
    assert rel_l2(xg.grad[0], conv(dy, kf.conj())) < 5e-6
    with torch.no_grad():
        cf = ops.cema_coeffs if cplx else ops.ema_coeffs
        out = (ops.cema_forward if cplx else ops.ema_forward)(
            xg.transpose(1, 2), *cf(*(t.cuda() for t in (alpha, delta, third, gamma))), omega.cuda(), bidirectional=True)
    assert rel_l2(out[0].t(), conv(x, kf)) < 5e-6
