"""fp32 rows on the tensor pipe: no further from float64 than the fp32 recurrence.

That recurrence, with its sums in fp32, is 1.05e-7 to 1.18e-7 (bidirectional, behind SequenceNorm) and 6.6e-8 to 7.3e-8 (causal)
of the result's norm off over these shapes; the rounding of the result alone is 3.4e-8."""
import pytest
import torch

from _util import rel_l2

pytestmark = pytest.mark.gpu


def _taps(q, c, length):
    t = torch.arange(length, dtype=torch.float64, device=q.device)
    return sum(torch.exp(t * torch.log(q[:, n:n + 1])) * c[:, n:n + 1] for n in range(q.size(1)))


@pytest.mark.parametrize("bidir", [False, True])
@pytest.mark.parametrize("bsz,length,dim", [(8, 4151, 64), (12, 624, 96), (6, 13194, 32)])
def test_error_of_fp32_rows(bidir, bsz, length, dim):
    import fairseq_apollo_b200 as M
    from fairseq_apollo_b200 import _lib
    from oracle import mega_oracle as O
    torch.manual_seed(length)
    norm, move = M.SequenceNorm(dim).cuda(), M.MultiHeadEMA(dim, ndim=16, bidirectional=bidir).cuda().eval()
    x = torch.randn(bsz, dim, length, device="cuda") * 1.1 + 0.05
    p, q, g = O.ema_coeffs(*(t.detach() for t in (move.alpha, move.delta, move.beta, move.gamma)), dtype=torch.float64)
    xd = x.double()
    with torch.no_grad():
        if bidir:
            y = M.sequence_norm_ema(norm, move, x)
            xd = (xd - xd.mean(-1, keepdim=True)) * (xd.var(-1, unbiased=False, keepdim=True) + norm.eps).rsqrt()
        else:
            y = move(x)
    assert _lib.last_kernel() == "rowres"
    n = 2 * length
    kernel = torch.zeros(dim, n, dtype=torch.float64, device="cuda")
    kernel[:, :length] = _taps(q[:dim], (p * g)[:dim], length)
    if bidir:
        kernel[:, n - length + 1:] += _taps(q[dim:], (p * g)[dim:], length)[:, :length - 1].flip(-1)
    want = torch.fft.irfft(torch.fft.rfft(xd, n=n) * torch.fft.rfft(kernel), n=n)[..., :length] + xd * move.omega.detach().double().view(dim, 1)
    assert rel_l2(y, want) < (1.18e-7 if bidir else 7.3e-8)
