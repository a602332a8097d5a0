"""The causal EMA's backward with states carried in and out: on the streamed kernel where channels are contiguous, the same as
the generic one (fp32 sums of at most B L terms in another order: 1e-4; dx 2e-5)."""
import pytest
import torch

from _util import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bsz,length,dim,ndim", [(2, 1, 64, 16), (3, 33, 72, 5), (1, 257, 8, 16), (2, 100, 136, 16)])
@pytest.mark.parametrize("masked", [False, True])
def test_states_on_the_streamed_kernel(bsz, length, dim, ndim, masked):
    from fairseq_apollo_b200 import _lib, ops
    gen = torch.Generator().manual_seed(length)
    r = lambda *s: torch.randn(*s, generator=gen).cuda()
    x, dy = r(bsz, length, dim).transpose(1, 2), r(bsz, length, dim).transpose(1, 2)
    p, q, g, om = r(dim, ndim), torch.rand(dim, ndim, generator=gen).cuda() * 0.8 + 0.1, r(dim, ndim), r(dim)
    h, dh = r(bsz, dim, ndim), r(bsz, dim, ndim)
    mask = None
    if masked:
        mask = torch.zeros(bsz, length, dtype=torch.bool, device="cuda")
        mask[-1, length // 2:] = True
    got = ops.ema_backward(dy, x, p, q, g, om, mask, h, dh, want_dh_in=True)
    assert _lib.last_kernel() == "ema_bwd_stream"
    want = ops.ema_backward(dy.contiguous(), x.contiguous(), p, q, g, om, mask, h, dh, want_dh_in=True)
    assert length == 1 or _lib.last_kernel() != "ema_bwd_stream"
    for i, (a, b) in enumerate(zip(got, want)):
        assert rel_l2(a, b) < (2e-5 if i in (0, 5) else 1e-4), i
