"""Channel counts that 16 bytes do not divide, in rows that start at 16-byte boundaries (a slice of a wider tensor): the EMA's
forms over time, forward and backward, against the float64 oracle.  What stands behind the last channel is not read."""
import pytest
import torch

from _util import make_ema_params, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,wide", [(37, 40), (65, 72), (1, 8)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("form", ["real", "complex", "bidirectional"])
def test_slices_of_wider_rows(dim, wide, dtype, form):
    from fairseq_apollo_b200 import functions, ops
    from oracle import mega_oracle as O
    gen = torch.Generator().manual_seed(dim)
    bsz, length, bidir, cplx = 2, 150, form == "bidirectional", form == "complex"
    prm = make_ema_params(gen, dim, 16, bidirectional=bidir)
    if cplx:
        prm[2], prm[3] = torch.randn(dim, 1, 1, generator=gen), torch.randn(dim, 16, 2, generator=gen)
    x, dy = (torch.randn(bsz, length, dim, generator=gen).to(dtype) for _ in range(2))
    fwd = O.cema_forward_recurrence if cplx else O.ema_forward_recurrence
    xr = x.double().transpose(1, 2).requires_grad_(True)
    leaves = [p.double().requires_grad_(True) for p in prm]
    want = fwd(xr, *leaves, bidirectional=bidir)
    want.backward(dy.double().transpose(1, 2))

    def slice_of(t):
        w = torch.full((bsz, length, wide), float("nan"), dtype=dtype, device="cuda")
        w[..., :dim] = t.cuda()
        return w[..., :dim]
    dev = [p.cuda().requires_grad_(True) for p in prm]
    xg = slice_of(x).detach().requires_grad_(True)
    y = functions.ema(xg, *dev, None, bidir, True, None, cplx, False, True)
    y.backward(slice_of(dy))
    limit = 5e-6 if dtype == torch.float32 else 2.0 ** -8
    assert rel_l2(y, want.transpose(1, 2)) < limit
    assert rel_l2(xg.grad, xr.grad.transpose(1, 2)) < 4 * limit
    for a, b in zip(dev, leaves):
        assert rel_l2(a.grad, b.grad) < 1e-4
    with torch.no_grad():
        co = (ops.cema_coeffs if cplx else ops.ema_coeffs)(*dev[:4])
        out = (ops.cema_forward if cplx else ops.ema_forward)(slice_of(x).transpose(1, 2), *co, dev[4], bidirectional=bidir)
    assert rel_l2(out, want) < limit
