"""TimestepNorm, per feature and per group, forward and backward, and SequenceNorm at the edges of their splits over time:
segments of at least 64 steps, tiles of 8 or 16 steps, 64 channels of a warp, 256 or 128 threads along time of a group.

Reference: the running statistics written out in float64 as cumulative sums, and autograd through them.  fp32: sums of L
values about a centre, a handful of approximate reciprocals and square roots (2^-22 each) per step: 1e-5 relative 2-norm;
the gradients of the priors and affine are sums over batch and time that cancel, 1e-4.  bf16: half a unit of inputs that
are already rounded, 2^-8 through dx's three terms."""
import pytest
import torch

from _util import rel_l2

pytestmark = pytest.mark.gpu


def _reference(x, mask, count, mean, logv, weight, bias, groups, eps):
    bsz, length, dim = x.shape
    g = groups or dim
    xg = x.view(bsz, length, g, dim // g)
    keep = torch.ones(bsz, length, 1, dtype=x.dtype) if mask is None else (~mask).to(x.dtype).unsqueeze(-1)
    m, q = xg.mean(-1) * keep, xg.pow(2).mean(-1) * keep
    n0 = count.to(x.dtype).view(-1, 1, 1)
    n = n0 + keep.cumsum(1)
    mu0, v0 = mean.view(1, 1, g), logv.exp().view(1, 1, g)
    u = (n0 * mu0 + m.cumsum(1)) / n
    var = (n0 * (v0 + mu0 * mu0) + q.cumsum(1)) / n - u * u
    y = ((xg - u.unsqueeze(-1)) * (var + eps).rsqrt().unsqueeze(-1)).reshape(bsz, length, dim)
    return (y * (weight + 1.0) + bias) * keep


@pytest.mark.parametrize("length,bsz,dim,groups,dtype,masked", [
    (1, 2, 64, None, torch.float32, False),
    (63, 1, 40, None, torch.float32, True),        # one short segment, channels beyond a warp's
    (129, 3, 72, None, torch.bfloat16, False),     # a third segment of one step
    (1000, 2, 136, None, torch.float32, True),
    (127, 2, 64, 4, torch.float32, False),         # fewer steps than threads along time
    (129, 1, 96, 3, torch.float32, True),
    (1100, 2, 128, 2, torch.bfloat16, False),      # nine steps per thread: a batch of loads and one over
    (2200, 2, 128, 2, torch.bfloat16, False),      # the same with 256 threads along time
    (255, 1, 64, 4, torch.float32, False),
    (257, 1, 96, 3, torch.float32, True),
    (127, 40, 64, 8, torch.float32, False),        # more pairs of groups than SMs: eight to a block, 128 threads along time
    (129, 50, 96, 6, torch.float32, True),         # eight to a block, two of them there are not
    (1100, 75, 64, 4, torch.bfloat16, False),
])
def test_timestep_norm_tiles(length, bsz, dim, groups, dtype, masked):
    import fairseq_apollo_b200 as M
    gen = torch.Generator().manual_seed(length)
    norm = M.TimestepNorm(dim, num_groups=groups, prior_count=3).train()
    with torch.no_grad():
        for p in norm.parameters():
            p.copy_(torch.randn(p.shape, generator=gen) * 0.3)
    mask = None
    if masked:
        mask = torch.zeros(bsz, length, dtype=torch.bool)
        mask[0, 2:9] = True
        mask[-1, length - length // 3:] = True
    x = (torch.randn(bsz, length, dim, generator=gen) * 1.2 + 0.4).to(dtype)
    dy = torch.randn(bsz, length, dim, generator=gen).to(dtype)
    ref = {n: p.detach().double().requires_grad_(True) for n, p in norm.named_parameters()}
    xr = x.double().requires_grad_(True)
    yr = _reference(xr, mask, torch.full((bsz,), 3), ref["prior_mean"].flatten(), ref["prior_logv"].flatten(), ref["weight"],
                    ref["bias"], groups, norm.eps)
    yr.backward(dy.double())
    norm = norm.cuda()
    xg = x.cuda().requires_grad_(True)
    y = norm(xg, None if mask is None else mask.cuda())
    y.backward(dy.cuda())
    fp32 = dtype == torch.float32
    assert rel_l2(y, yr) < (1e-5 if fp32 else 2.0 ** -8)
    assert rel_l2(xg.grad, xr.grad) < (1e-4 if fp32 else 2.0 ** -8)
    for name, p in norm.named_parameters():
        assert rel_l2(p.grad, ref[name].grad) < (1e-4 if fp32 else 2.0 ** -8), name


@pytest.mark.parametrize("length,bsz,dim,masked", [(1, 1, 32, False), (65, 2, 40, True), (515, 3, 96, True)])
def test_sequence_norm_channels_last_tiles(length, bsz, dim, masked):
    import fairseq_apollo_b200 as M
    gen = torch.Generator().manual_seed(length)
    norm = M.SequenceNorm(dim).train()
    with torch.no_grad():
        for p in norm.parameters():
            p.copy_(torch.randn(p.shape, generator=gen) * 0.3)
    keep = torch.ones(bsz, length, 1, dtype=torch.float64)
    if masked:
        keep[0, 3:10] = 0
        keep[-1, length // 2:] = 0
    x = torch.randn(bsz, length, dim, generator=gen) * 1.2 + 0.4
    dy = torch.randn(bsz, length, dim, generator=gen)
    w, b = (p.detach().double().requires_grad_(True) for p in (norm.weight, norm.bias))
    xr = x.double().requires_grad_(True)
    n = keep.sum(1, keepdim=True)
    u = (xr * keep).sum(1, keepdim=True) / n
    var = ((xr - u).pow(2) * keep).sum(1, keepdim=True) / n
    yr = ((xr - u) * (var + norm.eps).rsqrt() * (w + 1.0) + b) * keep
    yr.backward(dy.double())
    norm = norm.cuda()
    xg = x.cuda().requires_grad_(True)
    y = norm(xg, (keep[..., 0] == 0).cuda() if masked else None, length_last=False)
    y.backward(dy.cuda())
    assert rel_l2(y, yr) < 1e-5
    assert float((xg.grad.cpu().double() - xr.grad).norm()) < 1e-5 * float(dy.norm()) * float((var.detach().min() + norm.eps).rsqrt())
    assert rel_l2(norm.weight.grad, w.grad) < 1e-4 or length == 1   # (one position: the normalised input is zero)
    assert rel_l2(norm.bias.grad, b.grad) < 1e-5


@pytest.mark.parametrize("bsz,length,dim,cplx,xn", [(32, 128, 1024, False, True), (32, 64, 1024, True, False), (2, 2080, 96, False, False)])
def test_norm_ema_forms_agree(bsz, length, dim, cplx, xn):
    """The fused chain (1), its parts in turn (2) and the scan (3) on the same bf16 input.  Each rounds the normalised
    activations at most once more than the output: 2^-8 apart; statistics are fp32, from tf32 products in the chain."""
    from fairseq_apollo_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(length)
    rnd = lambda *s: torch.rand(*s, generator=gen, device="cuda")   # noqa: E731
    x = (torch.randn(bsz, length, dim, generator=gen, device="cuda") * 1.1 + 0.1).bfloat16()
    q = rnd(dim, 16) * 0.5 + 0.45
    g = (rnd(dim, 16) - 0.5) * 0.6
    if cplx:
        q, g = torch.polar(q, rnd(dim, 16) * 3.0), torch.complex(g, g.flip(1))
    args = (x, torch.full((bsz,), 2, device="cuda"), torch.zeros(bsz, dim, device="cuda"), torch.ones(bsz, dim, device="cuda"),
            rnd(dim) + 0.5, rnd(dim), 1e-5, rnd(dim, 16), q, g, rnd(dim))
    res = []
    for form in (1, 2, 3):
        _lib.set_option(5, form)
        try:
            res.append(ops.tsn_ema_forward(*args, None, None, True, True, xn, cplx))
        finally:
            _lib.set_option(5, 0)
    for r in res[1:]:
        assert rel_l2(r["y"].float(), res[0]["y"].float()) < 2.0 ** -7
        assert rel_l2(torch.view_as_real(r["h"]) if cplx else r["h"], torch.view_as_real(res[0]["h"]) if cplx else res[0]["h"]) < 2.0 ** -7
        assert rel_l2(r["mean"], res[0]["mean"]) < 1e-3 and rel_l2(r["var"], res[0]["var"]) < 1e-3
        assert torch.equal(r["count"], res[0]["count"])
        if xn:
            assert rel_l2(r["xn"].float(), res[0]["xn"].float()) < 2.0 ** -7


# Operands are bf16 (2^-9 each), squares about the first value tf32 (2^-10 of a variance): as with a prior.
@pytest.mark.parametrize("tile,cplx,masked", [
    (2, False, False), (4, False, False), (7, False, False), (8, False, False), (22, False, False), (71, False, False), (222, False, False),
    (224, False, False), (422, False, False), (124, False, False), (84, False, False), (16, False, False), (14, False, False),
    (7, False, True), (22, False, True), (16, False, True), (0, True, False)])
@pytest.mark.parametrize("normed", [False, True])
def test_first_values_without_a_prior(tile, cplx, masked, normed):
    """bf16, no count to begin with (the module's default), values far from zero: variances of the first few values, whose squares are
    large, and nothing counted ahead of them."""
    from fairseq_apollo_b200 import _lib, ops
    from oracle import mega_oracle as O
    gen = torch.Generator().manual_seed(tile + 1)
    bsz, length, dim = 9, 128 * 2 if tile == 84 else 96, 72
    rnd = lambda *s: torch.rand(*s, generator=gen)   # noqa: E731
    x = (torch.randn(bsz, length, dim, generator=gen) + 3.0).bfloat16()
    count = torch.zeros(bsz, dtype=torch.int64)
    count[4] = 2
    mean, var, gamma, beta = 3.0 * (count > 0).float()[:, None].expand(bsz, dim).contiguous(), torch.ones(bsz, dim), rnd(dim) + 0.5, rnd(dim) - 0.5
    mask = None
    if masked:
        mask = torch.zeros(bsz, length, dtype=torch.bool)
        mask[0, :41] = True
        mask[1, :5] = True
        mask[2, 30:] = True
        mask[3] = True
    p, q, g, om = rnd(dim, 16) * 0.2, rnd(dim, 16) * 0.5 + 0.45, rnd(dim, 16) - 0.5, rnd(dim)
    if cplx:
        q, g = torch.polar(q, rnd(dim, 16) * 3.0), torch.complex(g, g.flip(1))
    args = [t.cuda() for t in (x, count, mean, var, gamma, beta)] + [1e-5] + [t.cuda() for t in (p, q, g, om)]
    _lib.set_option(2, tile)
    _lib.set_option(5, 1)
    try:
        r = ops.tsn_ema_forward(*args, None if mask is None else mask.cuda(), want_normed=normed, **({"complex_poles": True} if cplx else {}))
        assert "tsn_ema_mma" in _lib.last_kernel()
        alone = ops.timestep_norm_fwd(*args[:6], None if mask is None else mask.cuda())
    finally:
        _lib.set_option(2, 0)
        _lib.set_option(5, 0)
    xn, cnt, mean, var = O.timestep_norm(x.double(), count, mean.double(), var.double(), gamma.double(), beta.double(), mask, acc_dtype=torch.float64)[:4]
    h, ys = torch.zeros(bsz, dim, 16, dtype=torch.complex128), []
    for t in range(length):
        h = q.to(torch.complex128) * h + p.double() * xn[:, t, :, None]
        ys.append((h * g.to(torch.complex128)).real.sum(-1) + om.double() * xn[:, t])
    assert rel_l2(r["y"].float(), torch.stack(ys, 1)) < 1e-2
    if normed:
        assert rel_l2(r["xn"].float(), xn) < 6e-3
    assert rel_l2(alone[0].float(), xn) < 6e-3
    assert torch.equal(r["count"].cpu(), cnt) and torch.equal(alone[1].cpu(), cnt)
    for m, v in ((r["mean"], r["var"]), alone[2:4]):
        assert rel_l2(m, mean) < 1e-4 and rel_l2(v, var) < 2e-3


def test_form_of_the_norm_alone_leaves_the_pair():
    """The form asked for of TimestepNorm by itself (4) is none of the pair, which runs as always."""
    from fairseq_apollo_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(9)
    rnd = lambda *s: torch.rand(*s, generator=gen, device="cuda")   # noqa: E731
    bsz, length, dim = 8, 1024, 2048
    x = torch.randn(bsz, length, dim, generator=gen, device="cuda").bfloat16()
    args = (x, torch.full((bsz,), 2, device="cuda"), rnd(bsz, dim) - 0.5, rnd(bsz, dim) + 0.5, rnd(dim) + 0.5, rnd(dim), 1e-5,
            rnd(dim, 16), rnd(dim, 16) * 0.5 + 0.45, rnd(dim, 16) - 0.5, rnd(dim))
    res = []
    for form in (0, 4):
        _lib.set_option(5, form)
        try:
            res.append((ops.tsn_ema_forward(*args)["y"], _lib.last_kernel()))
        finally:
            _lib.set_option(5, 0)
    assert res[0][1] == res[1][1] and torch.equal(res[0][0], res[1][0])


# The first step has no variance: its terms, of size eps^-1/2 = 316, cancel against what the later steps carry back, and leave what
# approximate roots and reciprocals (2^-22) and sums of a handful of such terms leave: 316 x 2^-20 of gradients of size one.  16 bits:
# the rounding of the output beside that.
@pytest.mark.parametrize("dtype,rounding", [(torch.float32, 0.0), (torch.bfloat16, 2.0 ** -9), (torch.float16, 2.0 ** -12)])
@pytest.mark.parametrize("length,dim,lead", [(64, 8, 0), (300, 72, 70), (1111, 136, 3)])
def test_backward_without_a_prior(dtype, rounding, length, dim, lead):
    """Nothing came in and the first steps (a whole segment of 64 and more) are padded: the first step that counts is the centre."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(length)
    bsz = 3
    x = (torch.randn(bsz, length, dim, generator=gen) + 100.0).to(dtype)
    dy = torch.randn(bsz, length, dim, generator=gen).to(dtype)
    gamma, dmean, dvar = torch.randn(dim, generator=gen), torch.randn(bsz, dim, generator=gen), torch.randn(bsz, dim, generator=gen)
    mask = torch.zeros(bsz, length, dtype=torch.bool)
    mask[1, :lead] = True
    mask[2, length // 2:length // 2 + 9] = True
    zero = torch.zeros(bsz, dim)
    got = ops.timestep_norm_bwd_stats(*[t.cuda() for t in (dy, dmean, dvar, x, torch.zeros(bsz, dtype=torch.int64), zero, zero + 1, gamma, mask)])
    xd, gd = x.double().requires_grad_(True), gamma.double().requires_grad_(True)
    keep = (~mask).double()[..., None]
    count = keep.cumsum(1).clamp(min=1)
    about = torch.stack([xd.detach()[b, int((~mask[b]).nonzero()[0])] for b in range(bsz)])[:, None]
    dev = (xd - about) * keep
    mean = dev.cumsum(1) / count
    var = (dev * dev).cumsum(1) / count - mean * mean
    y = (dev - mean) * (var.clamp(min=0) + 1e-5).rsqrt() * gd * keep
    total = (y * dy.double()).sum() + (mean[:, -1] * dmean.double()).sum() + (var[:, -1] * dvar.double()).sum()
    dx, dgamma = torch.autograd.grad(total, (xd, gd))
    assert rel_l2(got[0].float(), dx) < 316 * 2.0 ** -20 + rounding
    assert rel_l2(got[3], dgamma) < 1e-5
    assert rel_l2(got[4], (dy.double() * keep).sum((0, 1))) < 1e-5
    assert (got[0].cpu()[mask] == 0).all()
