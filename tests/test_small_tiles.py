"""The EMA's backward at the edges of its segments (32 steps, four per block, 32 channels of a warp), the element-wise gates
at the edges of their blocks, the query / key affine with a pitch and a cache, and softmax rows by warps.

EMA: float64 convolution with the layer's taps, autograd through it.  fp32 sums of L terms, parameter gradients over batch
and time: 2e-5 relative 2-norm.  Gates and softmax: the same formula in fp32; 16-bit results are rounded once, by at most
2^-8 of a bf16 value (8 significant bits) and 2^-11 of an fp16 one, from tanh.approx (2^-11) or exp in fp32."""
import pytest
import torch

from _util import make_ema_params, rel_l2, right_pad_mask

pytestmark = pytest.mark.gpu


def _taps(O, prm, cplx, length):
    t = torch.arange(length, dtype=torch.float64)
    if cplx:
        p, q, g = O.cema_coeffs(*prm[:4], dtype=torch.float64)
        return (p.unsqueeze(-1) * g.unsqueeze(-1) * q.unsqueeze(-1) ** t).sum(1).real
    p, q, g = O.ema_coeffs(*prm[:4], dtype=torch.float64)
    return (p.unsqueeze(-1) * g.unsqueeze(-1) * q.unsqueeze(-1) ** t).sum(1)


@pytest.mark.parametrize("length,bsz,dim", [(1, 1, 8), (31, 2, 40), (33, 1, 32), (130, 3, 72), (300, 2, 36)])
@pytest.mark.parametrize("cplx,bidir,masked", [(False, False, False), (False, True, True), (True, False, True), (True, True, False)])
def test_ema_backward_segments(length, bsz, dim, cplx, bidir, masked):
    from fairseq_apollo_b200.functions import ema
    from oracle import mega_oracle as O
    gen = torch.Generator().manual_seed(length)
    prm = make_ema_params(gen, dim, 16, bidirectional=bidir)
    k = 2 * dim if bidir else dim
    if cplx:
        prm[2], prm[3] = torch.randn(k, 1, 1, generator=gen), torch.randn(k, 16, 2, generator=gen)
    x, dy = (torch.randn(bsz, length, dim, generator=gen) for _ in range(2))
    mask = right_pad_mask(gen, bsz, length, 0.6) if masked else None
    ref = [t.double().requires_grad_(True) for t in (x, *prm)]
    keep = torch.ones(bsz, length, 1, dtype=torch.float64) if mask is None else (~mask).double().unsqueeze(-1)
    xm = (ref[0] * keep).transpose(1, 2)
    taps = _taps(O, ref[1:], cplx, length)
    lag = torch.arange(length).view(-1, 1) - torch.arange(length).view(1, -1)   # (t, s): t - s
    mat = taps[:dim][:, lag.clamp(min=0)] * (lag >= 0)
    if bidir:   # the anti-causal half starts at lag one
        mat = mat + taps[dim:][:, (-lag - 1).clamp(min=0)] * (lag < 0)
    yr = torch.einsum('dts,bds->btd', mat, xm) + ref[0] * ref[5]
    yr.backward(dy.double())
    dev = [t.cuda().requires_grad_(True) for t in (x, *prm)]
    y = ema(*dev, None if mask is None else mask.cuda(), bidir, True, None, cplx, False, channels_last=True)
    y.backward(dy.cuda())
    assert rel_l2(y, yr) < 1e-5
    for a, b in zip(dev, ref):
        assert rel_l2(a.grad, b.grad) < 2e-5 or float(b.grad.norm()) < 1e-12


@pytest.mark.parametrize("rows,cols,dtype", [(1, 8, torch.bfloat16), (5, 264, torch.float16), (9, 2056, torch.bfloat16), (33, 4, torch.float32),
                                             (7, 1000, torch.float32)])
def test_gates(rows, cols, dtype):
    from fairseq_apollo_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(cols)
    wide = torch.randn(rows, 3 * cols, generator=gen, device="cuda").to(dtype)   # (operands are column slices)
    a, u, h = wide[:, :cols], wide[:, cols:2 * cols], wide[:, 2 * cols:]
    b = torch.randn(rows, cols, generator=gen, device="cuda").to(dtype)
    fa, fu, fh, fb = (t.float() for t in (a, u, h, b))
    limit = {torch.float32: 1e-6, torch.bfloat16: 2.0 ** -8 + 2.0 ** -11, torch.float16: 2.0 ** -10}[dtype]
    silu = torch.nn.functional.silu
    assert rel_l2(ops.gate_silu(a).float(), silu(fa)) < limit
    assert rel_l2(ops.gate_mul_silu(b, u).float(), fb * silu(fu)) < limit
    assert rel_l2(ops.gate_output(b, u, h, b).float(), torch.lerp(fb, silu(fh + fb), torch.sigmoid(fu))) < limit


@pytest.mark.parametrize("cols,dtype", [(64, torch.bfloat16), (128, torch.float16), (256, torch.bfloat16), (96, torch.bfloat16), (64, torch.float32)])
@pytest.mark.parametrize("bsz,period,pitch", [(1, 1, 1), (3, 13, 16), (2, 40, 40)])
def test_query_key_rotary_cache(bsz, period, pitch, cols, dtype):
    from fairseq_apollo_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(cols)
    z = torch.randn(bsz * period, 2 * cols, generator=gen, device="cuda").to(dtype)[:, :cols]
    gamma, beta = torch.randn(2, cols, generator=gen, device="cuda"), torch.randn(2, cols, generator=gen, device="cuda")
    ang = torch.rand(period, cols // 2, generator=gen, device="cuda") * 6
    rot = torch.stack((ang.cos(), ang.sin()), -1).contiguous()
    q, k = (torch.full((bsz, pitch, cols), 7.0, device="cuda", dtype=dtype) for _ in range(2))
    raw = torch.empty(bsz * period, cols, device="cuda", dtype=dtype)
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.lib().mega_gate_qk_rotary_cache(z.data_ptr(), z.stride(0), gamma.data_ptr(), beta.data_ptr(), rot.data_ptr(), period,
                                                    period, 0, pitch, q.data_ptr(), cols, k.data_ptr(), cols, raw.data_ptr(),
                                                    ops._dt(z), bsz * period, cols, 1e-5, stream), "gate_qk_rotary")
    zn = torch.nn.functional.normalize(z.float(), dim=-1, eps=1e-5)
    aff = zn.unsqueeze(1) * (gamma + 1.0) + beta
    turned = torch.view_as_real(torch.view_as_complex(aff.view(bsz, period, 2, -1, 2)) * torch.view_as_complex(rot).unsqueeze(1)).flatten(-2)
    limit = {torch.float32: 1e-6, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    assert rel_l2(q[:, :period].float(), turned[:, :, 0]) < limit and rel_l2(k[:, :period].float(), turned[:, :, 1]) < limit
    assert rel_l2(raw.float(), aff[:, 1]) < limit
    assert (q[:, period:] == 7).all() and (k[:, period:] == 7).all()   # the rows between are left alone


@pytest.mark.parametrize("inner,dtype", [(8, torch.bfloat16), (264, torch.bfloat16), (1024, torch.float16), (2048, torch.bfloat16),
                                         (2056, torch.bfloat16), (4, torch.float32), (516, torch.float32), (1028, torch.float32)])
@pytest.mark.parametrize("causal", [True, False])
def test_softmax_rows(inner, dtype, causal):
    from fairseq_apollo_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(inner)
    x = (torch.randn(2, min(inner, 70), inner, generator=gen, device="cuda") * 3).to(dtype)
    dy = torch.randn(x.shape, generator=gen, device="cuda").to(dtype)
    s = x.float()
    if causal:
        off = inner - x.size(1)
        s = s.masked_fill(torch.ones(x.size(1), inner, device="cuda", dtype=torch.bool).triu(off + 1), float('-inf'))
    want = torch.softmax(s, -1)
    y = ops.attention_softmax_fwd(x, causal)
    limit = {torch.float32: 1e-6, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    assert rel_l2(y.float(), want) < limit
    dx = ops.attention_softmax_bwd(dy, y, causal)
    w = y.float()
    assert rel_l2(dx.float(), w * (dy.float() - (w * dy.float()).sum(-1, keepdim=True))) < 2 * limit
