"""The EMA layer in one launch at the edges of its split: segments of at least 16 steps (multiples of 8), eight per block,
one to eight blocks of a cluster, 32 channels each; short last segments, empty segments and blocks.

Reference: the float64 oracle.  fp32: a state is a sum of at most L terms with powers rounded once per segment and block;
5e-6 relative 2-norm.  16-bit outputs are rounded by at most 2^-8 (bf16, 8
significant bits) and 2^-11 (fp16) of their values; normalised activations are not rounded on the way."""
import pytest
import torch

from _util import make_ema_params, rel_l2

pytestmark = pytest.mark.gpu
LIMIT = {torch.float32: 5e-6, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _mask(bsz, length):
    mask = torch.zeros(bsz, length, dtype=torch.bool)
    mask[0, 1:min(length, 40) - 1:3] = True
    mask[-1, length - length // 2:] = True
    return mask


@pytest.mark.parametrize("length,bsz,dim,dtype,ndim", [
    (2, 1, 8, torch.float32, 16),        # one short segment
    (127, 2, 40, torch.bfloat16, 16),    # channels beyond a strip
    (129, 3, 32, torch.float32, 5),      # a second block with one step; inert poles
    (333, 5, 40, torch.float32, 16),     # a short block, then an empty one
    (1000, 1, 64, torch.float16, 16),
    (4104, 2, 72, torch.float32, 16),    # eight blocks, segments of 72
])
@pytest.mark.parametrize("form", ["plain", "mask", "state", "bidir", "complex", "norm", "norm_state", "norm_complex"])
def test_scan_cluster(length, bsz, dim, dtype, ndim, form):
    from fairseq_apollo_b200 import _lib, ops
    from oracle import mega_oracle as O
    gen = torch.Generator().manual_seed(length)
    x = (torch.randn(bsz, length, dim, generator=gen) * 1.1 + 0.2).to(dtype)
    bidir, cplx, norm, state = form == "bidir", "complex" in form, "norm" in form, "state" in form
    mask = _mask(bsz, length) if form in ("mask", "bidir", "norm_state", "norm_complex") else None
    prm = make_ema_params(gen, dim, ndim, bidirectional=bidir)
    h = None
    if cplx:
        prm[2] = torch.randn(dim, 1, 1, generator=gen)
        prm[3] = torch.randn(dim, ndim, 2, generator=gen)
        p, q, g = O.cema_coeffs(*prm[:4])
        fwd = O.cema_forward_recurrence
    else:
        p, q, g = O.ema_coeffs(*prm[:4])
        fwd = O.ema_forward_recurrence
    if state:
        h = torch.randn(bsz, dim, ndim, generator=gen) * 0.3
    dev = [None if t is None else t.cuda() for t in (p.reshape(p.shape[0], -1), q.reshape(q.shape[0], -1), g, prm[4], mask, h)]
    xg, ref, res = x.cuda(), x.double(), {}
    _lib.set_option(1, 1)   # (without the tensor-core kernel bf16 takes the same way as fp32)
    _lib.set_option(5, 0)
    try:
        if norm:
            pc, pm, pv = torch.full((bsz,), 3), torch.randn(bsz, dim, generator=gen) * 0.1, torch.rand(bsz, dim, generator=gen) + 0.5
            gamma, beta = torch.rand(dim, generator=gen) + 0.5, torch.randn(dim, generator=gen)
            _lib.set_option(1, 0)
            _lib.set_option(5, 3)
            res = ops.tsn_ema_forward(xg, pc.cuda(), pm.cuda(), pv.cuda(), gamma.cuda(), beta.cuda(), 1e-5, *dev[:4], dev[4], dev[5],
                                      state, False, True, cplx)
            y, ho = res["y"], res.get("h")
            ref, cnt, mean, var = O.timestep_norm(ref, pc, pm.double(), pv.double(), gamma.double(), beta.double(), mask,
                                                  acc_dtype=torch.float64)[:4]
            assert torch.equal(res["count"].cpu(), cnt)
            assert rel_l2(res["mean"], mean) < 5e-6 and rel_l2(res["var"], var) < 5e-6
            assert rel_l2(res["xn"], ref) < LIMIT[dtype]
        else:
            fn = ops.cema_forward if cplx else ops.ema_forward
            out = fn(xg.transpose(1, 2), *dev[:4], dev[4], dev[5], want_state=state, bidirectional=bidir)
            (y, ho) = out if state else (out, None)
            y = y.transpose(1, 2)
        assert _lib.last_kernel() == "scan_cluster"
    finally:
        _lib.set_option(1, 0)
        _lib.set_option(5, 0)
    kw = {"bidirectional": True} if bidir else {}
    want = fwd(ref.double().transpose(1, 2), *[t.double() for t in prm], mask, h=h, return_state=state, **kw)
    want, hw = want if state else (want, None)
    assert rel_l2(y, want.transpose(1, 2)) < LIMIT[dtype]
    if state:
        assert rel_l2(ho, hw) < (1e-5 if dtype == torch.float32 or norm else 5e-6)
