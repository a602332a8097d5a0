"""The native host side: what it refuses, the precision of parameters of several types, autograd around its Functions."""
import copy

import pytest
import torch

from _util import make_ema_params, rel_l2

pytestmark = pytest.mark.gpu


def _cuda(*ts):
    return [t.cuda() for t in ts]


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("wrong", ["rows", "bidirectional", "delta", "third", "gamma", "omega", "device"])
def test_training_ema_checks_its_parameters(cplx, wrong):
    from fairseq_apollo_b200 import functions
    gen = torch.Generator().manual_seed(0)
    dim, n = 16, 16
    prm = make_ema_params(gen, dim, n, device="cuda")
    if cplx:
        prm[2], prm[3] = torch.randn(dim, 1, 1).cuda(), torch.randn(dim, n, 2).cuda()
    x = torch.randn(2, 8, dim, device="cuda", requires_grad=True)
    bidir, error = False, ValueError
    if wrong == "rows":
        x = torch.randn(2, 8, dim + 8, device="cuda", requires_grad=True)
    elif wrong == "bidirectional":
        bidir = True
    elif wrong == "device":
        prm[1], error = prm[1].cpu(), RuntimeError
    else:
        at = {"delta": 1, "third": 2, "gamma": 3, "omega": 4}[wrong]
        prm[at] = prm[at][: dim // 2].contiguous()
    with pytest.raises(error):
        functions.ema(x, *prm, None, bidir, True, None, cplx, False, True)


@pytest.mark.parametrize("wrong", ["bias", "prior", "logv", "features", "device"])
def test_training_norms_checks_their_parameters(wrong):
    from fairseq_apollo_b200 import functions
    x = torch.randn(2, 8, 16, device="cuda", requires_grad=True)
    w, b, m, v = (torch.randn(16, device="cuda") for _ in range(4))
    count, error = torch.tensor(2, device="cuda"), ValueError
    if wrong == "bias":
        b = b[:8].contiguous()
    elif wrong == "prior":
        m, v = m[:8].contiguous(), v[:8].contiguous()
    elif wrong == "logv":
        v = v[:8].contiguous()
    elif wrong == "features":
        w, b = w[:8].contiguous(), b[:8].contiguous()
    else:
        b, error = b.cpu(), RuntimeError
    with pytest.raises(error):
        functions.timestep_norm(x, count, m, v, w, b, None, None, 1e-5)
    if wrong in ("bias", "features", "device"):
        with pytest.raises(error):
            functions.sequence_norm(x, w, b, None, 1e-5, False)


def test_fused_operators_checks_their_operands():
    from fairseq_apollo_b200 import ops
    x = torch.randn(2, 600, 16, device="cuda")
    c = torch.full((2,), 2, device="cuda")
    m, v = torch.zeros(2, 16, device="cuda"), torch.ones(2, 16, device="cuda")
    one = torch.ones(16, device="cuda")
    co = [torch.rand(16, 4, device="cuda") for _ in range(3)]
    ops.tsn_ema_forward(x, c, m, v, one, one, 1e-5, *co, one)
    bad = [dict(m=m[:1]), dict(v=v[:, :8]), dict(c=c[:1]), dict(ga=one[:8]), dict(be=one[:8]), dict(om=one[:8]),
           dict(co=[t[:8] for t in co]), dict(co=[co[0], co[1][:8], co[2]]), dict(h=torch.zeros(2, 8, 4, device="cuda"))]
    for b in bad:
        with pytest.raises(ValueError):
            ops.tsn_ema_forward(x, b.get("c", c), b.get("m", m), b.get("v", v), b.get("ga", one), b.get("be", one), 1e-5,
                                *b.get("co", co), b.get("om", one), None, b.get("h"), True)
    xt = x.transpose(1, 2).contiguous()
    for ga, om, k in ((one[:8], one, co), (one, one[:8], co), (one, one, [t[:8] for t in co])):
        with pytest.raises(ValueError):
            ops.sqn_ema_forward(xt, ga, one, 1e-5, *k, om)
    for ga, be in ((one[:8], one), (one, one[:8])):
        with pytest.raises(ValueError):
            ops.timestep_norm_fwd(x, c, m, v, ga, be)
        with pytest.raises(ValueError):
            ops.sequence_norm_fwd(x, ga, be, length_last=False)
    with pytest.raises(ValueError):
        ops.ema_forward(xt, *co, one[:8])


def test_real_coefficients_of_the_complex_layer():
    """q, gamma and the state given as real tensors are complex ones without an imaginary part."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(0)
    x = torch.randn(2, 16, 50, generator=gen).cuda()
    p, q, g = (torch.rand(16, 4, generator=gen).cuda() for _ in range(3))
    om, h = torch.randn(16, generator=gen).cuda(), torch.randn(2, 16, 4, generator=gen).cuda()
    y, hn = ops.cema_forward(x, p, q, g, om, None, h, want_state=True)
    want, hw = ops.ema_forward(x, p, q, g, om, None, h, want_state=True)
    assert rel_l2(y, want) < 1e-5 and rel_l2(hn.real, hw) < 1e-5


@pytest.mark.parametrize("wide", [torch.float32, torch.float64])
def test_parameters_of_several_types(wide):
    """bf16 scale and shift beside wider priors (and the other way round): no value passes through the narrower type."""
    import fairseq_apollo_b200 as M
    torch.manual_seed(3)
    norm = M.TimestepNorm(64, prior_count=4).cuda()
    with torch.no_grad():
        for p in norm.parameters():
            p.normal_(0, 0.3)
    x, dy = torch.randn(2, 100, 64, device="cuda"), torch.randn(2, 100, 64, device="cuda")
    for narrow in (("weight", "bias"), ("prior_mean", "prior_logv"), ("bias",), ("weight", "prior_logv"), ()):
        mixed, ref = copy.deepcopy(norm), copy.deepcopy(norm)
        for name, p in mixed.named_parameters():
            p.data = p.data.to(torch.bfloat16 if name in narrow else wide)
        for (name, p), q in zip(mixed.named_parameters(), ref.parameters()):
            q.data = p.data.float()
        out = []
        for m in (mixed, ref):
            xx = x.clone().requires_grad_(True)
            y = m(xx)
            y.backward(dy)
            out.append([y, xx.grad] + [p.grad for p in m.parameters()])
            with torch.no_grad():
                out[-1].append(m(x))
        for a, b in zip(*out):
            assert rel_l2(a, b.to(a.dtype)) < 1e-6
        for p in mixed.parameters():
            assert p.grad.dtype == p.dtype


def test_ema_parameters_of_several_types():
    import fairseq_apollo_b200 as M
    torch.manual_seed(4)
    x, dy = torch.randn(2, 32, 200, device="cuda"), torch.randn(2, 32, 200, device="cuda")
    for names in (("alpha",), ("omega",), ("gamma", "beta")):
        mixed = M.MultiHeadEMA(32, ndim=16).cuda()
        ref = copy.deepcopy(mixed)
        for name, p in mixed.named_parameters():
            if name in names:
                p.data = p.data.bfloat16()
        for p, q in zip(mixed.parameters(), ref.parameters()):
            q.data = p.data.float()
        if "alpha" in names:    # (the coefficients are made in alpha's type)
            for q in (ref.delta, ref.beta, ref.gamma):
                q.data = q.data.bfloat16().float()
        for m in (mixed, ref):
            m(x).backward(dy)
        for (name, p), q in zip(mixed.named_parameters(), ref.named_parameters()):
            assert rel_l2(p.grad.float(), q[1].grad) < (1e-2 if p.dtype == torch.bfloat16 or "alpha" in names else 1e-5), name


def test_block_with_fp32_affine_in_a_16_bit_block():
    """The query / key affine kept in fp32: its gradients are not rounded to the projections' type."""
    import fairseq_apollo_b200 as M
    torch.manual_seed(6)
    blk = M.MovingAverageGatedAttention(64, 64, 128, 16, efficient_attn=True, rel_pos_bias='rotary', chunk_size=32,
                                        moving_act='silu').cuda().bfloat16()
    for name in ("gamma", "beta"):
        p = getattr(blk, name)
        p.data = torch.randn_like(p.data, dtype=torch.float32) * 0.3
    x = torch.randn(2, 64, 64, device="cuda").bfloat16().requires_grad_(True)
    blk(x)[0].sum().backward()
    for p in (blk.gamma, blk.beta):
        assert p.grad.dtype == torch.float32
        assert (p.grad != p.grad.bfloat16().float()).float().mean() > 0.5


@pytest.mark.parametrize("silu", [None, "silu"])
def test_result_may_be_changed_in_place(silu):
    import fairseq_apollo_b200 as M
    torch.manual_seed(8)
    norm, move = M.TimestepNorm(64, prior_count=2).cuda(), M.MultiHeadEMA(64, ndim=16).cuda()
    x = torch.randn(2, 40, 64, device="cuda", requires_grad=True)
    grads = []
    for inplace in (False, True):
        x.grad = None
        y = M.timestep_norm_ema(norm, move, x, None, None, silu)
        y = y.mul_(2.0) if inplace else y * 2.0
        y.sum().backward()
        grads.append(x.grad.clone())
    assert torch.equal(*grads)


def test_more_sequences_than_a_grid_axis():
    """65537 sequences: the backward that takes the statistics again has no grid for them; the saved ones do."""
    import fairseq_apollo_b200 as M
    torch.manual_seed(9)
    bsz = 65537
    norm = M.TimestepNorm(8, prior_count=2).cuda()
    x = torch.randn(bsz, 2, 8, device="cuda")
    dy = torch.randn_like(x)
    xx = x.clone().requires_grad_(True)
    norm(xx).backward(dy)
    w, dx = norm.weight.grad.clone(), []
    norm.zero_grad()
    for part in (slice(0, 40000), slice(40000, bsz)):
        xp = x[part].clone().requires_grad_(True)
        norm(xp).backward(dy[part])
        dx.append(xp.grad)
    assert rel_l2(xx.grad, torch.cat(dx)) < 1e-5
    assert rel_l2(w, norm.weight.grad) < 1e-4


def test_backward_without_the_form_over_time():
    """The form that takes the statistics again refuses (no scratch memory; here: switched off between the passes)."""
    import fairseq_apollo_b200 as M
    from fairseq_apollo_b200 import _lib
    torch.manual_seed(9)
    norm = M.TimestepNorm(64, prior_count=2).cuda()
    x, dy, grads = torch.randn(3, 200, 64, device="cuda"), torch.randn(3, 200, 64, device="cuda"), []
    mask = torch.zeros(3, 200, dtype=torch.bool, device="cuda")
    mask[1, 100:] = True
    for off in (0, 1):
        norm.zero_grad()
        xx = x.clone().requires_grad_(True)
        y = norm(xx, mask)
        _lib.set_option(0, off)
        try:
            y.backward(dy)
        finally:
            _lib.set_option(0, 0)
        grads.append([xx.grad] + [p.grad.clone() for p in norm.parameters()])
    for a, b in zip(*grads):
        assert rel_l2(a, b) < 1e-5


@pytest.mark.parametrize("bidir", [False, True])
def test_second_derivative_through_the_block(bidir):
    """A gradient penalty on the projections' inputs: as the block's own sequence of operations gives it."""
    import fairseq_apollo_b200 as M
    from fairseq_apollo_b200 import block_function
    torch.manual_seed(10)
    kw = dict(bidirectional=True, rel_pos_bias='simple', max_positions=32) if bidir else \
        dict(efficient_attn=True, rel_pos_bias='rotary')
    blk = M.MovingAverageGatedAttention(32, 64, 64, 16, chunk_size=-1 if bidir else 16, moving_act='silu', **kw).cuda()
    with torch.no_grad():
        for lin in (blk.v_proj, blk.mx_proj, blk.h_proj):
            lin.weight.normal_(0, 0.2)
    x = torch.randn(2, 32, 32, device="cuda")
    res = []
    mode_of = block_function.mode_of
    for own in (False, True):
        block_function.mode_of = (lambda *a: None) if own else mode_of
        try:
            xx = x.clone().requires_grad_(True)
            y = blk(xx)[0]
            g, = torch.autograd.grad(y.square().sum(), xx, create_graph=True)
            blk.zero_grad()
            g.square().sum().backward()
        finally:
            block_function.mode_of = mode_of
        res.append([g.detach()] + [p.grad.clone() for p in blk.parameters() if p.grad is not None])
    assert len(res[0]) == len(res[1])
    for a, b in zip(*res):
        assert rel_l2(a, b) < 1e-4


@pytest.mark.parametrize("rows", [1, 5, 9, 63, 65])
@pytest.mark.parametrize("zdim", [64, 128, 256])
def test_query_key_rows_that_end_inside_a_warp(rows, zdim):
    """16 bytes per access against the same rows an element off, which take one value per access."""
    from fairseq_apollo_b200 import ops
    torch.manual_seed(rows)
    buf = torch.randn(rows * zdim + 8, device="cuda").bfloat16()
    g, b = torch.randn(2, zdim, device="cuda"), torch.randn(2, zdim, device="cuda")
    rot = torch.polar(torch.ones(7, zdim // 2), torch.rand(7, zdim // 2)).cuda()
    one = buf[1:1 + rows * zdim].view(rows, zdim)
    for a, c in zip(ops.gate_qk_rotary(one.clone(), g, b, rot, 7), ops.gate_qk_rotary(one, g, b, rot, 7)):
        assert rel_l2(a, c) < 2.0 ** -9


def test_bidirectional_block_beyond_a_grid_axis():
    """65536 sequences: more than the relative-bias softmax takes in a launch."""
    import fairseq_apollo_b200 as M
    torch.manual_seed(13)
    blk = M.MovingAverageGatedAttention(8, 8, 16, 4, bidirectional=True, rel_pos_bias='simple', max_positions=4, moving_act='silu').cuda()
    x = torch.randn(65536, 4, 8, device="cuda")
    dx, dw = [], []
    for parts in ((x,), x.split(40000)):
        blk.zero_grad()
        got = []
        for p in parts:
            p = p.clone().requires_grad_(True)
            blk(p)[0].square().sum().backward()
            got.append(p.grad)
        dx.append(torch.cat(got))
        dw.append(blk.h_proj.weight.grad.clone())
    assert rel_l2(*dx) < 1e-5 and rel_l2(*dw) < 1e-4


def test_saved_tensors_of_a_training_pass():
    """What hooks on saved tensors see (offloading, compression): every activation once per Function that needs it."""
    import fairseq_apollo_b200 as M
    from collections import Counter
    torch.manual_seed(14)
    blk = M.MovingAverageGatedAttention(64, 64, 128, 16, efficient_attn=True, rel_pos_bias='rotary', chunk_size=32,
                                        moving_act='silu').cuda().bfloat16()
    x = torch.randn(2, 64, 64, device="cuda").bfloat16()
    grads = []
    for hooks in (False, True):
        blk.zero_grad()
        xx, seen = x.clone().requires_grad_(True), Counter()

        def pack(t):
            if t.numel() >= x.numel():
                seen[t.data_ptr()] += 1
            return t.cpu() if hooks else t
        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
            y = blk(xx)[0]
        y.sum().backward()
        assert max(seen.values()) <= 2      # (the block's input and the norm's output: a Function on either side)
        grads.append([xx.grad] + [p.grad.clone() for p in blk.parameters() if p.grad is not None])
    for a, b in zip(*grads):
        assert rel_l2(a, b) < 1e-2
