"""The causal EMA as matrix products of chunks (csrc/chunk_ema.cu), forward and backward, against the recurrence in float64: at
the edges of its chunks (16), steps (32), tiles (64, 128), segments and blocks of channels (8, 16)."""
import pytest
import torch

from _util import rel_l2

pytestmark = pytest.mark.gpu

# y and dx: one rounding of the result (2^-8 or 2^-11 of a value at most, 1.7e-3 or 2.1e-4 in the 2-norm of many, so 2^-9 and 2^-12
# beyond 1000 of them; leading parts alone are 3.3e-3 off in bf16 and would not pass); fp32: products of three bf16 parts leave 2^-24 of each term of sums of some forty (taps, poles, omega x), 2e-7 in the 2-norm for poles
# that forget within the 512 positions between the corrections of q^16 (test_slow_poles: the others).  States: as fp32.  Sums over
# B L positions: 2^-24 times the square root of the additions of a channel (under 64), in sums that cancel to a tenth
LIMIT = {torch.float32: 5e-7, torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -12}
SUMS = 5e-6


def limit_of(dtype, values):
    return LIMIT[dtype] * (2 if dtype != torch.float32 and values.numel() < 1000 else 1)


@pytest.fixture
def forced():
    from fairseq_apollo_b200 import _lib
    _lib.set_option(6, 2)
    yield _lib
    _lib.set_option(6, 0)
    _lib.set_option(7, 0)


def problem(gen, bsz, length, dim, ndim, dtype, cplx):
    p = torch.rand(dim, ndim, generator=gen) * 0.9 + 0.05
    mag = 1 - p * torch.sigmoid(torch.randn(dim, ndim, generator=gen))
    g = torch.randn(dim, ndim, generator=gen) * 0.25
    if cplx:
        mag = torch.polar(mag, torch.rand(dim, ndim, generator=gen) * 6.28)
        g = torch.complex(g, torch.randn(dim, ndim, generator=gen) * 0.25)
    omega = torch.randn(dim, generator=gen)
    x, dy = ((torch.randn(bsz, length, dim, generator=gen) + 0.1).to(dtype) for _ in range(2))
    return x, dy, p, mag, g, omega


def recurrence(x, p, q, g, omega, h=None):
    """(B, L, D) in double -> outputs, last state"""
    h = torch.zeros(x.size(0), *p.shape, dtype=q.dtype) if h is None else h
    out = []
    for xt in x.unbind(1):
        h = q * h + p * xt.unsqueeze(-1)
        y = (g * h).sum(-1)
        out.append((y.real if y.is_complex() else y) + omega * xt)
    return torch.stack(out, 1), h


def double(t):
    return t.to(torch.complex128) if t.is_complex() else t.double()


SHAPES = [(1, 2, 8, 16), (2, 15, 16, 16), (1, 17, 24, 5), (3, 33, 8, 16), (9, 64, 16, 1), (2, 65, 40, 16), (1, 127, 16, 16),
          (2, 129, 8, 16), (1, 700, 136, 16), (5, 321, 24, 7)]


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bsz,length,dim,ndim", SHAPES)
def test_against_float64(forced, bsz, length, dim, ndim, dtype, cplx):
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(length)
    x, dy, p, q, g, omega = problem(gen, bsz, length, dim, ndim, dtype, cplx)
    leaves = [double(t).requires_grad_(True) for t in (x, p, q, g, omega)]
    want, _ = recurrence(*leaves)
    want.backward(dy.double())
    fwd, bwd = (ops.cema_forward, ops.cema_backward) if cplx else (ops.ema_forward, ops.ema_backward)
    c = [t.cuda() for t in (p, q, g, omega)]
    xc, dyc = x.cuda().transpose(1, 2), dy.cuda().transpose(1, 2)
    y = fwd(xc, *c)
    assert forced.last_kernel() == "chunk_ema"
    assert rel_l2(y.transpose(1, 2), want) < limit_of(dtype, x)
    got = bwd(dyc, xc, *c)
    assert forced.last_kernel() == "chunk_ema"
    assert rel_l2(got[0].transpose(1, 2), leaves[0].grad) < limit_of(dtype, x)
    for name, a, b in zip(("p", "q", "g", "omega"), got[1:5], leaves[1:]):
        b = b.grad
        if a.is_complex():
            a, b = torch.view_as_real(a.cpu()), torch.view_as_real(b)
        assert rel_l2(a, b) < SUMS, name
    # with a state, activated
    h = torch.randn(bsz, dim, ndim, dtype=q.dtype, generator=gen)
    wanted, last = recurrence(*[double(t) for t in (x, p, q, g, omega)], double(h))
    y, out = fwd(xc, *c, None, h.cuda(), True, silu=True)
    assert forced.last_kernel() == "chunk_ema"
    assert rel_l2(y.transpose(1, 2), torch.nn.functional.silu(wanted)) < limit_of(dtype, x)
    if cplx:
        out, last = torch.view_as_real(out.cpu()), torch.view_as_real(last)
    assert rel_l2(out, last) < 5e-7


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bsz,length,dim,ndim", [(2, 37, 16, 5), (3, 130, 24, 16), (9, 200, 16, 16), (2, 1500, 8, 16)])
def test_padded_positions(forced, bsz, length, dim, ndim, dtype, cplx):
    """Zero to the states whatever stands there, NaN included in omega x's own position; their input gradient is omega dy."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(length)
    x, dy, p, q, g, omega = problem(gen, bsz, length, dim, ndim, dtype, cplx)
    mask = torch.rand(bsz, length, generator=gen) < 0.2
    mask[-1, length // 2:] = True
    leaves = [double(t).requires_grad_(True) for t in (x, p, q, g, omega)]
    masked = leaves[0].masked_fill(mask.unsqueeze(-1), 0.)
    want = recurrence(masked, *leaves[1:4], torch.zeros(dim, dtype=torch.float64))[0] + leaves[4] * leaves[0]
    want.backward(dy.double())
    fwd, bwd = (ops.cema_forward, ops.cema_backward) if cplx else (ops.ema_forward, ops.ema_backward)
    c = [t.cuda() for t in (p, q, g, omega)]
    xc, dyc, mc = x.cuda().transpose(1, 2), dy.cuda().transpose(1, 2), mask.cuda()
    y, got = fwd(xc, *c, mc), bwd(dyc, xc, *c, mc)
    assert forced.last_kernel() == "chunk_ema"
    assert rel_l2(y.transpose(1, 2), want) < LIMIT[dtype] and rel_l2(got[0].transpose(1, 2), leaves[0].grad) < LIMIT[dtype]
    for a, b in zip(got[1:5], leaves[1:]):
        b = b.grad
        if a.is_complex():
            a, b = torch.view_as_real(a.cpu()), torch.view_as_real(b)
        assert rel_l2(a, b) < SUMS
    h = torch.randn(bsz, dim, ndim, dtype=q.dtype, generator=gen)
    _, last = recurrence(masked.detach(), *[t.detach() for t in leaves[1:]], double(h))
    out = fwd(xc, *c, mc, h.cuda(), True)[1]
    assert forced.last_kernel() == "chunk_ema"
    if cplx:
        out, last = torch.view_as_real(out.cpu()), torch.view_as_real(last)
    assert rel_l2(out, last) < 5e-7
    bad = xc.clone()
    bad[-1, :, length - 1] = float("nan")
    z = fwd(bad, *c, mc)
    assert torch.equal(z[..., :length - 1], y[..., :length - 1]) and z[-1, :, -1].isnan().all() and torch.equal(z[:-1], y[:-1])
    bad = dyc.clone()
    bad[-1, :, length - 1] = float("inf")
    dx = bwd(bad, xc, *c, mc)[0]
    there = mask[-1].nonzero().flatten()[:-1].cuda()
    assert torch.equal(dx[-1][:, there], got[0][-1][:, there]) and not torch.isfinite(dx[-1, :, -1]).any()
    assert torch.equal(dx[:-1], got[0][:-1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_many_segments_and_any_strides(forced, dtype):
    """Sequences cut into segments, the last one ragged; time-major memory and slices of wider rows."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(1)
    x, dy, p, q, g, omega = problem(gen, 2, 5000, 16, 16, dtype, False)
    c = [t.cuda() for t in (p, q, g, omega)]
    xc, dyc = x.cuda().transpose(1, 2), dy.cuda().transpose(1, 2)
    y, grads = ops.ema_forward(xc, *c), ops.ema_backward(dyc, xc, *c)
    assert forced.last_kernel() == "chunk_ema"
    xt = x.cuda().transpose(0, 1).contiguous().permute(1, 2, 0)
    wide = torch.full((2, 5000, 48), float("nan"), dtype=dtype, device="cuda")
    wide[..., 16:32] = dy.cuda()
    y2, grads2 = ops.ema_forward(xt, *c), ops.ema_backward(wide[..., 16:32].transpose(1, 2), xt, *c)
    assert torch.equal(y, y2) and torch.equal(grads[0], grads2[0])
    forced.set_option(6, 1)
    y3, grads3 = ops.ema_forward(xc.float(), *c), ops.ema_backward(dyc.float(), xc.float(), *c)
    assert rel_l2(y, y3) < LIMIT[dtype] and rel_l2(grads[0], grads3[0]) < LIMIT[dtype]
    for a, b in zip(grads2[1:5], grads3[1:5]):
        assert rel_l2(a, b) < SUMS


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("at", [0, 15, 16, 40, 99])
def test_nothing_before_a_non_finite_input(forced, value, dtype, at, cplx):
    """Outputs ahead of an infinity or a NaN are as without it, and not finite from there on; the input's gradient the other
    way round in time."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(at)
    x, dy, p, q, g, omega = problem(gen, 2, 100, 16, 16, dtype, cplx)
    fwd, bwd = (ops.cema_forward, ops.cema_backward) if cplx else (ops.ema_forward, ops.ema_backward)
    c = [t.cuda() for t in (p, q, g, omega)]
    xc, dyc = x.cuda().transpose(1, 2), dy.cuda().transpose(1, 2)
    clean, grad = fwd(xc, *c), bwd(dyc, xc, *c)[0]
    bad, bad_dy = xc.clone(), dyc.clone()
    bad[1, 3, at] = value
    bad_dy[1, 3, at] = value
    y, dx = fwd(bad, *c), bwd(bad_dy, xc, *c)[0]
    assert forced.last_kernel() == "chunk_ema"
    assert torch.equal(y[1, 3, :at], clean[1, 3, :at]) and not torch.isfinite(y[1, 3, at:]).any()
    assert torch.equal(dx[1, 3, at + 1:], grad[1, 3, at + 1:]) and not torch.isfinite(dx[1, 3, :at + 1]).any()
    keep = torch.ones(16, dtype=torch.bool)
    keep[3] = False
    assert torch.equal(y[:, keep], clean[:, keep]) and torch.equal(dx[:, keep], grad[:, keep])
    assert torch.equal(y[0], clean[0])


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("bsz,length,dim,ndim", SHAPES)
def test_leading_parts(forced, bsz, length, dim, ndim, cplx):
    """bf16 in leading parts alone: matrices, states and outputs are rounded once each (2^-9), which adds up to 2^-8."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(length)
    x, _, p, q, g, omega = problem(gen, bsz, length, dim, ndim, torch.bfloat16, cplx)
    want, _ = recurrence(*[double(t) for t in (x, p, q, g, omega)])
    fwd = ops.cema_forward if cplx else ops.ema_forward
    c = [t.cuda() for t in (p, q, g, omega)]
    forced.set_option(6, 3)
    y = fwd(x.cuda().transpose(1, 2), *c, silu=True)
    assert forced.last_kernel() == "chunk_ema"
    assert rel_l2(y.transpose(1, 2), torch.nn.functional.silu(want)) < 1.5 * 2.0 ** -8


@pytest.mark.parametrize("cplx", [False, True])
def test_chosen_calls_agree_with_the_scan(cplx):
    """A call that the estimate gives to the chunks, against the forms that walk position by position."""
    from fairseq_apollo_b200 import _lib, ops
    gen = torch.Generator().manual_seed(4)
    x, dy, p, q, g, omega = problem(gen, 4, 2048, 512, 16, torch.bfloat16, cplx)
    bwd = ops.cema_backward if cplx else ops.ema_backward
    c = [t.cuda() for t in (p, q, g, omega)]
    xc, dyc = x.cuda().transpose(1, 2), dy.cuda().transpose(1, 2)
    got = bwd(dyc, xc, *c)
    assert _lib.last_kernel() == "chunk_ema"
    _lib.set_option(6, 1)
    try:
        want = bwd(dyc, xc, *c)
        assert _lib.last_kernel() != "chunk_ema"
    finally:
        _lib.set_option(6, 0)
    assert rel_l2(got[0], want[0]) < 2.0 ** -8
    for a, b in zip(got[1:5], want[1:5]):
        if a.is_complex():
            a, b = torch.view_as_real(a), torch.view_as_real(b)
        assert rel_l2(a, b) < 1e-5   # (the scan's own error: 3e-6)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bsz,length,dim", [(1, 33, 8), (2, 200, 24), (3, 513, 40)])
@pytest.mark.parametrize("normed", [False, True])
def test_behind_timestep_norm(forced, bsz, length, dim, dtype, cplx, normed):
    """TimestepNorm -> EMA with states in and out: the products take the normalised activations in fp32, not as they are
    rounded for the second output."""
    from fairseq_apollo_b200 import ops
    from oracle import mega_oracle as O
    gen = torch.Generator().manual_seed(length)
    x, _, p, q, g, omega = problem(gen, bsz, length, dim, 16, dtype, cplx)
    if dtype == torch.bfloat16 and not cplx and not normed:
        pytest.skip("another form's call")
    pc = torch.full((bsz,), 3, dtype=torch.int64)
    pm, pv = torch.randn(bsz, dim, generator=gen) * 0.1, torch.rand(bsz, dim, generator=gen) + 0.5
    gamma, beta = torch.randn(dim, generator=gen) * 0.1 + 1, torch.randn(dim, generator=gen) * 0.1
    h = torch.randn(bsz, dim, 16, dtype=q.dtype, generator=gen)
    xn, cnt, mean, var = O.timestep_norm(x.double(), pc, pm.double(), pv.double(), gamma.double(), beta.double(), None,
                                         acc_dtype=torch.float64)[:4]
    want, last = recurrence(xn, *[double(t) for t in (p, q, g, omega)], double(h))
    c = [t.cuda() for t in (pc, pm, pv, gamma, beta)]
    got = ops.tsn_ema_forward(x.cuda(), *c, 1e-5, p.cuda(), q.cuda(), g.cuda(), omega.cuda(), None, h_in=h.cuda(), want_state=True,
                              want_normed=normed, complex_poles=cplx)
    assert forced.last_kernel() == "chunk_ema"
    limit = max(LIMIT[dtype], 4e-6)   # (the statistics: reciprocals and roots to 2^-22, sums of up to 513 deviations)
    assert rel_l2(got["y"], want) < limit
    if normed:
        assert rel_l2(got["xn"], xn) < limit
    out = got["h"]
    if cplx:
        out, last = torch.view_as_real(out.cpu()), torch.view_as_real(last)
    assert rel_l2(out, last) < 4e-6
    assert torch.equal(got["count"].cpu(), cnt) and rel_l2(got["mean"], mean) < 4e-6 and rel_l2(got["var"], var) < 4e-6


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("slow", [1e-3, 1e-4])
@pytest.mark.parametrize("steps", [0, 4096, 16384])
def test_slow_poles(forced, slow, cplx, steps):
    """Poles near the unit circle over many chunks: a power of a pole that is rounded alike in every chunk or segment would add up
    to 2^-25 / (1 - q^16), 6e-6 at 1e-4.  What is left is the rounding of each chunk's sum, of either sign: 2^-25 times the square
    root of the 1 / (32 slow) that a state holds, and 2^-25 for each of the 16 chunks, on average, between the corrections."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(2)
    forced.set_option(7, steps)
    bsz, length, dim, ndim = 2, 16384 - 5, 16, 4
    x, dy, p, _, g, omega = problem(gen, bsz, length, dim, ndim, torch.float32, cplx)
    q = 1 - slow * (torch.rand(dim, ndim, generator=gen) + 0.5)
    if cplx:
        q = torch.polar(q, torch.rand(dim, ndim, generator=gen) * 6.28)
    h = torch.randn(bsz, dim, ndim, dtype=q.dtype, generator=gen)
    args = [double(t) for t in (p, q, g, omega)]
    want, last = recurrence(x.double(), *args, double(h))
    dx = recurrence(dy.double().flip(1), *args)[0].flip(1)
    fwd, bwd = (ops.cema_forward, ops.cema_backward) if cplx else (ops.ema_forward, ops.ema_backward)
    c = [t.cuda() for t in (p, q, g, omega)]
    y, out = fwd(x.cuda().transpose(1, 2), *c, None, h.cuda(), True)
    assert forced.last_kernel() == "chunk_ema"
    grad = bwd(dy.cuda().transpose(1, 2), x.cuda().transpose(1, 2), *c)[0]
    assert forced.last_kernel() == "chunk_ema"
    if cplx:
        out, last = torch.view_as_real(out.cpu()), torch.view_as_real(last)
    limit = 2.0 ** -25 * ((1 / (32 * slow)) ** 0.5 + 16)
    assert rel_l2(out, last) < limit and rel_l2(y.transpose(1, 2), want) < limit and rel_l2(grad.transpose(1, 2), dx) < limit


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("state", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("at", [0, 15, 40, 70, 191])
def test_infinities_are_the_recurrences(forced, dtype, at, state, masked):
    """From an infinite input on, outputs and states are infinite where the recurrence's are (weights of one sign), not NaN, in
    later segments too and for poles that forget within a chunk; the input's gradient the other way round in time."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(at)
    bsz, length, dim, ndim = 2, 300, 16, 5
    x, dy, p, q, g, omega = problem(gen, bsz, length, dim, ndim, dtype, False)
    q[:, 0] = 1e-4
    g, omega = g.abs() + 0.1, omega.abs() + 0.1
    mask = None
    if masked:
        mask = torch.rand(bsz, length, generator=gen) < 0.2
        mask[1, at] = False
    c = [t.cuda() for t in (p, q, g, omega)]
    bad, bad_dy = x.clone(), dy.clone()
    bad[1, at, 3], bad_dy[1, at, 3] = float("inf"), float("-inf")
    mc = None if mask is None else mask.cuda()
    h = torch.randn(bsz, dim, ndim, generator=gen) if state else None
    out = ops.ema_forward(bad.cuda().transpose(1, 2), *c, mc, None if h is None else h.cuda(), state)
    assert forced.last_kernel() == "chunk_ema"
    keep = torch.ones(bsz, length, 1) if mask is None else (~mask).double().unsqueeze(-1)
    args = [t.double() for t in (p, q, g, omega)]
    want, last = recurrence(torch.where(keep > 0, bad.double(), 0.0), *args, None if h is None else h.double())
    want = want + omega.double() * torch.where(keep > 0, 0.0, x.double())
    y = (out[0] if state else out).transpose(1, 2).cpu().double()
    assert torch.equal(y.isinf(), want.isinf()) and not y.isnan().any() and y[1, at:, 3].isinf().all()
    fine = ~want.isinf()
    assert rel_l2(y[fine], want[fine]) < LIMIT[dtype]
    if state:
        assert torch.equal(out[1].isinf().cpu(), last.isinf()) and last[1, 3].isinf().all()
        fine = ~last.isinf()
        assert rel_l2(out[1].cpu()[fine], last[fine]) < 5e-7
        return
    got = ops.ema_backward(bad_dy.cuda().transpose(1, 2), x.cuda().transpose(1, 2), *c, mc)
    assert forced.last_kernel() == "chunk_ema"
    back = recurrence(bad_dy.double().flip(1), *args)[0].flip(1)
    want = torch.where(keep > 0, back, omega.double() * dy.double())
    dx = got[0].transpose(1, 2).cpu().double()
    assert torch.equal(dx.isinf(), want.isinf()) and not dx.isnan().any()
    fine = ~want.isinf()
    assert rel_l2(dx[fine], want[fine]) < LIMIT[dtype]
    assert not any(torch.isfinite(t[3]).any() for t in got[1:5])


@pytest.mark.parametrize("cplx", [False, True])
def test_values_that_bf16_takes_for_infinite(forced, cplx):
    """fp32 values above bf16's largest: finite, as the recurrence has them."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(3)
    x, dy, p, q, g, omega = problem(gen, 2, 300, 16, 5, torch.float32, cplx)
    g, omega = g * 0.1, omega.clamp(-0.4, 0.4)
    x[1, 37, 3], dy[0, 250, 5] = 3.4e38, -3.4e38
    args = [double(t) for t in (p, q, g, omega)]
    want, back = recurrence(x.double(), *args)[0], recurrence(dy.double().flip(1), *args)[0].flip(1)
    c = [t.cuda() for t in (p, q, g, omega)]
    fwd, bwd = (ops.cema_forward, ops.cema_backward) if cplx else (ops.ema_forward, ops.ema_backward)
    y = fwd(x.cuda().transpose(1, 2), *c).transpose(1, 2).cpu().double()
    dx = bwd(dy.cuda().transpose(1, 2), x.cuda().transpose(1, 2), *c)[0].transpose(1, 2).cpu().double()
    for a, b, row, ch in ((y, want, 1, 3), (dx, back, 0, 5)):
        assert torch.isfinite(a).all()
        there = torch.zeros_like(a, dtype=torch.bool)
        there[row, :, ch] = True
        assert rel_l2(a[there] * 2.0 ** -64, b[there] * 2.0 ** -64) < 5e-7 and rel_l2(a[~there], b[~there]) < 5e-7


# Long segments: from five tiles of 128 (or ten of 64) positions on, and a last one of a few positions or tiles
LONG = [(192, 2, 1000, 24, 16), (640, 3, 1283, 16, 16), (704, 1, 1500, 40, 5), (1536, 9, 1536 - 7, 16, 16), (1088, 2, 1089, 8, 16)]


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("steps,bsz,length,dim,ndim", LONG)
def test_many_tiles_of_a_segment(forced, steps, bsz, length, dim, ndim, dtype, cplx, masked):
    """Slots, buffers and padding bits used again from the third tile on, outputs that leave while the next tile arrives, a state
    exported from a late tile; forward with a state, and backward."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(length)
    x, dy, p, q, g, omega = problem(gen, bsz, length, dim, ndim, dtype, cplx)
    mask = None
    if masked:
        mask = torch.rand(bsz, length, generator=gen) < 0.15
        mask[-1, length - length // 3:] = True
    forced.set_option(7, steps)
    leaves = [double(t).requires_grad_(True) for t in (x, p, q, g, omega)]
    seen = leaves[0] if mask is None else leaves[0].masked_fill(mask.unsqueeze(-1), 0.)
    want = recurrence(seen, *leaves[1:4], torch.zeros(dim, dtype=torch.float64))[0] + leaves[4] * leaves[0]
    want.backward(dy.double())
    fwd, bwd = (ops.cema_forward, ops.cema_backward) if cplx else (ops.ema_forward, ops.ema_backward)
    c = [t.cuda() for t in (p, q, g, omega)]
    xc, dyc, mc = x.cuda().transpose(1, 2), dy.cuda().transpose(1, 2), None if mask is None else mask.cuda()
    y = fwd(xc, *c, mc)
    assert forced.last_kernel() == "chunk_ema"
    assert rel_l2(y.transpose(1, 2), want) < LIMIT[dtype]
    got = bwd(dyc, xc, *c, mc)
    assert forced.last_kernel() == "chunk_ema"
    assert rel_l2(got[0].transpose(1, 2), leaves[0].grad) < LIMIT[dtype]
    for a, b in zip(got[1:5], leaves[1:]):
        b = b.grad
        if a.is_complex():
            a, b = torch.view_as_real(a.cpu()), torch.view_as_real(b)
        assert rel_l2(a, b) < SUMS
    h = torch.randn(bsz, dim, ndim, dtype=q.dtype, generator=gen)
    extra, last = recurrence(torch.zeros_like(seen), *[t.detach() for t in leaves[1:]], double(h))
    _, own = recurrence(seen.detach(), *[t.detach() for t in leaves[1:]])
    y, out = fwd(xc, *c, mc, h.cuda(), True)
    assert forced.last_kernel() == "chunk_ema"
    assert rel_l2(y.transpose(1, 2), want.detach() + extra) < LIMIT[dtype]
    out, last = out.cpu(), last + own
    if cplx:
        out, last = torch.view_as_real(out), torch.view_as_real(last)
    assert rel_l2(out, last) < (1e-6 if masked else 5e-7)   # (a state that only decays: 2^-25 for each of 32 chunks)


@pytest.mark.parametrize("cplx", [False, True])
def test_many_tiles_in_leading_parts(forced, cplx):
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(8)
    x, _, p, q, g, omega = problem(gen, 3, 1500, 24, 16, torch.bfloat16, cplx)
    want, _ = recurrence(*[double(t) for t in (x, p, q, g, omega)])
    c = [t.cuda() for t in (p, q, g, omega)]
    forced.set_option(6, 3)
    forced.set_option(7, 704)
    y = (ops.cema_forward if cplx else ops.ema_forward)(x.cuda().transpose(1, 2), *c)
    assert forced.last_kernel() == "chunk_ema"
    assert rel_l2(y.transpose(1, 2), want) < 1.5 * 2.0 ** -8


def _normed_problem(gen, bsz, length, dim, mask):
    from oracle import mega_oracle as O
    pc = torch.full((bsz,), 3, dtype=torch.int64)
    pm, pv = torch.randn(bsz, dim, generator=gen) * 0.1, torch.rand(bsz, dim, generator=gen) + 0.5
    gamma, beta = torch.randn(dim, generator=gen) * 0.1 + 1, torch.randn(dim, generator=gen) * 0.1
    norm = lambda x: O.timestep_norm(x.double(), pc, pm.double(), pv.double(), gamma.double(), beta.double(), mask,
                                     acc_dtype=torch.float64)
    return [t.cuda() for t in (pc, pm, pv, gamma, beta)], norm


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("normed", [False, True])
@pytest.mark.parametrize("masked", [False, True])
def test_many_tiles_behind_timestep_norm(forced, dtype, cplx, normed, masked):
    """TimestepNorm with padding in the middle and at the end, which the products then know nothing of; long segments from fp32
    scratch memory into each type."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(17)
    bsz, length, dim = 3, 1283, 40
    x, _, p, q, g, omega = problem(gen, bsz, length, dim, 16, dtype, cplx)
    mask = None
    if masked:
        mask = torch.rand(bsz, length, generator=gen) < 0.1
        mask[-1, length - length // 4:] = True
    if dtype == torch.bfloat16 and not cplx and not normed and not masked:
        pytest.skip("another form's call")
    stats, norm = _normed_problem(gen, bsz, length, dim, mask)
    xn, cnt, mean, var = norm(x)[:4]
    want, last = recurrence(xn, *[double(t) for t in (p, q, g, omega)])
    forced.set_option(7, 704)
    got = ops.tsn_ema_forward(x.cuda(), *stats, 1e-5, *[t.cuda() for t in (p, q, g, omega)], None if mask is None else mask.cuda(),
                              want_state=not masked, want_normed=normed, complex_poles=cplx)
    assert forced.last_kernel() == "chunk_ema"
    limit = max(LIMIT[dtype], 4e-6)   # (the statistics: reciprocals and roots to 2^-22, sums of up to 1283 deviations)
    assert rel_l2(got["y"], want) < limit
    if normed:
        assert rel_l2(got["xn"], xn) < limit
    if not masked:
        out = got["h"].cpu()
        if cplx:
            out, last = torch.view_as_real(out), torch.view_as_real(last)
        assert rel_l2(out, last) < 4e-6
    assert torch.equal(got["count"].cpu(), cnt) and rel_l2(got["mean"], mean) < 4e-6 and rel_l2(got["var"], var) < 4e-6


def test_leading_parts_behind_timestep_norm():
    """A bf16 call without a state that would run on the tensor cores: TimestepNorm in bf16, then the leading parts.  Its roundings:
    the normalised activations (2^-9), matrices, states and outputs."""
    from fairseq_apollo_b200 import _lib, ops
    gen = torch.Generator().manual_seed(21)
    bsz, length, dim = 22, 129, 1176
    x, _, p, q, g, omega = problem(gen, bsz, length, dim, 16, torch.bfloat16, True)
    stats, norm = _normed_problem(gen, bsz, length, dim, None)
    xn = norm(x)[0]
    want, _ = recurrence(xn, *[double(t) for t in (p, q, g, omega)])
    got = ops.tsn_ema_forward(x.cuda(), *stats, 1e-5, *[t.cuda() for t in (p, q, g, omega)], None, want_normed=True, complex_poles=True)
    assert _lib.last_kernel() == "chunk_ema"
    assert rel_l2(got["y"], want) < 2 * 2.0 ** -8 and rel_l2(got["xn"], xn) < 2.0 ** -9


@pytest.mark.parametrize("steps", [64, 1024])
def test_complex_poles_over_many_segments(forced, steps):
    """No mask, sequences cut into up to 47 segments, time-major memory: against the forms that walk position by position."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator().manual_seed(1)
    x, dy, p, q, g, omega = problem(gen, 2, 3000, 16, 16, torch.float32, True)
    forced.set_option(7, steps)
    c = [t.cuda() for t in (p, q, g, omega)]
    xt, dyc = x.cuda().transpose(0, 1).contiguous().permute(1, 2, 0), dy.cuda().transpose(1, 2)
    y, grads = ops.cema_forward(xt, *c), ops.cema_backward(dyc, xt, *c)
    assert forced.last_kernel() == "chunk_ema"
    leaves = [double(t).requires_grad_(True) for t in (x, p, q, g, omega)]
    want, _ = recurrence(*leaves)
    want.backward(dy.double())
    assert rel_l2(y.transpose(1, 2), want) < LIMIT[torch.float32] and rel_l2(grads[0].transpose(1, 2), leaves[0].grad) < LIMIT[torch.float32]
    for a, b in zip(grads[1:5], leaves[1:]):
        b = b.grad
        if a.is_complex():
            a, b = torch.view_as_real(a.cpu()), torch.view_as_real(b)
        assert rel_l2(a, b) < SUMS
