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
    for key in (1, 2, 5, 6):
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


def _norm_call(form, gen, bsz, length, dim, count):
    """(run(mean_out, var_out) -> (y, count), prev_mean, prev_var, reference) of a TimestepNorm form of the C interface"""
    from fairseq_apollo_b200 import _lib, ops
    from oracle import mega_oracle as O
    groups = 4 if form == "group" else dim
    x = torch.randn(bsz, length, dim, generator=gen) * 1.1 + 0.2
    mask = torch.zeros(bsz, length, dtype=torch.bool)
    mask[0, 3:length - 4:5] = True
    mask[-1, length - length // 3:] = True
    pc = torch.full((bsz,), count)
    pm, pv = torch.randn(bsz, groups, generator=gen) * 0.3, torch.rand(bsz, groups, generator=gen) + 0.5
    gamma, beta = torch.rand(dim, generator=gen) + 0.5, torch.randn(dim, generator=gen)
    if groups == dim:
        want = O.timestep_norm(x.double(), pc, pm.double(), pv.double(), gamma.double(), beta.double(), mask, acc_dtype=torch.float64)
    else:
        want = O.group_timestep_norm(x.double(), pc, pm.double(), pv.double(), gamma.double(), beta.double(), mask, groups,
                                     acc_dtype=torch.float64)
    dev = [t.cuda() for t in (x, pc, pm, pv, gamma, beta, mask)]
    prm = [t.cuda() for t in (torch.rand(dim, 16, generator=gen) * 0.2, torch.rand(dim, 16, generator=gen) * 0.5 + 0.4,
                              torch.randn(dim, 16, generator=gen), torch.randn(dim, generator=gen))]

    def run(mean_out, var_out):
        xg, pcg, pmg, pvg, ga, be, mk = dev
        y, xn, cnt = torch.empty_like(xg), torch.empty_like(xg), torch.empty_like(pcg)
        s = xg.stride()
        P = lambda t: t.data_ptr()
        stream = torch.cuda.current_stream().cuda_stream
        if form in ("group", "norm"):
            rc = _lib.lib().mega_timestep_norm_fwd(P(xg), P(y), 0, bsz, length, dim, *s, *s, P(pcg), P(pmg), P(pvg), P(ga), P(be), P(mk),
                                                   groups, 1e-5, P(cnt), P(mean_out), P(var_out), stream)
            xn = y
        else:
            rc = _lib.lib().mega_tsn_ema_fwd(P(xg), P(y), P(xn), 0, bsz, length, dim, *s, *s, P(pcg), P(pmg), P(pvg), P(ga), P(be), 1e-5,
                                             P(cnt), P(mean_out), P(var_out), *(P(t) for t in prm), 16, P(mk), None, None, 0, stream)
        assert rc == 0
        return xn, cnt
    return run, dev[2], dev[3], want


@pytest.mark.parametrize("form,length,bsz,dim,split", [
    ("norm", 700, 2, 72, 0),          # several segments of at least 64 steps
    ("group", 700, 2, 128, 0),        # 256 threads along time, the last ones without steps
    ("fused", 700, 2, 72, 3),         # a cluster of blocks
    ("fused", 100, 1, 32, 3),         # one block
    ("fused", 2200, 64, 96, 3),       # the scan of several launches
])
def test_statistics_updated_in_place(form, length, bsz, dim, split, option):
    """mean_out and var_out may be prev_mean and prev_var."""
    gen = torch.Generator().manual_seed(length)
    run, pm, pv, want = _norm_call(form, gen, bsz, length, dim, 5)
    option(5, split)
    y, cnt = run(pm, pv)
    assert rel_l2(y, want[0]) < 1e-5
    assert torch.equal(cnt.cpu(), want[1])
    assert rel_l2(pm, want[2]) < 1e-5 and rel_l2(pv, want[3]) < 1e-5


def _pair_call(bsz, length, dim, gen, shift, in_place, normed=True):
    """mega_tsn_ema_fwd in bf16, its first output `shift` elements behind a 16-byte boundary; count, mean and variance before and after"""
    from fairseq_apollo_b200 import _lib
    rnd = lambda *s: torch.rand(*s, generator=gen, device="cuda")   # noqa: E731
    x = (torch.randn(bsz, length, dim, generator=gen, device="cuda") * 1.1 + 0.2).bfloat16()
    y, xn = torch.empty(x.numel() + 8, dtype=x.dtype, device="cuda")[shift:shift + x.numel()].view_as(x), torch.empty_like(x)
    pc, pm, pv = torch.full((bsz,), 5, device="cuda"), rnd(bsz, dim) * 0.3, rnd(bsz, dim) + 0.5
    ga, be, prm = rnd(dim) + 0.5, rnd(dim), (rnd(dim, 16) * 0.2, rnd(dim, 16) * 0.5 + 0.4, rnd(dim, 16) - 0.5, rnd(dim))
    before = [t.clone() for t in (pc, pm, pv, ga, be)]
    mean, var, cnt = (pm, pv, torch.empty_like(pc)) if in_place else (torch.empty_like(pm), torch.empty_like(pv), torch.empty_like(pc))
    s, P = x.stride(), lambda t: t.data_ptr()
    rc = _lib.lib().mega_tsn_ema_fwd(P(x), P(y), P(xn) if normed else None, 1, bsz, length, dim, *s, *s, P(pc), P(pm), P(pv), P(ga), P(be), 1e-5,
                                     P(cnt), P(mean), P(var), *(P(t) for t in prm), 16, None, None, None, 0,
                                     torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return x, y, xn, before, (cnt, mean, var)


@pytest.mark.parametrize("split", [2, 0])
@pytest.mark.parametrize("shift", [0, 4])
def test_statistics_in_place_where_the_second_launch_is_refused(split, shift, option):
    """bf16: TimestepNorm could run by itself, but the EMA behind it takes no output off the 16-byte boundaries.  What runs in their
    place starts from the statistics that came in.  (Outputs are bf16; the variance may come from tf32 products.)"""
    from oracle import mega_oracle as O
    option(5, split)
    x, y, xn, before, after = _pair_call(8, 1024, 2048, torch.Generator(device="cuda").manual_seed(3), shift, True)
    want = O.timestep_norm(x[:, :, ::64].cpu().double(), before[0].cpu(), *(t[..., ::64].cpu().double() for t in before[1:]), None,
                           acc_dtype=torch.float64)
    assert rel_l2(xn[:, :, ::64].float(), want[0]) < 2.0 ** -8
    assert torch.equal(after[0].cpu(), want[1])
    assert rel_l2(after[1][:, ::64], want[2]) < 1e-4 and rel_l2(after[2][:, ::64], want[3]) < 1e-3
    _, apart, _, _, _ = _pair_call(8, 1024, 2048, torch.Generator(device="cuda").manual_seed(3), shift, False)
    assert rel_l2(y.float(), apart.float()) < 2.0 ** -7


@pytest.mark.parametrize("bsz,length,dim", [(6, 768, 32), (5, 3616, 960), (48, 2272, 48)])
def test_statistics_in_place_keep_fp32(bsz, length, dim, option):
    """Where the forms over time are the faster ones, bf16 calls with statistics updated in place run in fp32 throughout: the scan's
    outputs but for single roundings (2^-9 at one in a hundred); operands rounded to bf16 would be 3e-3 off."""
    run = lambda own: _pair_call(bsz, length, dim, torch.Generator(device="cuda").manual_seed(6), 0, own)   # noqa: E731
    _, y, xn, _, own = run(True)
    option(5, 3)
    _, want, wantn, _, new = run(False)
    assert rel_l2(y.float(), want.float()) < 3e-4 and rel_l2(xn.float(), wantn.float()) < 3e-4
    assert torch.equal(own[0], new[0]) and rel_l2(own[1], new[1]) < 1e-5 and rel_l2(own[2], new[2]) < 1e-5


def test_outputs_off_the_boundaries():
    """Outputs that start between 16-byte boundaries keep to the forms over time (several launches), whatever is estimated for the
    kernels that cannot write them; a thread for every row of the whole sequence is the last resort."""
    from fairseq_apollo_b200 import _lib
    run = lambda shift: _pair_call(4, 2048, 1024, torch.Generator(device="cuda").manual_seed(4), shift, False, False)   # noqa: E731
    _, want, _, _, (_, mean, var) = run(0)
    before = _lib.launch_count()
    _, y, _, _, after = run(4)
    assert _lib.launch_count() - before > 1
    assert rel_l2(y.float(), want.float()) < 2.0 ** -7
    assert rel_l2(after[1], mean) < 1e-4 and rel_l2(after[2], var) < 1e-3


@pytest.mark.parametrize("bsz,length,dim,tile", [(8, 1088, 48, 14), (9, 1088, 48, 16), (8, 31, 48, 16), (9, 2144, 40, 164)])
def test_statistics_in_place_in_bf16(bsz, length, dim, tile, option):
    """In tensor memory, four and eight sequences to a block, in one and four runs: to the bit what new arrays receive."""
    from fairseq_apollo_b200 import _lib
    option(2, tile)
    run = lambda own: _pair_call(bsz, length, dim, torch.Generator(device="cuda").manual_seed(5), 0, own)   # noqa: E731
    _, y, xn, _, own = run(True)
    assert "tmem" in _lib.last_kernel()
    _, yn, xnn, _, new = run(False)
    assert torch.equal(y, yn) and torch.equal(xn, xnn) and all(torch.equal(a, b) for a, b in zip(own, new))


@pytest.mark.parametrize("bsz,dim", [(8, 64), (16, 1024)])   # four and eight sequences to a block
@pytest.mark.parametrize("masked", [False, True])
def test_norm_alone_in_place_in_bf16(bsz, dim, masked, option):
    from fairseq_apollo_b200 import _lib
    gen = torch.Generator(device="cuda").manual_seed(dim)
    rnd = lambda *s: torch.rand(*s, generator=gen, device="cuda")   # noqa: E731
    x, length = (torch.randn(bsz, 610, dim, generator=gen, device="cuda") + 0.2).bfloat16(), 610
    mask = torch.zeros(bsz, length, dtype=torch.bool, device="cuda")
    mask[0], mask[1, 40:77] = True, True
    pc, pm, pv, ga, be = torch.full((bsz,), 5, device="cuda"), rnd(bsz, dim), rnd(bsz, dim) + 0.5, rnd(dim) + 0.5, rnd(dim)
    s, P, res = x.stride(), lambda t: t.data_ptr(), []
    option(5, 4)
    for own in (False, True):
        y, cnt, mean, var = torch.empty_like(x), torch.empty_like(pc), pm if own else torch.empty_like(pm), pv if own else torch.empty_like(pv)
        assert _lib.lib().mega_timestep_norm_fwd(P(x), P(y), 1, bsz, length, dim, *s, *s, P(pc), P(pm), P(pv), P(ga), P(be),
                                                 P(mask) if masked else None, dim, 1e-5, P(cnt), P(mean), P(var),
                                                 torch.cuda.current_stream().cuda_stream) == 0
        assert _lib.last_kernel() == "tsn_ema_mma tmem norm"
        res.append((y, cnt, mean, var))
    assert all(torch.equal(a, b) for a, b in zip(*res))


@pytest.mark.parametrize("form,length,bsz,dim,split", [
    ("norm", 700, 2, 72, 0), ("group", 700, 2, 128, 0), ("fused", 700, 2, 72, 3), ("fused", 1, 1, 32, 3), ("fused", 2200, 64, 96, 3),
    ("norm", 1, 2, 64, 0),
])
@pytest.mark.parametrize("count", [2 ** 24 + 1, 2 ** 31 + 5])
def test_counts_stay_whole_numbers(form, length, bsz, dim, split, count, option):
    gen = torch.Generator().manual_seed(length)
    run, pm, pv, want = _norm_call(form, gen, bsz, length, dim, count)
    option(5, split)
    mean, var = torch.empty_like(pm), torch.empty_like(pv)
    y, cnt = run(mean, var)
    assert torch.equal(cnt.cpu(), want[1])
    assert rel_l2(y, want[0]) < 1e-5 and rel_l2(mean, want[2]) < 1e-5 and rel_l2(var, want[3]) < 1e-5


@pytest.mark.parametrize("groups", [None, 4])
def test_prior_gradients_of_a_long_stream(groups):
    """Backward with an incoming count of 2^27: one more step has to be seen.  dprior = n0 / n times the output's share."""
    import fairseq_apollo_b200 as M
    torch.manual_seed(1)
    dim = 64
    norm = M.TimestepNorm(dim, num_groups=groups, prior_count=2 ** 27).cuda()
    x = torch.randn(2, 3, dim, device="cuda")
    norm(x).sum().backward()
    # mean and variance stay at the prior's: dy/dmean = -rstd per channel, dy/dlogv = -(x - mean) rstd / 2 (prior variance 1)
    per = dim // (groups or dim)
    want = torch.full((dim // per,), -6.0 * per, device="cuda")
    assert rel_l2(norm.prior_mean.grad, want) < 1e-4
    dv = (-0.5 * x.sum((0, 1))).view(-1, per).sum(-1)
    assert rel_l2(norm.prior_logv.grad, dv) < 1e-4


def test_variance_of_long_segments(option):
    """Statistics after 5000 steps to 8e-7 of their size: 5000 terms summed 32 at a time, about their mean (2^-24 for each
    of a few hundred roundings that mostly cancel)."""
    from fairseq_apollo_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(5)
    bsz, length, dim = 2, 5000, 2048
    x = torch.randn(bsz, length, dim, generator=gen, device="cuda") * 1.1 + 0.3
    one, zero = torch.ones(dim, device="cuda"), torch.zeros(bsz, dim, device="cuda")
    co = [torch.rand(dim, 16, generator=gen, device="cuda") * 0.5 for _ in range(3)]
    option(5, 3)
    res = ops.tsn_ema_forward(x, torch.full((bsz,), 2, device="cuda"), zero, zero + 1, one, one, 1e-5, *co, one)
    xd, n = x.double(), length + 2
    mean = xd.sum(1) / n
    var = (2 + xd.pow(2).sum(1)) / n - mean.pow(2)
    assert rel_l2(res["mean"], mean) < 8e-7
    assert rel_l2(res["var"], var) < 8e-7


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("normed", [None, False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("length", [40, 64 * 11 + 1])
def test_pole_states_in_place(cplx, normed, dtype, length, option):
    """h_out is h_in (C interface): one segment, and more segments than a block of the chunks takes, the last of one position."""
    from fairseq_apollo_b200 import _lib
    gen = torch.Generator().manual_seed(length)
    bsz, dim, ndim, code = 3, 24, 16, {torch.float32: 0, torch.bfloat16: 1}[dtype]
    x = torch.randn(bsz, length, dim, generator=gen).to(dtype).cuda()
    pc, pm, pv = torch.full((bsz,), 2).cuda(), torch.zeros(bsz, dim).cuda(), torch.ones(bsz, dim).cuda()
    ga, be = torch.ones(dim).cuda(), torch.zeros(dim).cuda()
    two = (2,) if cplx else ()
    p, om = torch.rand(dim, ndim, generator=gen).cuda(), torch.randn(dim, generator=gen).cuda()
    q = (torch.rand(dim, ndim, *two, generator=gen) * 0.3 + (0.3 if cplx else 0.6)).cuda()
    g = torch.randn(dim, ndim, *two, generator=gen).cuda()
    start = torch.randn(bsz, dim, ndim, *two, generator=gen).cuda()
    P = lambda t: None if t is None else t.data_ptr()
    sb, sl, sd = x.stride()
    lib = _lib.lib()

    def run(h_in, h_out):
        y, xn = torch.empty_like(x), torch.empty_like(x) if normed else None
        cnt, mean, var = torch.empty_like(pc), torch.empty_like(pm), torch.empty_like(pv)
        stream = torch.cuda.current_stream().cuda_stream
        if normed is None:
            rc = (lib.mega_cema_fwd if cplx else lib.mega_ema_fwd)(
                P(x), P(y), code, bsz, dim, length, sb, sd, sl, sb, sd, sl, P(p), P(q), P(g), P(om), ndim, None, P(h_in), P(h_out), 0, 0,
                stream)
        else:
            rc = (lib.mega_tsn_cema_fwd if cplx else lib.mega_tsn_ema_fwd)(
                P(x), P(y), P(xn), code, bsz, length, dim, sb, sl, sd, sb, sl, sd, P(pc), P(pm), P(pv), P(ga), P(be), 1e-5, P(cnt),
                P(mean), P(var), P(p), P(q), P(g), P(om), ndim, None, P(h_in), P(h_out), 0, stream)
        assert rc == 0
        return y

    for form in (2, 0):
        option(6, form)
        apart, own = torch.empty_like(start), start.clone()
        want = run(start, apart)
        for _ in range(3):
            own.copy_(start)
            y = run(own, own)   # (not every form takes both: bf16 operands differ by 2^-9, a wrong start by its whole size)
            limit = 1e-5 if dtype == torch.float32 else 2.0 ** -7
            assert rel_l2(y, want) < limit and rel_l2(own, apart) < limit
