"""TimestepNorm -> EMA, and either by itself, with accumulators in tensor memory (bf16, real poles): edges of the tiles (16 channels,
8 sequences, 256 positions in chunks of 16 and parts of 32), runs of a sequence, padding, values that are not finite, waits that run
out."""
import time

import pytest
import torch

from _util import make_ema_params, rel_l2, right_pad_mask

pytestmark = pytest.mark.gpu


@pytest.fixture
def option():
    from fairseq_apollo_b200 import _lib
    yield _lib.set_option
    for key in (2, 3, 4, 5, 6):
        _lib.set_option(key, 0)


def _case(bsz, length, dim, ndim, state, masked, seed=0):
    gen = torch.Generator().manual_seed(seed + length)
    prm = make_ema_params(gen, dim, ndim)
    x = (torch.randn(bsz, length, dim, generator=gen) * 1.1 - 0.3).to(torch.bfloat16)
    count = torch.full((bsz,), 2, dtype=torch.int64)
    count[0] = 0
    stats = (count, torch.randn(bsz, dim, generator=gen) * 0.1 - 0.3, torch.rand(bsz, dim, generator=gen) + 0.5,
             torch.randn(dim, generator=gen) * 0.1 + 1, torch.randn(dim, generator=gen) * 0.1)
    h0 = torch.randn(bsz, dim, ndim, generator=gen) * 0.3 if state else None
    mask = None
    if masked:
        mask = right_pad_mask(gen, bsz, length, 0.5)
        mask[0, :min(3, length)] = True
        mask[-1, min(70, length // 2):min(130, length)] = True
    return x, stats, prm, h0, mask


def _run(x, stats, prm, h0, mask, **kw):
    from fairseq_apollo_b200 import ops
    dev = lambda t: None if t is None else t.cuda()
    p, q, g = ops.ema_coeffs(*[t.cuda() for t in prm[:4]])
    return ops.tsn_ema_forward(x.cuda(), *[t.cuda() for t in stats], 1e-5, p, q, g, prm[4].cuda(), dev(mask), h_in=dev(h0), **kw)


# Outputs: operands are bf16 (2^-9 each), sums fp32; the statistics are plain fp32 sums (1e-6 of the variance and less).
@pytest.mark.parametrize("bsz,length,dim,ndim,state,normed,silu,masked,tile", [
    (8, 256, 16, 16, False, False, False, False, 16),     # one whole tile
    (8, 257, 16, 16, False, True, False, False, 16),      # one position of another one
    (5, 31, 72, 16, False, False, True, False, 16),       # parts, channels and sequences that are not whole
    (4, 33, 8, 1, False, True, True, False, 16),          # half a tile of channels, one pole
    (9, 544, 40, 16, True, True, True, False, 16),        # states in and out
    (4, 777, 24, 5, False, True, False, False, 16),
    (8, 1, 16, 16, False, False, False, False, 16),
    (16, 1024, 208, 16, True, False, False, False, 16),
    (8, 1000, 64, 16, False, False, False, True, 16),     # padding
    (6, 512, 40, 16, True, True, True, True, 16),
    (5, 96, 24, 16, False, False, True, True, 16),
    (8, 256, 16, 16, False, False, False, False, 14),     # four sequences to a block
    (5, 290, 72, 16, False, True, True, False, 14),
    (7, 544, 40, 16, True, False, False, False, 14),
    (6, 1000, 24, 5, False, True, True, True, 14),
    (8, 1024, 48, 16, True, False, False, False, 162),    # runs
    (20, 2048 + 96, 40, 16, True, True, True, False, 164),
    (9, 2048 + 17, 64, 7, False, False, True, False, 168),
])
def test_against_oracle(option, bsz, length, dim, ndim, state, normed, silu, masked, tile):
    from fairseq_apollo_b200 import _lib
    from oracle import mega_oracle as O
    x, stats, prm, h0, mask = _case(bsz, length, dim, ndim, state, masked)
    want = state and length % 32 == 0
    option(2, tile)
    r = _run(x, stats, prm, h0, mask, want_state=want, want_normed=normed, silu=silu)
    name = _lib.last_kernel()
    assert "tmem" in name and ("segmented" in name) == (tile > 100)
    xn, cnt, mean, var = O.timestep_norm(x.float(), *stats, mask, acc_dtype=torch.float64)[:4]
    y, h = O.ema_forward_recurrence(xn.transpose(1, 2), *prm, mask, h=h0, return_state=True, silu=silu)
    assert rel_l2(r["y"].float(), y.transpose(1, 2)) < 6e-3
    assert torch.equal(r["count"].cpu(), cnt)
    assert rel_l2(r["mean"], mean) < 2e-6 and rel_l2(r["var"], var) < 2e-6
    if want:
        assert rel_l2(r["h"], h) < 6e-3
    if normed:
        assert rel_l2(r["xn"].float(), xn) < 4e-3
        if masked:
            assert (r["xn"].cpu()[mask] == 0).all()
    assert _lib.device_error() == 0


@pytest.mark.parametrize("tile", [14, 16, 162])
def test_long_sequence_far_from_zero(option, tile):
    """Values about 100 with a deviation of 1: the statistics keep their accuracy over 16384 positions."""
    from fairseq_apollo_b200 import _lib
    from oracle import mega_oracle as O
    x, stats, prm, h0, mask = _case(8, 16384, 16, 16, False, False, seed=5)
    x = (x.float() + 100).to(torch.bfloat16)
    stats[0].fill_(2)
    option(2, tile)
    r = _run(x, stats, prm, None, None, want_normed=True)
    xn, _, mean, var = O.timestep_norm(x.float(), *stats, None, acc_dtype=torch.float64)[:4]
    assert rel_l2(r["mean"], mean) < 1e-6 and rel_l2(r["var"], var) < 2e-5
    assert rel_l2(r["xn"].float(), xn) < 4e-3
    assert _lib.device_error() == 0


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("tile,at", [(14, 300), (16, 300), (16, 0), (162, 511)])
def test_not_finite_stays_in_its_channel(option, value, tile, at):
    option(2, tile)
    x, stats, prm, h0, mask = _case(8, 1024, 48, 16, True, False, seed=2)
    clean = _run(x, stats, prm, h0, mask, want_state=True, want_normed=True)
    x[2, at, 21] = value
    r = _run(x, stats, prm, h0, mask, want_state=True, want_normed=True)
    rest = torch.ones(8, 48, dtype=torch.bool)
    rest[2, 21] = False
    for k in ("y", "xn"):
        a, b = r[k].cpu().transpose(1, 2), clean[k].cpu().transpose(1, 2)
        assert torch.equal(a[rest], b[rest]) and torch.equal(a[2, 21, :at], b[2, 21, :at])
        assert not torch.isfinite(a[2, 21, at:].float()).any()
    for k in ("h", "mean", "var"):
        assert torch.equal(r[k].cpu()[rest], clean[k].cpu()[rest])
    assert not torch.isfinite(r["h"][2, 21]).any() and not torch.isfinite(r["mean"][2, 21])


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("tile", [14, 16])
def test_not_finite_ahead_of_padding(option, value, tile):
    """The normalised activations of padded positions are zero, behind such a value too; at the others its channel is not finite."""
    option(2, tile)
    x, stats, prm, _, _ = _case(8, 700, 48, 16, False, False, seed=4)
    mask = torch.zeros(8, 700, dtype=torch.bool)
    mask[2, 310:340] = True
    mask[2, 512:] = True
    x[2, 300, 21] = value
    xn = _run(x, stats, prm, None, mask, want_normed=True)["xn"].cpu()
    assert (xn[mask] == 0).all()
    late = ~mask[2]
    late[:300] = False
    assert not torch.isfinite(xn[2, late, 21].float()).any()


def _ema(x, prm, h0, tile, option, **kw):
    from fairseq_apollo_b200 import _lib, ops
    p, q, g = ops.ema_coeffs(*[t.cuda() for t in prm[:4]])
    option(2, tile)
    r = ops.ema_forward(x.cuda().transpose(1, 2), p, q, g, prm[4].cuda(), h_in=None if h0 is None else h0.cuda(), **kw)
    assert "ema_mma tmem" == _lib.last_kernel()
    y, h = r if isinstance(r, tuple) else (r, None)
    return y.float().cpu(), None if h is None else h.cpu()


# As above: operands and outputs are bf16 (2^-9 each), sums fp32.
@pytest.mark.parametrize("bsz,length,dim,ndim,state,silu,tile", [
    (8, 256, 16, 16, False, False, 16),
    (5, 257, 72, 16, False, True, 16),
    (9, 544, 40, 16, True, True, 16),
    (4, 31, 24, 5, False, False, 16),
    (8, 17, 16, 1, False, False, 16),
    (7, 544, 40, 16, True, False, 14),
    (6, 1000, 24, 5, False, True, 14),
    (4, 33, 8, 16, False, False, 14),
    (8, 1024, 48, 16, True, False, 162),
    (9, 2048 + 17, 64, 7, False, True, 168),
])
def test_ema_by_itself(option, bsz, length, dim, ndim, state, silu, tile):
    from oracle import mega_oracle as O
    x, _, prm, h0, _ = _case(bsz, length, dim, ndim, state, False)
    y, h = _ema(x, prm, h0, tile, option, want_state=state, silu=silu)
    want, last = O.ema_forward_recurrence(x.double().transpose(1, 2), *prm, None, h=h0, return_state=True, silu=silu)
    assert rel_l2(y, want) < 6e-3
    if state:
        assert rel_l2(h, last) < 6e-3


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("tile,at", [(14, 300), (16, 0), (16, 1023), (162, 511), (162, 512)])
@pytest.mark.parametrize("state", [False, True])
def test_ema_by_itself_not_finite(option, value, tile, at, state):
    """From such an input on its row is the recurrence's (weights of one sign: infinite, not NaN), in the state too; a state that comes in
    infinite makes an infinite row; the other rows know nothing of it."""
    x, _, prm, h0, _ = _case(8, 1024, 48, 16, True, False, seed=3)
    prm = [prm[0], prm[1], prm[2].abs(), prm[3].abs(), prm[4].abs()]   # p, g and omega of one sign
    h0 = h0 if state else None
    clean, last = _ema(x, prm, h0, tile, option, want_state=state)
    x[2, at, 21] = value
    if state:
        h0[5, 7, 3] = float("inf")
    y, h = _ema(x, prm, h0, tile, option, want_state=state)
    rest = torch.ones(8, 48, dtype=torch.bool)
    rest[2, 21] = False
    rest[5, 7] = not state
    assert torch.equal(y[rest], clean[rest]) and torch.equal(y[2, 21, :at], clean[2, 21, :at])
    same = (lambda t: t.isnan()) if value != value else (lambda t: t == value)
    assert same(y[2, 21, at:]).all()
    if state:
        assert torch.equal(h[rest], last[rest]) and same(h[2, 21]).all()
        assert (y[5, 7] == float("inf")).all() and h[5, 7, 3] == float("inf") and torch.isfinite(h[5, 7, :3]).all()


@pytest.mark.parametrize("bsz,length,dim,silu,state", [(8, 2000, 1024, False, False), (16, 4096, 1024, True, False), (8, 4096, 1024, False, True),
                                                       (3, 4096, 2048, False, False)])
def test_ema_by_itself_is_chosen(option, bsz, length, dim, silu, state):
    """Against the form in the same roundings that walks a sequence as one chain: both are 2.3e-3 from float64 (5e-3 apart at most)."""
    from fairseq_apollo_b200 import _lib, ops
    x, _, prm, h0, _ = _case(bsz, length, dim, 16, state, False)
    y, h = _ema(x, prm, h0, 0, option, want_state=state, silu=silu)
    p, q, g = ops.ema_coeffs(*[t.cuda() for t in prm[:4]])
    option(2, 224)
    r = ops.ema_forward(x.cuda().transpose(1, 2), p, q, g, prm[4].cuda(), h_in=None if h0 is None else h0.cuda(), want_state=state, silu=silu)
    assert "tmem" not in _lib.last_kernel()
    want, last = r if isinstance(r, tuple) else (r, None)
    assert rel_l2(y, want.float()) < 5e-3
    if state:
        assert rel_l2(h, last) < 5e-3


@pytest.mark.parametrize("tile", [14, 16, 164])
def test_wait_that_runs_out(option, tile):
    """x of 64 positions never arrives: the kernel gives up, says so, and the next call is as always."""
    from fairseq_apollo_b200 import _lib
    x, stats, prm, h0, mask = _case(8, 4096, 64, 16, False, False)
    assert _lib.device_error(reset=True) == 0
    option(2, tile)
    good = _run(x, stats, prm, h0, mask)["y"]
    option(3, 2_000_000)   # SM cycles, about a millisecond
    option(4, 5)
    start = time.time()
    _run(x, stats, prm, h0, mask)
    torch.cuda.synchronize()
    assert time.time() - start < 5.0
    assert _lib.device_error(reset=True) != 0
    option(3, 0)
    option(4, 0)
    assert torch.equal(_run(x, stats, prm, h0, mask)["y"], good)
    assert _lib.device_error() == 0


@pytest.mark.parametrize("tile,step", [(14, 5), (16, 62), (164, 5), (164, 14)])   # (of 64 loads, of 16 of a run)
@pytest.mark.parametrize("alone", [False, True])
def test_waits_that_run_out_at_once(option, tile, step, alone):
    """The same with a limit below what a copy takes: whoever waits leaves at once, and what is under way is still waited for, also once
    the last load has been issued."""
    from fairseq_apollo_b200 import _lib
    x, stats, prm, h0, mask = _case(8, 4096, 64, 16, False, False)
    assert _lib.device_error(reset=True) == 0
    call = lambda: _ema(x, prm, None, tile, option)[0] if alone else _run(x, stats, prm, h0, mask)["y"]   # noqa: E731
    option(2, tile)
    good = call()
    option(3, 1)
    option(4, step)
    for _ in range(3):
        call()
    assert _lib.device_error(reset=True) != 0
    option(3, 0)
    option(4, 0)
    assert torch.equal(call(), good)
    assert _lib.device_error() == 0


def test_strides_and_views(option):
    """Rows that are not 32-byte aligned and a time-major view give what contiguous tensors give."""
    from fairseq_apollo_b200 import _lib, ops
    x, stats, prm, h0, mask = _case(8, 320, 32, 16, False, False)
    option(2, 16)
    want = _run(x, stats, prm, None, None)["y"]
    wide = torch.zeros(8, 320, 40, dtype=torch.bfloat16)
    wide[:, :, 8:] = x
    major = x.transpose(0, 1).contiguous()
    p, q, g = ops.ema_coeffs(*[t.cuda() for t in prm[:4]])
    for v in (wide.cuda()[:, :, 8:], major.cuda().transpose(0, 1)):
        r = ops.tsn_ema_forward(v, *[t.cuda() for t in stats], 1e-5, p, q, g, prm[4].cuda())["y"]
        assert "tmem" in _lib.last_kernel()
        assert torch.equal(r, want)


@pytest.mark.parametrize("value", [None, float("nan"), float("inf")])
def test_ema_over_its_inputs(option, value):
    """Behind TimestepNorm by itself, whose outputs lie where the EMA's go: what it gives from a place of their own.  From a value that is
    not finite on its row is NaN, in the state too, and the other rows know nothing of it."""
    from fairseq_apollo_b200 import _lib
    x, stats, prm, h0, _ = _case(8, 4096, 1024, 16, True, False, seed=6)
    if value is not None:
        x[2, 300, 21] = value
    option(5, 2)
    option(6, 1)
    apart = _run(x, stats, prm, h0, None, want_state=True, want_normed=True)
    assert _lib.last_kernel() == "ema_mma tmem"
    over = _run(x, stats, prm, h0, None, want_state=True)
    assert _lib.last_kernel() == "ema_mma tmem"
    a, b = over["y"].transpose(1, 2), apart["y"].transpose(1, 2)
    rest = torch.ones(8, 1024, dtype=torch.bool)
    rest[2, 21] = value is None
    assert torch.equal(a[rest], b[rest]) and torch.equal(over["h"][rest], apart["h"][rest])
    assert torch.equal(a[2, 21, :300], b[2, 21, :300])
    if value is not None:
        assert a[2, 21, 300:].isnan().all() and over["h"][2, 21].isnan().all()


# What a call takes by itself, real poles, against the other form.  The two are apart by no more than their distances from float64
# together, which their own tests bound by 6e-3 (above) and 1e-2 (the chain: test_tensor_core_path_with_padding_mask).
@pytest.mark.parametrize("bsz,length,dim,masked,normed,name", [
    (16, 4096, 1024, False, False, "tsn_ema_mma tmem"),
    (16, 4096, 1024, True, False, "tsn_ema_mma tmem mask"),
    (8, 1024, 2048, False, True, "tsn_ema_mma tmem"),
    (8, 1024, 2048, True, True, "tsn_ema_mma tmem mask"),
    (3, 4096, 2048, False, False, "tsn_ema_mma tmem"),      # fewer than four sequences
    (16, 60, 1024, False, False, "tsn_ema_mma tile=2 warps_per_column=2 pipe=4 norm ema"),      # the chain of mma.sync
    (24, 1500, 1000, False, False, "tsn_ema_mma tile=2 warps_per_column=2 pipe=1 norm ema"),
    (58, 96, 1096, False, False, "tsn_ema_mma tile=8 warps_per_column=1 pipe=1 norm ema"),      # (37 us, in tensor memory 49)
    (37, 154, 1120, False, True, "tsn_ema_mma tile=2 warps_per_column=2 pipe=1 norm ema xn"),   # (43, 54)
])
def test_pair_is_chosen(option, bsz, length, dim, masked, normed, name):
    from fairseq_apollo_b200 import _lib
    x, stats, prm, _, mask = _case(bsz, length, dim, 16, False, masked)
    r = _run(x, stats, prm, None, mask, want_normed=normed)
    assert _lib.last_kernel() == name
    option(2, 16 if "tile" in name else 22 if masked or normed else 224)
    other = _run(x, stats, prm, None, mask, want_normed=normed)
    assert ("tmem" in _lib.last_kernel()) == ("tile" in name)
    assert rel_l2(r["y"].float(), other["y"].float()) < 1.6e-2
    assert rel_l2(r["mean"], other["mean"]) < 1e-4 and rel_l2(r["var"], other["var"]) < 2e-3
    if normed:
        assert rel_l2(r["xn"].float(), other["xn"].float()) < 1.4e-2   # (4e-3 and 1e-2)


@pytest.mark.parametrize("bsz,length,dim,masked", [(8, 256, 16, False), (5, 290, 72, False), (4, 33, 8, True), (16, 1000, 40, True),
                                                   (20, 2048, 1100 // 4 * 8, False), (9, 1, 24, False)])
def test_norm_alone(option, bsz, length, dim, masked):
    from fairseq_apollo_b200 import _lib, ops
    from oracle import mega_oracle as O
    x, stats, _, _, mask = _case(bsz, length, dim, 1, False, masked)
    _lib.set_option(5, 4)
    try:
        r = ops.timestep_norm_fwd(x.cuda(), *[t.cuda() for t in stats], None if mask is None else mask.cuda())
        assert _lib.last_kernel() == "tsn_ema_mma tmem norm"
    finally:
        _lib.set_option(5, 0)
    ref = O.timestep_norm(x.float(), *stats, mask, acc_dtype=torch.float64)
    assert rel_l2(r[0].float(), ref[0]) < 4e-3 and torch.equal(r[1].cpu(), ref[1])
    assert rel_l2(r[2], ref[2]) < 2e-6 and rel_l2(r[3], ref[3]) < 2e-6
    if masked:
        assert (r[0].cpu()[mask] == 0).all()
    assert _lib.device_error() == 0


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_norm_alone_not_finite(option, value):
    """As in the scan: such a value's channel is not finite from there on, the others know nothing of it."""
    from fairseq_apollo_b200 import _lib, ops
    x, stats, _, _, _ = _case(8, 600, 16, 1, False, False)
    clean = x.clone()
    x[3, 270, 5] = value
    _lib.set_option(5, 4)
    try:
        a, b = [ops.timestep_norm_fwd(v.cuda(), *[t.cuda() for t in stats])[0].cpu() for v in (x, clean)]
    finally:
        _lib.set_option(5, 0)
    rest = torch.ones(8, 16, dtype=torch.bool)
    rest[3, 5] = False
    assert torch.equal(a.transpose(1, 2)[rest], b.transpose(1, 2)[rest]) and torch.equal(a[3, :270, 5], b[3, :270, 5])
    assert not torch.isfinite(a[3, 270:, 5].float()).any()
