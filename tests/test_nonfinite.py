"""Infinities and NaN: where they were an output's own business, they still are."""
import pytest
import torch

from _util import make_ema_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sequence_norm_backward_ignores_padding(dtype):
    """(B, L, D): what stands at padded positions takes no part, NaN included."""
    import fairseq_apollo_b200 as M
    torch.manual_seed(2)
    norm = M.SequenceNorm(64).cuda()
    x = torch.randn(2, 200, 64, device="cuda").to(dtype)
    mask = torch.zeros(2, 200, dtype=torch.bool, device="cuda")
    mask[1, 150:] = True
    grads = []
    for fill in (0.0, float("nan"), float("inf")):
        norm.zero_grad()
        xx = x.masked_fill(mask.unsqueeze(-1), fill).requires_grad_(True)
        norm(xx, mask, length_last=False).backward(torch.ones_like(x))
        grads.append((xx.grad, norm.weight.grad.clone(), norm.bias.grad.clone()))
    for other in grads[1:]:
        for a, b in zip(grads[0], other):
            torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)


def test_running_variance_of_nan_is_nan():
    from fairseq_apollo_b200 import ops
    x = torch.randn(1, 300, 64, device="cuda")
    x[0, 40, 5] = float("nan")
    one = torch.ones(64, device="cuda")
    _, _, mean, var = ops.timestep_norm_fwd(x, torch.full((1,), 2, device="cuda"), torch.zeros(1, 64, device="cuda"),
                                            torch.ones(1, 64, device="cuda"), one, one)
    assert mean[0, 5].isnan() and var[0, 5].isnan()
    assert var.isnan().sum() == 1 and mean.isnan().sum() == 1


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("length,at", [(600, 17), (600, 64), (1300, 1055), (5000, 4998)])
def test_causal_rows_keep_the_past(value, dtype, length, at):
    """Length-contiguous causal EMA: what comes before a non-finite input is as without it."""
    from fairseq_apollo_b200 import _lib, ops
    from oracle import mega_oracle as O
    gen = torch.Generator().manual_seed(at)
    bsz, dim = 2, 3
    x = torch.randn(bsz, dim, length, generator=gen).to(dtype).cuda()
    prm = make_ema_params(gen, dim, 16)
    c = [t.cuda() for t in (*O.ema_coeffs(*prm[:4]), prm[4])]
    clean = ops.ema_forward(x, *c)
    assert _lib.last_kernel() == "rowres"
    bad = x.clone()
    bad[1, 2, at] = value
    bad[0, 0, at] = value
    bad[0, 0, at - 3] = value
    y = ops.ema_forward(bad, *c)
    assert torch.equal(y[1, 2, :at], clean[1, 2, :at])
    assert torch.equal(y[0, 0, :at - 3], clean[0, 0, :at - 3])
    assert not torch.isfinite(y[1, 2, at:]).any() and not torch.isfinite(y[0, 0, at - 3:]).any()
    rest = [(0, 1), (0, 2), (1, 0), (1, 1)]
    assert all(torch.equal(y[i, j], clean[i, j]) for i, j in rest)
