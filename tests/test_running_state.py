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
    for key in (1, 5):
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
