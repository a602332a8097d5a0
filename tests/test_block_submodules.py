"""The block's projections are modules: their hooks run, and what stands in their place is what is called."""
import copy

import pytest
import torch

from _util import rel_l2

pytestmark = pytest.mark.gpu


class Adapter(torch.nn.Linear):
    """A linear layer with something beside it, as low-rank adapters and quantised layers are built."""

    def forward(self, x):
        return 3.0 * super().forward(x) + 1.0


def _adapted(lin):
    new = Adapter(lin.in_features, lin.out_features, bias=lin.bias is not None)
    new.load_state_dict(lin.state_dict())
    return new.to(lin.weight)


def _block(M, bidir):
    torch.manual_seed(5)
    kw = dict(bidirectional=True, rel_pos_bias='simple', max_positions=64) if bidir else \
        dict(efficient_attn=True, rel_pos_bias='rotary')
    blk = M.MovingAverageGatedAttention(64, 64, 128, 16, chunk_size=-1 if bidir else 32, moving_act='silu', moving_layer='ema', **kw)
    with torch.no_grad():
        for lin in (blk.v_proj, blk.mx_proj, blk.h_proj):
            lin.weight.normal_(0, 0.1)
    return blk.cuda().bfloat16()


def _run(blk, x, how):
    if how == "train":
        xx = x.clone().requires_grad_(True)
        y = blk.train()(xx)[0]
        y.sum().backward()
        return y.detach()
    blk.eval()
    with torch.no_grad():
        if how == "infer":
            return blk(x)[0]
        inc = {}
        return torch.cat([blk(x[:, t:t + 1].contiguous(), incremental_state=inc)[0] for t in range(x.size(1))], 1)


@pytest.mark.parametrize("how,bidir", [("train", False), ("train", True), ("infer", False), ("decode", False)])
@pytest.mark.parametrize("name", ["v_proj", "mx_proj", "h_proj"])
def test_hooks_and_replacements(how, bidir, name):
    import fairseq_apollo_b200 as M
    blk = _block(M, bidir)
    length = 8 if how == "decode" else 32
    x = torch.randn(2, length, 64, device="cuda").bfloat16()
    plain = _run(blk, x, how)
    seen = []
    handles = [getattr(blk, name).register_forward_hook(lambda m, i, o: seen.append("forward")),
               getattr(blk, name).register_forward_pre_hook(lambda m, i: seen.append("pre"))]
    if how == "train":
        handles.append(getattr(blk, name).register_full_backward_hook(lambda m, a, b: seen.append("backward")))
    hooked = _run(blk, x, how)
    calls = length if how == "decode" else 1
    assert seen.count("forward") == calls and seen.count("pre") == calls
    assert how != "train" or seen.count("backward") == 1
    assert rel_l2(hooked, plain) < 1e-2
    for h in handles:
        h.remove()
    assert torch.equal(_run(blk, x, how), plain)
    ref = copy.deepcopy(blk).float()
    setattr(blk, name, _adapted(getattr(blk, name)))
    setattr(ref, name, _adapted(getattr(ref, name)))
    got = _run(blk, x, how)
    assert rel_l2(got.float(), _run(ref, x.float(), how)) < 2e-2
    assert rel_l2(got, plain) > 2e-2


@pytest.mark.parametrize("what", ["hook", "global", "forward", "replaced", "positions"])
def test_changes_during_a_generation(what):
    import fairseq_apollo_b200 as M
    blk = _block(M, False).eval()
    x = torch.randn(2, 6, 64, device="cuda").bfloat16()
    seen, inc, handle = [], {}, None
    with torch.no_grad():
        for t in range(6):
            if t == 3:
                note = lambda m, *a: seen.append(1) if m in (blk.v_proj, blk.rel_pos_bias) else None
                if what == "hook":
                    blk.v_proj.register_forward_hook(note)
                elif what == "positions":
                    blk.rel_pos_bias.register_forward_pre_hook(note)
                elif what == "global":
                    handle = torch.nn.modules.module.register_module_forward_hook(note)
                elif what == "forward":
                    own = blk.v_proj.forward
                    blk.v_proj.forward = lambda v: (seen.append(1), own(v))[1]
                else:
                    blk.v_proj = _adapted(blk.v_proj)
                    blk.v_proj.register_forward_hook(note)
            blk(x[:, t:t + 1].contiguous(), incremental_state=inc)
    if handle is not None:
        handle.remove()
    assert len(seen) >= 3


def test_hooks_of_the_moving_average_run_in_training():
    import fairseq_apollo_b200 as M
    blk = _block(M, False).train()
    x = torch.randn(2, 32, 64, device="cuda").bfloat16().requires_grad_(True)
    seen = []
    h = blk.move.register_full_backward_pre_hook(lambda m, g: seen.append(1))
    blk(x)[0].sum().backward()
    assert seen
    h.remove()


class Scaled:
    """mix-in: a moving average with a forward of its own"""

    def forward(self, *args, **kw):
        return 2.0 * super().forward(*args, **kw)


def test_derived_moving_average_in_training():
    import fairseq_apollo_b200 as M
    blk = _block(M, False).train()
    x = torch.randn(2, 32, 64, device="cuda").bfloat16().requires_grad_(True)
    first = M.timestep_norm_ema(blk.norm, blk.move, x).detach()
    blk.move.__class__ = type("ScaledEMA", (Scaled, type(blk.move)), {})
    assert rel_l2(M.timestep_norm_ema(blk.norm, blk.move, x), 2 * first) < 1e-2
