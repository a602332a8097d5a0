"""The Mega block's native paths against its own sequence of operations in fp32: decoding by one library call per token
(prompt lengths that are no multiple of eight, batches at the edges of the 8-row tiles, across the end of a chunk), and the
training pass as one autograd Function.

bf16 rounds operands and intermediate activations a few times (2^-8 each at most): 1e-2; fp16 an eighth of that.  Gradients are
sums over positions of products of such values; those of the query / key affine and the relative bias cancel, and the fp32
path's own sequence at the same precision is as far away: 4e-2 (fp16 1e-2, fp32 2e-5)."""
import copy

import pytest
import torch

from _util import rel_l2

pytestmark = pytest.mark.gpu


def _block(M, dim, zdim, chunk, cplx, bidir=False, groups=None, length=0):
    kw = dict(bidirectional=True, rel_pos_bias='simple', max_positions=length) if bidir else \
        dict(efficient_attn=True, rel_pos_bias='rotary', norm_num_groups=groups)
    blk = M.MovingAverageGatedAttention(dim, zdim, 2 * dim, 16, chunk_size=chunk, moving_layer='cema' if cplx else 'ema',
                                        moving_act='silu', **kw)
    with torch.no_grad():
        for name, p in blk.named_parameters():
            if name in ('gamma', 'beta'):
                p.normal_(0, 0.5)
            elif p.dim() == 1 and name.endswith('bias'):
                p.normal_(0, 0.1)
    return blk.cuda()


@pytest.mark.parametrize("bsz,dim,zdim,chunk,prompt,steps,dtype,cplx", [
    (1, 32, 64, 16, 0, 18, torch.bfloat16, False),     # no prompt, into the second chunk
    (3, 96, 128, 64, 13, 6, torch.float16, True),
    (8, 64, 256, 64, 61, 5, torch.bfloat16, False),    # over the end of the chunk
    (9, 64, 64, 128, 33, 4, torch.float16, False),     # two tiles of sequences
    (33, 32, 64, -1, 40, 3, torch.bfloat16, True),     # no chunks; eight tiles' form
])
def test_decoding_step(bsz, dim, zdim, chunk, prompt, steps, dtype, cplx):
    import fairseq_apollo_b200 as M
    torch.manual_seed(bsz)
    blk = _block(M, dim, zdim, chunk, cplx).eval().to(dtype)
    ref = copy.deepcopy(blk).float()
    x = torch.randn(bsz, prompt + steps, dim, device="cuda").to(dtype)
    got, want, a, b = [], [], {}, {}
    with torch.no_grad():
        if prompt:
            got.append(blk(x[:, :prompt].contiguous(), incremental_state=a)[0])
            want.append(ref(x[:, :prompt].float(), incremental_state=b)[0])
        before = M.launch_count()
        for t in range(prompt, prompt + steps):
            got.append(blk(x[:, t:t + 1].contiguous(), incremental_state=a)[0])
        if chunk < 0 or prompt + steps <= chunk:
            assert M.launch_count() - before <= 5 * steps + 8   # (five launches a step, a few to set the first one up)
        for t in range(prompt, prompt + steps):
            want.append(ref(x[:, t:t + 1].float().contiguous(), incremental_state=b)[0])
    limit = 1e-2 if dtype == torch.bfloat16 else 2e-3
    assert rel_l2(torch.cat(got, 1).float(), torch.cat(want, 1)) < limit
    sa, sb = ({k.split('.')[-1] + '.' + n: v for k, d in s.items() for n, v in d.items() if v is not None} for s in (a, b))
    assert sa.keys() == sb.keys()
    for name in sa:
        assert rel_l2(sa[name].to(sb[name].dtype), sb[name]) < limit, name


@pytest.mark.parametrize("bsz,length,dim,zdim,chunk,dtype,cplx,bidir,groups,pad", [
    (2, 64, 64, 64, 32, torch.float32, False, False, None, False),
    (2, 96, 128, 128, 32, torch.float16, True, False, 4, False),
    (1, 40, 64, 256, 40, torch.bfloat16, False, False, None, False),
    (3, 57, 72, 64, -1, torch.float32, False, True, None, True),       # rows in no whole pieces
    (3, 256, 64, 64, -1, torch.bfloat16, True, True, None, True),      # one piece per lane of a warp
    (2, 520, 64, 64, -1, torch.float16, False, True, None, True),      # a third piece of one lane
])
def test_training_function(bsz, length, dim, zdim, chunk, dtype, cplx, bidir, groups, pad, monkeypatch):
    import fairseq_apollo_b200 as M
    from fairseq_apollo_b200 import block_function
    torch.manual_seed(length)
    blk = _block(M, dim, zdim, chunk, cplx, bidir, groups, length).train().to(dtype)
    ref = copy.deepcopy(blk).float()
    x, dy = (torch.randn(bsz, length, dim, device="cuda").to(dtype) for _ in range(2))
    mask = None
    if pad:
        mask = torch.zeros(bsz, length, dtype=torch.bool, device="cuda")
        mask[0, length // 2:] = True
        mask[-1] = True          # padded throughout
    xs = [x.clone().requires_grad_(True), x.float().requires_grad_(True)]
    assert block_function.mode_of(blk, x, mask, None, False, False) is not None
    y = blk(xs[0], mask)[0]
    y.backward(dy)
    monkeypatch.setattr(block_function, "mode_of", lambda *a: None)
    want = ref(xs[1], mask)[0]
    want.backward(dy.float())
    out, grad = {torch.float32: (1e-5, 2e-5), torch.bfloat16: (1e-2, 4e-2), torch.float16: (2e-3, 1e-2)}[dtype]
    assert rel_l2(y.float(), want) < out
    assert rel_l2(xs[0].grad.float(), xs[1].grad) < grad
    for (name, p), (_, r) in zip(blk.named_parameters(), ref.named_parameters()):
        assert (p.grad is None) == (r.grad is None), name
        if p.grad is not None:
            assert rel_l2(p.grad.float(), r.grad) < grad, name
