"""The length-contiguous EMA kernel at the edges of its tiles: segments of 32 positions, groups of 16 segments, warps of
two, four or eight groups, several rows per block.

Reference: the float64 oracle on the same inputs.  Tolerance: a product of two floats taken in three bf16 parts each is
right to 3 * 2^-24, a sum over a tile truncates at 2^-24 of it at most 12 times in a row, and a value passes three such
products (states, outputs, entering states) and two scans: 1e-5 relative 2-norm bounds them with the powers' roundings;
16-bit outputs are rounded by at most 2^-8 (bf16,
8 significant bits) and 2^-11 (fp16) of their values."""
import pytest
import torch

from _util import make_ema_params, rel_l2

pytestmark = pytest.mark.gpu
LIMIT = {torch.float32: 1e-5, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


@pytest.mark.parametrize("bidir,norm,shift", [(True, True, True), (True, False, False), (False, True, True), (False, False, True)])
@pytest.mark.parametrize("length,bsz,ndim,dtype,masked", [
    (512, 9, 16, torch.float32, False),     # the shortest row, more rows than a block takes
    (1023, 3, 16, torch.bfloat16, True),
    (1024, 8, 3, torch.float32, True),      # inert poles
    (1025, 2, 16, torch.float16, False),
    (4096, 2, 16, torch.float32, True),
    (4097, 2, 16, torch.bfloat16, True),    # four groups per warp
    (12000, 1, 16, torch.float32, True),    # a last warp that is partly beyond the row
    (40000, 1, 16, torch.float32, False),   # the longest rows: eight groups per warp, causal only
])
def test_row_tiles(length, bsz, ndim, dtype, masked, bidir, norm, shift):
    from fairseq_apollo_b200 import _lib, ops
    from oracle import mega_oracle as O
    if length == 40000 and (bidir or norm):
        pytest.skip("one direction is enough at this length")
    gen = torch.Generator().manual_seed(length + 2 * bidir + norm)
    dim = 3
    x = (torch.randn(bsz, dim, length, generator=gen) * 1.1 + 0.3).to(dtype)
    mask = None
    if masked:
        mask = torch.zeros(bsz, length, dtype=torch.bool)
        mask[0, 5:70] = True                   # inside the row
        mask[-1, length - length // 2:] = True   # whole segments and warps at its end
    params = make_ema_params(gen, dim, ndim, bidirectional=bidir)
    gamma, beta = torch.rand(dim, generator=gen) + 0.5, torch.randn(dim, generator=gen)
    p, q, g = (t.cuda() for t in O.ema_coeffs(*params[:4]))
    m = None if mask is None else mask.cuda()
    xg = x.cuda()
    if norm:
        y = ops.sqn_ema_forward(xg, gamma.cuda(), beta.cuda(), 1e-5, p, q, g, params[4].cuda(), m, bidir, shift)
    else:
        y = ops.ema_forward(xg, p, q, g, params[4].cuda(), m, bidirectional=bidir, shift=shift, silu=True)
    assert y is not None and "rowres" in _lib.last_kernel()
    ref = O.sequence_norm(x.double(), gamma.double(), beta.double(), mask)[0] if norm else x.double()
    ref = O.ema_forward_recurrence(ref.double(), *[t.double() for t in params], mask, bidirectional=bidir, shift=shift)
    if not norm:
        ref = torch.nn.functional.silu(ref)
    assert rel_l2(y, ref) < LIMIT[dtype]
