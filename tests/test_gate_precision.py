"""The training pass's gates where they are nearly closed or open: every value to the precision of its type.

Rounding to a type of p significant bits is at most 2^-p of a (normal) value: 2^-8 in bf16, 2^-11 in fp16.  Before it, fp32
values are a few 2^-23 off: 2^-20, and sixteen times that where two terms of a derivative cancel to a twentieth."""
import pytest
import torch

pytestmark = pytest.mark.gpu
ROUND = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 0.0}
CODE = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}


def _operands(dtype, n=5):
    gen = torch.Generator().manual_seed(1)
    v = torch.cat([torch.linspace(-10, -5, 2048), torch.linspace(-5, 5, 2048), torch.linspace(5, 10, 2048)])
    one = [v.to(dtype).cuda().view(24, 256)]
    return one + [(torch.rand(24, 256, generator=gen) + 0.5).to(dtype).cuda() for _ in range(n - 1)]


def _close(got, want, dtype, keep=None):
    """keep: where the terms of the value do not cancel; values below the type's normal range are on a fixed grid"""
    err = (got.double() - want).abs() / want.abs().clamp(min=torch.finfo(dtype).tiny)
    if keep is not None:
        err = err[keep]
    assert float(err.max()) < ROUND[dtype] + 2.0 ** -20 * (1 if keep is None else 16), float(err.max())


def _call(name, *args):
    from fairseq_apollo_b200 import _lib
    rc = getattr(_lib.lib(), name)(*args, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()


@pytest.mark.parametrize("dtype", list(CODE))
def test_backward_gates(dtype):
    v, g, a, c, d = _operands(dtype)
    p = lambda t: (t.data_ptr(), 256)
    s = lambda t: torch.sigmoid(t.double())
    one = lambda t: 1 + t.double() * s(-t.double())          # d silu(t) / dt = sigmoid(t) (1 + t sigmoid(-t))
    ds = lambda t: s(t) * one(t)
    far = lambda t: one(t).abs() > 0.05
    o0, o1, o2 = (torch.empty_like(v) for _ in range(3))
    _call("mega_gate_silu_bwd", *p(g), *p(v), *p(o0), None, CODE[dtype], 24, 256)
    _close(o0, g.double() * ds(v), dtype, far(v))
    _call("mega_gate_mul_silu_bwd", *p(g), *p(a), *p(v), *p(o0), *p(o1), None, CODE[dtype], 24, 256)
    _close(o0, g.double() * v.double() * s(v), dtype)
    _close(o1, g.double() * a.double() * ds(v), dtype, far(v))
    _call("mega_gate_output_bwd", *p(g), *p(a), *p(v), *p(c), *p(d), *p(o0), *p(o1), *p(o2), None, None, CODE[dtype], 24, 256)
    t = c.double() + d.double()
    _close(o0, g.double() * s(-v.double()), dtype)
    diff = t * s(t) - a.double()
    _close(o1, g.double() * diff * s(v) * s(-v.double()), dtype, diff.abs() > 0.05)
    _close(o2, g.double() * s(v) * ds(t), dtype, far(t))


@pytest.mark.parametrize("dtype", list(CODE))
def test_forward_gates(dtype):
    from fairseq_apollo_b200 import ops
    v, a, b, c, _ = _operands(dtype)
    s = torch.sigmoid(v.double())
    _close(ops.gate_silu(v), v.double() * s, dtype)
    _close(ops.gate_mul_silu(a, v), a.double() * v.double() * s, dtype)
    t = b.double() + c.double()
    h = t * torch.sigmoid(t)
    want = a.double() + s * (h - a.double())
    _close(ops.gate_output(a, v, b, c), want, dtype, want.abs() > 0.05)
