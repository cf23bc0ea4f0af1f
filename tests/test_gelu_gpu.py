"""The GELU kernels at the sizes where their launch changes, and over the whole range of arguments, against 64 bits."""
import pytest
import torch

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.ops import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def reference(y, g):
    y = y.double().requires_grad_()
    out = torch.nn.functional.gelu(y, approximate="tanh")
    out.backward(g.double())
    return out.detach(), y.grad


# one group of eight, a CTA and one more, the last size of one group a thread and the first of four, a ragged last CTA of four
@pytest.mark.parametrize("rows,F", [(1, 8), (257, 8), (148 * 8 - 1, 8192), (148 * 8, 8192), (2997, 6400)])
def test_sizes(rows, F):
    torch.manual_seed(rows)
    y = (3 * torch.randn(rows, F, device=DEV)).to(torch.bfloat16).requires_grad_()
    out = ops.activation(y, "gelu")
    g = torch.randn_like(out)
    out.backward(g)
    ref, dref = reference(y.detach(), g)
    # one rounding to 16 bits; 1 + tanh cancels in the 64-bit reference, 2^-53 of x / 2; in the gradient x s (1 - s) (...)
    # cancels against s around its zero at -0.75: a few fp32 units of the terms, which are below 1
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-14).all()
    assert ((y.grad.double() - dref).abs() <= 2.0 ** -8 * dref.abs() + 2e-6 * g.double().abs()).all()
    _lib.assert_healthy()


def test_every_argument():
    y = torch.arange(-32768, 32768, device=DEV, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)   # all 16-bit floats
    y = y[torch.isfinite(y) & (y.abs() < 1e18)]                # beyond, the gradient's x * x overflows, as it always did
    y = y[: y.numel() // 8 * 8].clone().requires_grad_()
    out = ops.activation(y.view(-1, 8), "gelu")
    out.backward(torch.ones_like(out))
    ref, dref = reference(y.detach(), torch.ones_like(y))
    err, derr = (out.view(-1).double() - ref).abs(), (y.grad.double() - dref).abs()
    # bounds as above; where the gate underflows (an exponential above 2^126, below -10) the result is zero and should be 1e-36
    assert (err <= 2.0 ** -8 * ref.abs() + 1e-14).all() and (derr <= 2.0 ** -8 * dref.abs() + 2e-6).all()
    special = torch.tensor([float("inf"), float("nan"), 0.0, -0.0] * 2, device=DEV, dtype=torch.bfloat16)
    got = ops.activation(special.view(1, 8), "gelu")[0].tolist()
    assert got[0] == float("inf") and got[1] != got[1] and got[2] == 0.0 and got[3] == 0.0
    _lib.assert_healthy()


@pytest.mark.parametrize("kind", ["gelu", "geglu"])
def test_gradient_of_the_largest_arguments(kind):
    """The gradient is that of a step, 0 below and 1 above, up to where 0.107 x * x overflows."""
    y = torch.arange(-32768, 32768, device=DEV, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    y = y[(y.double().abs() >= 1e18) & (y.double().abs() <= (3.4e38 / 0.10704) ** 0.5)]
    y = y[: y.numel() // 8 * 8].view(-1, 8)
    x = (torch.cat([y, torch.ones_like(y)], 1) if kind == "geglu" else y.clone()).requires_grad_()
    out = ops.activation(x, kind)
    out.backward(torch.ones_like(out))
    assert torch.equal(x.grad[:, :8], (y > 0).to(y.dtype)) and torch.equal(out, torch.where(y > 0, y, torch.zeros_like(y)))
    _lib.assert_healthy()
