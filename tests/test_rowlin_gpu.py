"""Linear layers of a few fp32 rows with bf16 weights (csrc/rowlin.cu) against fp64."""
import pytest
import torch
import torch.nn.functional as F

from teletron_b200 import ops
from teletron_b200.ops import _lib

pytestmark = pytest.mark.gpu


def _err(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("B", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("N,K", [(1, 8), (17, 256), (150, 2056), (9216, 1536), (37, 5120)])
@pytest.mark.parametrize("bias,main", [(True, False), (False, True)])
def test_row_linear(B, N, K, bias, main):
    torch.manual_seed(0)
    x = torch.randn(B, K, device="cuda", requires_grad=True)
    w = torch.nn.Parameter((torch.randn(N, K, device="cuda") / K ** 0.5).bfloat16())
    b = torch.nn.Parameter(torch.randn(N, device="cuda").bfloat16()) if bias else None
    if main:
        w.main_grad = torch.randn(N, K, device="cuda")
        start = w.main_grad.double()
    dy = torch.randn(B, N, device="cuda")
    before = _lib.launch_count()
    y = ops.row_linear(x, w, b)
    y.backward(dy)
    assert (_lib.launch_count() > before) == (B <= 4)          # more rows go to the library
    xd, wd = x.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    yd = F.linear(xd, wd, None if b is None else b.detach().double())
    yd.backward(dy.double())
    # fp32 sums over K or N in another order; a bf16 gradient is rounded once, by at most half of
    # its last place (2^-8 of the value), which bounds the norm of the error however few elements there are
    assert y.dtype == torch.float32 and _err(y, yd) < 2e-6 and _err(x.grad, xd.grad) < 2e-6
    if main and B <= 4:
        assert w.grad is None and w.grad_written and _err(w.main_grad - start, wd.grad) < 1e-5
    else:
        assert _err(w.grad, wd.grad) < 2 ** -8
    if bias:
        assert _err(b.grad, dy.double().sum(0)) < 2 ** -8
