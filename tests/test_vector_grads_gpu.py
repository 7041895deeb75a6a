"""Gradients of biases, norm weights and small projections that kernels add to the fp32 buffer, and what has to stay an
ordinary autograd gradient."""
import pytest
import torch

from teletron_b200 import ops
from teletron_b200.models import WanModel, wan_config
from teletron_b200.parallel.ddp import ParamBuffer

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _err(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def _vec(n):
    p = torch.nn.Parameter((torch.rand(n, device="cuda") + 0.5).to(BF16))
    p.main_grad = torch.randn(n, device="cuda")
    return p


def _op(kind, x, w, b, n):
    """(output, fp64 output) of one op with a vector parameter b (and n for the norm's weight)."""
    xd, bd, nd, wd = (t.detach().double() for t in (x, b, n, w))
    bd.requires_grad_(), nd.requires_grad_()
    if kind == "linear":
        return ops.linear(x, w, b), xd @ wd.t() + bd, bd, None
    if kind == "residual":
        return ops.linear_residual(x, w, b, x), xd + xd @ wd.t() + bd, bd, None
    if kind == "layernorm":
        ref = torch.nn.functional.layer_norm(xd, (x.shape[1],), nd, bd, 1e-6)
        return ops.layernorm_affine(x, n, b), ref, bd, nd
    y = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * nd
    return ops.rmsnorm_rope(x, n, None, 128), y, None, nd


@pytest.mark.parametrize("kind", ["linear", "residual", "layernorm", "rmsnorm"])
@pytest.mark.parametrize("rows", [1, 37, 1500])
def test_vector_gradients_add_up_in_the_buffer(kind, rows):
    """Two backward passes, a buffer that is not zero: start + the sums in fp64.  fp32 column sums: 1e-5."""
    torch.manual_seed(0)
    C = 256
    x = torch.randn(rows, C, device="cuda", dtype=BF16)
    w = (torch.randn(C, C, device="cuda") / 16).to(BF16)
    b, n = _vec(C), _vec(C)
    start = [p.main_grad.double() for p in (b, n)]
    want = [torch.zeros(C, device="cuda", dtype=torch.float64) for _ in range(2)]
    for _ in range(2):
        dy = torch.randn(rows, C, device="cuda", dtype=BF16)
        y, ref, bd, nd = _op(kind, x, w, b, n)
        y.backward(dy)
        ref.backward(dy.double())
        for acc, t in zip(want, (bd, nd)):
            if t is not None:
                acc += t.grad
    for p, s, acc in zip((b, n), start, want):
        used = acc.norm() > 0
        assert p.grad is None and _err(p.main_grad, s + acc) < 1e-5
        assert hasattr(p, "grad_written") == bool(used)


@pytest.mark.parametrize("kind", ["linear", "residual", "layernorm", "rmsnorm", "rows"])
def test_gradients_that_somebody_reads(kind):
    """Tensor hooks, post-accumulate hooks and ``autograd.grad`` get the gradient, and the buffer stays as it was; the
    gradient of another input leaves the buffer alone."""
    torch.manual_seed(1)
    C = 128
    x = torch.randn(4, C, device="cuda", dtype=BF16).requires_grad_()
    w = (torch.randn(C, C, device="cuda") / 11).to(BF16)
    b, n = _vec(C), _vec(C)
    p = n if kind == "rmsnorm" else b
    if kind == "rows":
        p = torch.nn.Parameter(w)
        p.main_grad = torch.randn(C, C, device="cuda")
        make = lambda: ops.row_linear(x, p)  # noqa: E731
    else:
        make = lambda: _op(kind, x, w, b, n)[0]  # noqa: E731
    others = [t.main_grad.clone() for t in (b, n)]
    start = p.main_grad.clone()
    dy = torch.randn_like(make())
    g, = torch.autograd.grad(make(), [p], dy)
    assert g is not None and g.shape == p.shape and torch.equal(p.main_grad, start)
    torch.autograd.grad(make(), [x], dy)
    assert torch.equal(p.main_grad, start) and all(torch.equal(t.main_grad, o) for t, o in zip((b, n), others))
    seen = []
    handle = p.register_hook(lambda t: seen.append(t))
    make().backward(dy)
    handle.remove()
    assert len(seen) == 1 and seen[0] is not None and torch.equal(seen[0], g) and torch.equal(p.grad, g)
    assert torch.equal(p.main_grad, start)
    p.grad = None
    handle = p.register_post_accumulate_grad_hook(lambda t: seen.append(t.grad))
    make().backward(dy)
    handle.remove()
    assert len(seen) == 2 and torch.equal(seen[1], g) and torch.equal(p.main_grad, start)
    p.grad = None
    make().backward(dy)
    # the same sums without the rounding to bf16: half of its last place
    assert p.grad is None and _err(p.main_grad - start, g.double()) < 2 ** -8


@pytest.mark.parametrize("recompute", [False, True])
def test_model_gradients_equal_the_plain_route(recompute):
    """Every parameter of a Wan model in a ParamBuffer, two micro-batches, one frozen bias, against the gradients of
    the same model outside a buffer."""
    kw = dict(recompute_granularity="full", recompute_method="block", recompute_num_layers=2) if recompute else {}
    cfg = wan_config("wan2.1-1.3b-t2v", dim=256, num_heads=2, num_layers=2, ffn_dim=640, **kw)
    models = []
    for _ in range(2):
        torch.manual_seed(2)
        with torch.device("cuda"):
            m = WanModel(cfg).to(BF16).train()
        m.blocks[0].ffn[0].bias.requires_grad_(False)
        models.append(m)
    plain, m = models
    buf = ParamBuffer(m)
    buf.grads.normal_()
    start = buf.grads.clone()
    ctx = torch.randn(2, 24, cfg.text_dim, device="cuda", dtype=BF16)
    want = {}
    for i in range(2):
        x = torch.randn(2, 16, 1, 12, 16, device="cuda", dtype=BF16)
        t = torch.tensor([200.0, 700.0], device="cuda")
        dy = torch.randn_like(x)
        plain(x, t, ctx).backward(dy)
        m(x, t, ctx).backward(dy)
        for n, p in plain.named_parameters():
            if p.grad is not None:
                want[n] = want.get(n, 0) + p.grad.double()
                p.grad = None
    direct = [n for n, p in m.named_parameters() if p.grad is None and p.requires_grad]
    assert {"blocks.1.norm3.weight", "blocks.1.norm3.bias", "blocks.0.self_attn.norm_q.weight", "blocks.0.self_attn.qkv.bias",
            "blocks.1.cross_attn.norm_k.weight", "blocks.1.ffn.2.bias", "time_embedding.0.weight"} <= set(direct)
    buf.collect_grads()
    assert "blocks.0.ffn.0.bias" not in buf.index and m.blocks[0].ffn[0].bias.grad is None
    for n, p in buf.named:
        o, cnt, shape = buf.index[n]
        got = p.main_grad.double() - start[o:o + cnt].view(shape).double()
        # the plain route rounds each pass' gradient to bf16: half of its last place
        assert _err(got, want[n]) < 2 ** -7, n
