"""What has to keep working where native calls stand in for chains of torch operators."""
import pytest
import torch
import torch.autograd.forward_ad as fwd
import torch.nn.functional as F
from torch.utils.flop_counter import FlopCounterMode

from teletron_b200 import ops
from teletron_b200.models import WanModel, wan, wan_config
from teletron_b200.models.encoders import UMT5Encoder, WanVideoVAE, wan_vae_native
from teletron_b200.models.hunyuan import HunyuanVideoModel, hunyuan_config
from teletron_b200.ops import _lib

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _vae(dtype=torch.float32):
    torch.manual_seed(0)
    return WanVideoVAE(dim=16).to("cuda", dtype).eval()


def _t5():
    torch.manual_seed(0)
    enc = UMT5Encoder(vocab=50, dim=64, dim_attn=64, dim_ffn=128, num_heads=4, num_layers=1)
    return enc.to("cuda", BF16).eval().requires_grad_(False), torch.randint(1, 50, (1, 8), device="cuda")


def _wan():
    torch.manual_seed(0)
    cfg = wan_config("wan2.1-1.3b-t2v", dim=256, num_heads=2, num_layers=1, ffn_dim=640)
    with torch.device("cuda"):
        m = WanModel(cfg).to(BF16).eval()
    x = torch.randn(24, 256, device="cuda", dtype=BF16)
    return m.blocks[0], (x, torch.randn(1, 16, 256, device="cuda", dtype=BF16), torch.randn(1, 6, 256, device="cuda"),
                         torch.randn(24, 64, 2, device="cuda"), 1, None)


def _single():
    torch.manual_seed(0)
    cfg = hunyuan_config("hunyuan-tiny", num_layers=1, num_single_layers=1)
    with torch.device("cuda"):
        m = HunyuanVideoModel(cfg).to(BF16).eval()
    x = torch.randn(24, cfg.hidden_size, device="cuda", dtype=BF16)
    return m.single_transformer_blocks[0], (x, 16, torch.randn(1, cfg.hidden_size, device="cuda"),
                                            torch.randn(16, 64, 2, device="cuda"), 1, None)


@torch.no_grad()
def _routes():
    """The five routes' answers: whether each would run natively now."""
    vae, (enc, ids), (blk, args), (single, sargs) = _vae(), _t5(), _wan(), _single()
    before = _lib.launch_count()
    ops.row_linear(torch.randn(1, 64, device="cuda"), torch.randn(8, 64, device="cuda").to(BF16))
    rows = _lib.launch_count() > before
    return [wan_vae_native.usable(vae.model.encoder, torch.randn(1, 3, 1, 16, 16, device="cuda")), enc._native(ids, None),
            wan.wan_block_infer(blk, *args) is not None, single.packs(*sargs), rows]


def test_routes_are_native():
    assert all(_routes())


def test_forward_mode():
    with fwd.dual_level():
        assert not any(_routes())
        vae = _vae()
        x, dx = (torch.randn(3, 1, 16, 16, device="cuda") for _ in range(2))
        z = fwd.unpack_dual(vae.encode([fwd.make_dual(x, dx)])).tangent
        h, x, dx, vae = 1e-4, x.double(), dx.double(), vae.double()
        num = (vae.encode([x + h * dx]) - vae.encode([x - h * dx])) / (2 * h)
        # TF32 products (2^-11 each way) through about twenty layers
        assert z is not None and ((z[0] - num[0]).norm() / num.norm()).item() < 0.02
        w = torch.randn(8, 64, device="cuda").to(BF16)
        x, dx = (torch.randn(2, 64, device="cuda") for _ in range(2))
        y = fwd.unpack_dual(ops.row_linear(fwd.make_dual(x, dx), w)).tangent
        torch.testing.assert_close(y, F.linear(dx, w.float()))


def test_vmap_and_operator_counts():
    w, x = torch.randn(8, 64, device="cuda").to(BF16), torch.randn(3, 1, 64, device="cuda")
    y = torch.func.vmap(lambda r: ops.row_linear(r, w))(x)
    torch.testing.assert_close(y, F.linear(x, w.float()))
    vae = _vae(BF16)
    with FlopCounterMode(display=False) as count:
        vae.encode([torch.randn(3, 1, 16, 16, device="cuda", dtype=BF16)])
    # a 16 x 16 frame through the first residual block alone: two 3 x 3 x 3 convolutions of 16 channels
    assert count.get_total_flops() > 2 * 2 * 256 * 16 * 16 * 27


def test_another_device_is_current(monkeypatch):
    """Kernels are launched on the current device: tensors of another one take the torch operators."""
    dev = torch.cuda.current_device
    monkeypatch.setattr(torch.cuda, "current_device", lambda: dev() + 1)
    vae, (enc, ids), (blk, args), (single, sargs) = _vae(), _t5(), _wan(), _single()
    with torch.no_grad():
        assert wan.wan_block_infer(blk, *args) is None and not single.packs(*sargs) and not enc._native(ids, None)
        assert not wan_vae_native.usable(vae.model.encoder, torch.randn(1, 3, 1, 16, 16, device="cuda"))


@pytest.mark.parametrize("dtype", [BF16, torch.float32])
def test_vae_with_parameters_in_one_flat_buffer(dtype):
    """Views that start anywhere: the same bits as parameters of their own."""
    vae = _vae(dtype)
    x = torch.randn(3, 1, 24, 40, device="cuda").to(dtype)
    ref = vae.encode([x])
    flat, at = torch.empty(1 + sum(p.numel() for p in vae.parameters()), device="cuda", dtype=dtype), 1
    for p in vae.parameters():
        p.data = flat[at:at + p.numel()].copy_(p.data.reshape(-1)).view(p.shape)
        at += p.numel()
    assert any(p.data_ptr() % 16 for p in vae.parameters())
    assert wan_vae_native.usable(vae.model.encoder, x[None]) and torch.equal(vae.encode([x]), ref)


def test_row_linear_of_a_slice():
    """A contiguous row that does not start on 16 bytes, forward and backward."""
    torch.manual_seed(1)
    t = torch.randn(1, 257, device="cuda", requires_grad=True)
    w = torch.nn.Parameter(torch.randn(24, 256, device="cuda").to(BF16))
    x = t[:, 1:]
    assert x.is_contiguous() and x.data_ptr() % 16
    y = ops.row_linear(x, w)
    y.backward(torch.ones_like(y))
    torch.testing.assert_close(y, F.linear(x, w.float()), rtol=1e-5, atol=1e-4)
    torch.testing.assert_close(t.grad[:, 1:], w.float().sum(0, keepdim=True), rtol=1e-5, atol=1e-4)
    torch.testing.assert_close(w.grad, x.detach().to(BF16).expand(24, -1))


def test_row_linear_second_derivatives():
    torch.manual_seed(2)
    x = torch.randn(2, 64, device="cuda", requires_grad=True)
    w = torch.nn.Parameter(torch.randn(8, 64, device="cuda").to(BF16))
    b = torch.nn.Parameter(torch.randn(8, device="cuda").to(BF16))

    def penalty(f):
        gx, gw, gb = torch.autograd.grad(f().square().sum(), [x, w, b], create_graph=True)
        return torch.autograd.grad(gx.square().sum() + gw.float().square().sum() + gb.float().sum(), [x, w, b])

    got = penalty(lambda: ops.row_linear(x, w, b))
    for g, r in zip(got, penalty(lambda: F.linear(x, w.float(), b.float()))):
        torch.testing.assert_close(g, r, rtol=1e-2, atol=1e-2 * r.abs().max().item())   # bf16 gradients


def test_row_linear_refuses_what_linear_refuses():
    """A bias of another length or device is an error; no weights is an empty result."""
    x, w = torch.randn(2, 64, device="cuda"), torch.randn(8, 64, device="cuda").to(BF16)
    for b in (torch.zeros(5, device="cuda", dtype=BF16), torch.zeros(8, dtype=BF16)):
        with pytest.raises(RuntimeError):
            ops.row_linear(x, w, b)
    assert ops.row_linear(x, w[:0]).shape == (2, 0)
    # a bias that broadcasts, as F.linear has it
    b = torch.ones(1, device="cuda", dtype=BF16)
    torch.testing.assert_close(ops.row_linear(x, w, b), F.linear(x, w.float(), b.float()))


def test_block_call_looks_at_the_shapes():
    """Parameters that do not fit the block go to the op layer, which refuses them."""
    blk, args = _wan()
    with torch.no_grad():
        assert wan.wan_block_infer(blk, *args) is not None
        for mod, name in ((blk, "modulation"), (blk.self_attn.qkv, "bias"), (blk.ffn[2], "weight"), (blk.cross_attn.norm_k, "weight")):
            old = getattr(mod, name)
            setattr(mod, name, torch.nn.Parameter(old.data[..., :-8].contiguous()))
            assert wan.wan_block_infer(blk, *args) is None
            setattr(mod, name, old)
        assert wan.wan_block_infer(blk, args[0][:, :-8], *args[1:]) is None
        assert wan.wan_block_infer(blk, *args) is not None


def test_block_call_leaves_an_empty_context_to_the_op_layer():
    blk, args = _wan()
    with torch.no_grad():
        assert wan.wan_block_infer(blk, args[0], args[1][:, :0], *args[2:]) is None


class _Lora(torch.nn.Module):
    """A wrapper in the manner of low-rank adapters: shows its base layer's weight and computes something else."""

    def __init__(self, base):
        super().__init__()
        self.base = base

    weight = property(lambda self: self.base.weight)
    bias = property(lambda self: self.base.bias)

    def forward(self, x, **kw):
        return self.base(x, **kw) * 2


def test_modules_put_in_the_place_of_others():
    """Wrapped layers, instance-level forwards and other epsilons are computed, not skipped."""
    blk, args = _wan()
    single, sargs = _single()
    vae, (enc, ids) = _vae(BF16), _t5()
    x = torch.randn(3, 1, 16, 16, device="cuda", dtype=BF16)

    def single_out():
        from teletron_b200.models.hunyuan import _PairBlock

        return _PairBlock(single)(sargs[0], sargs[1], sargs[2], sargs[3], 1, None, None)

    calls = [(lambda: blk(*args), blk.self_attn, "qkv"), (lambda: blk(*args), blk.cross_attn, "kv"),
             (single_out, single, "proj_mlp"), (lambda: vae.encode([x]), vae.model.encoder.middle[0].residual, "2"),
             (lambda: enc(ids), enc.blocks[0], "norm1")]
    with torch.no_grad():
        for f, owner, name in calls:
            ref, old = f(), owner._modules[name]
            owner._modules[name] = _Lora(old)
            assert not torch.equal(f(), ref), name
            owner._modules[name] = old
            own = old.forward
            old.forward = lambda *a, **kw: own(*a, **kw) * 2
            assert not torch.equal(f(), ref), name
            del old.forward
            assert torch.equal(f(), ref)
        blk.self_attn.eps = 0.5
        assert wan.wan_block_infer(blk, *args) is None
