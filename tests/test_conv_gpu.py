"""VAE convolution kernels (csrc/conv.cu) and the native encoder / decoder against torch in 64 bits."""
import pytest
import torch
import torch.nn.functional as F

from teletron_b200.models.encoders import WanVideoVAE, wan_vae, wan_vae_native
from teletron_b200.ops import _lib
from teletron_b200.ops import conv as C

pytestmark = pytest.mark.gpu

# relative 2-norm errors: bf16 output rounding is 2^-9 uniform, about 1.7e-3; TF32 operands rounded to nearest carry
# 2^-12 uniform each, about 2e-4 for a sum of products
TOL = {torch.bfloat16: 2.5e-3, torch.float32: 5e-4}
DTYPES = [torch.bfloat16, torch.float32]


def _close(y, ref, dtype):
    err = ((y.double() - ref).norm() / ref.norm()).item()
    assert err < TOL[dtype], err


def _rand(*shape, dtype, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("ci,co,t,h,w", [(96, 96, 3, 16, 16), (96, 192, 2, 33, 21), (384, 384, 2, 15, 52), (16, 384, 2, 9, 11),
                                         (3, 96, 5, 17, 33), (96, 3, 3, 18, 40), (192, 384, 1, 1, 3), (32, 16, 3, 16, 50)])
def test_causal_conv(dtype, ci, co, t, h, w):
    torch.manual_seed(0)
    x, k, b = _rand(ci, t, h, w, dtype=dtype), _rand(co, ci, 3, 3, 3, dtype=dtype, scale=(27 * ci) ** -0.5), _rand(co, dtype=dtype)
    ref = F.conv3d(F.pad(x.double()[None], (1, 1, 1, 1, 2, 0)), k.double(), b.double())[0]
    xb, pk = C.from_planar(x, True), C.PackedConv(k, b, C.CONV_SPATIAL, (t, h, w) if w % 2 else (t, 480, 832))
    if co % 16:
        y = C.conv(xb, pk, t, (h, w), t_off=-2, planar=True)
    else:
        res = _rand(co, t, h, w, dtype=dtype)
        y = C.to_planar(C.conv(xb, pk, t, (h, w), t_off=-2, res=C.from_planar(res)))
        ref = ref + res.double()
        if t > 2:   # history frames in front instead of zeros
            _close(C.to_planar(C.conv(xb, pk, t - 2, (h, w), res=C.from_planar(res[:, 2:]))), ref[:, 2:], dtype)
    _close(y, ref, dtype)
    _lib.check_status()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("h,w", [(21, 30), (20, 33), (32, 32), (2, 2)])
def test_resampling_convs(dtype, h, w):
    torch.manual_seed(1)
    c, t = 192, 3
    x, b = _rand(c, t, h, w, dtype=dtype), _rand(c, dtype=dtype)
    xb, xd = C.from_planar(x, True), x.double()
    k = _rand(c, c, 3, 3, dtype=dtype, scale=(9 * c) ** -0.5)
    ref = F.conv2d(F.pad(xd.transpose(0, 1), (0, 1, 0, 1)), k.double(), b.double(), stride=2).transpose(0, 1)
    _close(C.to_planar(C.conv(C.phases2(xb), C.PackedConv(k, b, C.CONV_STRIDE2, (t, h // 2, w // 2)), t, (h // 2, w // 2))), ref, dtype)
    ref = F.conv2d(F.interpolate(xd.transpose(0, 1), scale_factor=2.0, mode="nearest-exact"), k.double(), b.double(), padding=1)
    _close(C.to_planar(C.conv(C.enlarge2(xb), C.PackedConv(k, b, C.CONV_SPATIAL, (t, 2 * h, 2 * w)), t, (2 * h, 2 * w))), ref.transpose(0, 1), dtype)
    k, b2 = _rand(2 * c, c, 3, 1, 1, dtype=dtype, scale=(3 * c) ** -0.5), _rand(2 * c, dtype=dtype)
    ref = F.conv3d(F.pad(xd[None], (0, 0, 0, 0, 2, 0)), k.double(), b2.double())[0].reshape(2, c, t, h, w)
    y = C.conv(xb, C.PackedConv(k, b2, C.CONV_POINT, (t, h, w)), t, (h, w), t_off=-2, t_mul=2)
    _close(C.to_planar(y), ref.permute(1, 2, 0, 3, 4).reshape(c, 2 * t, h, w), dtype)
    k = _rand(c, c, 3, 1, 1, dtype=dtype, scale=(3 * c) ** -0.5)
    ref = F.conv3d(xd[None], k.double(), b.double(), stride=(2, 1, 1))[0]
    _close(C.to_planar(C.conv(xb, C.PackedConv(k, b, C.CONV_POINT, (1, h, w)), 1, (h, w), t_stride=2)), ref, dtype)
    _lib.check_status()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("c", [16, 96, 192, 384])
def test_chan_norm(dtype, c):
    torch.manual_seed(2)
    x, g = _rand(c, 2, 13, 11, dtype=dtype), (torch.rand(c, device="cuda") + 0.5).to(dtype)
    x[:, 0, 0, 0] = 0                                         # a pixel without a direction
    xb = C.from_planar(x)
    y = C.to_planar(C.chan_norm(xb, g, torch.empty_like(xb)))
    ref = F.silu(F.normalize(x.double(), dim=0) * c ** 0.5 * g.double().view(-1, 1, 1, 1))
    _close(y, ref, dtype)
    x[3, 1, 2, 2] = float("nan")                              # spreads over its pixel, and no further
    xb = C.from_planar(x)
    bad = C.to_planar(C.chan_norm(xb, g, torch.empty_like(xb))).isnan()
    assert bad[:, 1, 2, 2].all() and bad.sum() == c


@pytest.mark.parametrize("rows,n", [(3, 1), (5, 8), (64, 1023), (7, 6240), (2, 1032)])
def test_softmax_split(rows, n):
    torch.manual_seed(4)
    padded = -(-n // 8) * 8
    s = torch.randn(rows, padded, device="cuda") * 4
    s[:, n:] = float("nan")                                   # not read
    s[0, 0] = -float("inf") if n > 1 else 0.0
    p = C.softmax_split(s, n)
    ref = torch.softmax(s[:, :n].double(), dim=1)
    got = p[:, :padded].double() + p[:, padded:].double()
    assert (got[:, n:] == 0).all()
    # two bf16 parts: 2^-17 of the value
    assert ((got[:, :n] - ref).norm() / ref.norm()).item() < 2 ** -16


@pytest.mark.parametrize("t,h,w", [(2, 5, 7), (1, 30, 53), (1, 2, 2)])
def test_frame_attention(t, h, w):
    """Against fp64; the error may not exceed the library path's."""
    torch.manual_seed(5)
    m = wan_vae.AttentionBlock(384)
    torch.nn.init.normal_(m.proj.weight, std=0.05)
    m = m.to("cuda", torch.bfloat16).requires_grad_(False)
    x = _rand(384, t, h, w, dtype=torch.bfloat16)
    out = C.to_planar(wan_vae_native.Run().attention(m, C.from_planar(x)))
    old = m(x[None])[0]
    ref = m.double()(x.double()[None])[0]
    e_new, e_old = (((a.double() - ref).norm() / ref.norm()).item() for a in (out, old))
    assert e_new <= e_old * 1.05 + 1e-5, (e_new, e_old)
    _lib.check_status()


def _vae(dtype, dim):
    torch.manual_seed(3)
    vae = WanVideoVAE(dim=dim)
    for m in (vae.model.encoder.middle[1], vae.model.decoder.middle[1]):
        torch.nn.init.normal_(m.proj.weight, std=0.02)
    return vae.to("cuda", dtype).eval()


@pytest.mark.parametrize("dim,frames,h,w", [(96, 1, 16, 16), (16, 9, 40, 56), (96, 5, 24, 72), (16, 37, 33, 18)])
def test_native_encoder_matches_modules(monkeypatch, dim, frames, h, w):
    """Whole clips and chunks, against the module chain in fp64; the error may not exceed the module chain's own."""
    vae = _vae(torch.bfloat16, dim)
    x = _rand(3, frames, h, w, dtype=torch.bfloat16).clamp(-1, 1)
    before = _lib.launch_count()
    z = vae.encode([x])
    assert _lib.launch_count() > before
    monkeypatch.setattr(wan_vae, "open_run", lambda net, t: None)
    old = vae.encode([x])
    ref = vae.double().encode([x.double()])
    assert z.shape == ref.shape and z.dtype == torch.bfloat16

    def err(a):
        return ((a.double() - ref).norm() / ref.norm()).item()

    assert err(z) < 1.2 * err(old) + 1e-3, (err(z), err(old))
    _lib.check_status()


@pytest.mark.parametrize("dim,frames,h,w,tiled", [(16, 3, 5, 7, False), (96, 2, 4, 6, False), (16, 10, 6, 9, False), (16, 2, 9, 8, True)])
def test_native_decoder_matches_modules(monkeypatch, dim, frames, h, w, tiled):
    vae = _vae(torch.float32, dim)
    z = _rand(1, 16, frames, h, w, dtype=torch.float32)
    kw = dict(tiled=tiled, tile_size=(6, 5), tile_stride=(3, 3))
    before = _lib.launch_count()
    v = vae.decode(z, **kw)
    assert _lib.launch_count() > before
    monkeypatch.setattr(wan_vae, "open_run", lambda net, t: None)
    old = vae.decode(z, **kw)
    ref = None
    with monkeypatch.context() as mp:      # the enlargement layers cast to fp32: keep them in fp64 for the oracle
        mp.setattr(torch.Tensor, "float", lambda t: t.double())
        ref = vae.double().decode(z.double(), **kw)

    def err(a):
        return ((a.double() - ref).norm() / ref.norm()).item()

    assert v.shape == ref.shape and v.dtype == torch.float32
    assert err(v) < 1.2 * err(old) + 1e-4, (err(v), err(old))
    _lib.check_status()


def test_route_to_the_modules():
    """What the native path does not take: gradients, hooks, fp32 without TF32, fp16, batches."""
    vae = _vae(torch.float32, 16)
    x = torch.randn(1, 3, 1, 16, 16, device="cuda")
    net = vae.model.encoder
    assert wan_vae_native.usable(net, x)
    assert not wan_vae_native.usable(net, x.cpu()) and not wan_vae_native.usable(net, x.half())
    assert not wan_vae_native.usable(net, x.expand(2, -1, -1, -1, -1))
    assert not wan_vae_native.usable(net, x.clone().requires_grad_())
    old = torch.backends.cudnn.allow_tf32
    try:
        torch.backends.cudnn.allow_tf32 = False
        assert not wan_vae_native.usable(net, x)
    finally:
        torch.backends.cudnn.allow_tf32 = old
    old = torch.backends.cudnn.conv.fp32_precision
    try:
        torch.backends.cudnn.conv.fp32_precision = "ieee"
        assert not wan_vae_native.usable(net, x)
    finally:
        torch.backends.cudnn.conv.fp32_precision = old
    handle = net.conv1.register_forward_hook(lambda *a: None)
    assert not wan_vae_native.usable(net, x)
    handle.remove()
    assert wan_vae_native.usable(net, x)
