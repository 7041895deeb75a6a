"""The native VAE beyond single kernels: attention (csrc/softmax.cu around two GEMMs: fp32 probabilities, any number of
pixels) and the memory of its default chunks."""
import pytest
import torch

from teletron_b200.models.encoders import WanVideoVAE, wan_vae, wan_vae_native
from teletron_b200.ops import conv as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n", [(3, 1), (5, 8), (64, 1023), (7, 6240)])
def test_three_parts_are_the_fp32_probability(rows, n):
    torch.manual_seed(0)
    padded = -(-n // 8) * 8
    s = torch.randn(rows, padded, device="cuda") * 4
    s[:, n:] = float("nan")                                   # not read
    p = C.softmax_split(s, n, 3).view(rows, 3, padded).double().sum(1)
    ref = torch.softmax(s[:, :n].double(), dim=1)
    assert (p[:, n:] == 0).all()
    # fp32 exponential, sum and product: a few times 2^-24; two parts leave 2^-18
    assert torch.equal(p, p.float().double())
    assert ((p[:, :n] - ref).norm() / ref.norm()).item() < 2 ** -21


@pytest.mark.parametrize("h,w", [(8, 16), (24, 40)])
def test_attention_multiplies_fp32_probabilities(monkeypatch, h, w):
    """The operands of the product with the values: all 24 bits of every probability."""
    torch.manual_seed(1)
    n, c, seen = h * w, 64, []
    m = wan_vae.AttentionBlock(c).to("cuda", torch.bfloat16).requires_grad_(False)
    gemm = wan_vae_native.ops.gemm

    def spy(a, b, **kw):
        if kw.get("b_mn"):
            seen.append((a, b))
        return gemm(a, b, **kw)

    monkeypatch.setattr(wan_vae_native.ops, "gemm", spy)
    x = torch.randn(c, 1, h, w, device="cuda").to(torch.bfloat16)
    wan_vae_native.Run().attention(m, C.from_planar(x))
    p, v = seen[0]
    parts = p.shape[1] // n
    prob = p.view(n, parts, n).double().sum(1)
    assert torch.equal(v, v[:n].repeat(parts, 1)) and ((prob.sum(1) - 1).abs() < 2 ** -20).all()
    assert parts == 3 and torch.equal(prob, prob.float().double())


@pytest.mark.parametrize("t,h,w,scores", [(1, 192, 193, None), (2, 30, 53, 1 << 19), (1, 17, 16, 1)])
def test_query_rows_in_blocks(monkeypatch, t, h, w, scores):
    """Frames whose scores exceed what is held at a time (the first by its real size), against fp64."""
    torch.manual_seed(2)
    if scores is not None:
        monkeypatch.setattr(wan_vae_native, "SCORES", scores)
    m = wan_vae.AttentionBlock(64)
    torch.nn.init.normal_(m.proj.weight, std=0.1)
    m = m.to("cuda", torch.bfloat16).requires_grad_(False)
    x = torch.randn(64, t, h, w, device="cuda").to(torch.bfloat16)
    xb = C.from_planar(x)
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_allocated()
    out = C.to_planar(wan_vae_native.Run().attention(m, xb))
    assert torch.cuda.max_memory_allocated() - held < 3 * 2 ** 30
    old = m(x[None])[0]
    m, ref = m.double(), torch.empty(64, t, h, w, device="cuda", dtype=torch.float64)
    for f in range(t):
        ref[:, f:f + 1] = m(x[None, :, f:f + 1].double())[0]
    e_new, e_old = (((a.double() - ref).norm() / ref.norm()).item() for a in (out, old))
    assert e_new <= e_old * 1.05 + 1e-5, (e_new, e_old)


@pytest.mark.parametrize("decoder", [False, True])
def test_default_chunks_need_no_more_memory_than_the_modules(monkeypatch, decoder):
    torch.manual_seed(3)
    vae = WanVideoVAE().to("cuda", torch.float32 if decoder else torch.bfloat16).eval()
    x = torch.randn(1, 16, 10, 68, 68, device="cuda") if decoder else torch.rand(1, 3, 37, 544, 544, device="cuda").bfloat16()

    def peak():
        torch.cuda.empty_cache()
        torch.cuda.reset_peak_memory_stats()
        held = torch.cuda.memory_allocated()
        (vae.decode if decoder else vae.encode)(x)
        return (torch.cuda.max_memory_allocated() - held) / 2 ** 30

    native = peak()
    monkeypatch.setattr(wan_vae, "open_run", lambda net, t: None)
    modules = peak()
    assert native < modules + 0.2, (native, modules)


def test_default_chunks():
    f = WanVideoVAE._default_chunk
    assert [f(False, d, 480, 832, 2) for d in (False, True)] == [4, 1]
    assert [f(True, d, 512, 512, 2) for d in (False, True)] == [16, 4]
    assert [f(True, d, 512, 520, 2) for d in (False, True)] == [8, 2]
    assert f(True, True, 240, 416, 4) == 4 and f(True, True, 480, 832, 4) == 2
