"""That the native block call and the split-K kernel are what runs where the tests of their results assume it."""
import importlib
import math

import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from teletron_b200.models import WanModel, wan, wan_config
from teletron_b200.ops import _lib

G = importlib.import_module("teletron_b200.ops.gemm")
pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("frames,h,w", [(1, 4, 4), (8, 64, 64), (9, 60, 62)])     # below, at and above 8,192 rows
def test_wan_block_call_runs(monkeypatch, frames, h, w):
    torch.manual_seed(0)
    cfg = wan_config("wan2.1-1.3b-t2v", dim=256, num_heads=2, num_layers=2, ffn_dim=640)
    with torch.device("cuda"):
        m = WanModel(cfg).to(BF16).eval()
    x = torch.randn(1, 16, frames, h, w, device="cuda", dtype=BF16)
    ctx, t = torch.randn(1, 40, cfg.text_dim, device="cuda", dtype=BF16), torch.tensor([300.0], device="cuda")
    native, call = [], wan.wan_block_infer

    def spy(*a):
        out = call(*a)
        native.append(out is not None)
        return out

    monkeypatch.setattr(wan, "wan_block_infer", spy)
    ref = m(x, t, ctx).detach()
    assert native == [False, False]
    with torch.no_grad():
        out = m(x, t, ctx)
        assert native[2:] == [True, True] and torch.equal(out, ref)
        handle = m.blocks[0].ffn[0].register_forward_hook(lambda *a: None)
        assert torch.equal(m(x, t, ctx), ref) and native[4:] == [False, True]
        handle.remove()
    _lib.check_status()


def _kernels(fn):
    fn()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = fn()
        torch.cuda.synchronize()
    return out, " ".join(e.key for e in prof.key_averages())


# on 148 SMs: at most 74 tiles of 128 x 128; K of at least 512 from the pair kernel (256 x 256 outputs), 1,024 from the other
@pytest.mark.parametrize("M,N,K,split", [(256, 1536, 8960, True), (128, 136, 1024, True), (2176, 512, 512, True),
                                         (2432, 512, 512, False), (128, 136, 960, False), (256, 264, 448, False),
                                         (512, 512, 5120, True), (256, 64, 2048, False)])
@pytest.mark.parametrize("form", ["null gate", "fp32", "fp32 accumulate"])
def test_splitk_forms(M, N, K, split, form):
    torch.manual_seed(1)
    a, b = torch.randn(M, K, device="cuda", dtype=BF16), torch.randn(N, K, device="cuda", dtype=BF16)
    kw = dict(alpha=1 / math.sqrt(K))
    if form == "null gate":
        kw.update(epi=G.EPI_GATE_RES, residual=torch.randn(M, N, device="cuda", dtype=BF16), gate=None, rows_per_gate=M)
    base = torch.randn(M, N, device="cuda")
    if form == "fp32 accumulate":
        run = lambda: G.gemm(a, b, out=base.clone(), epi=G.EPI_ACCUM, **kw)  # noqa: E731
        ref = G.gemm_ref(a, b, out=base.clone(), epi=G.EPI_ACCUM, **kw)
    else:
        dt = torch.float32 if form == "fp32" else BF16
        run = lambda: G.gemm(a, b, out_dtype=dt, **kw)  # noqa: E731
        ref = G.gemm_ref(a, b, out_dtype=torch.float32, **kw)
    out, names = _kernels(run)
    assert ("gemm_splitk" in names) == (split and torch.cuda.get_device_properties(0).multi_processor_count == 148), names
    # fp32 sums in another order; one bf16 rounding (1.7e-3 of the norm) of a bf16 result
    assert ((out.float() - ref.float()).norm() / ref.float().norm()).item() < (2.5e-3 if form == "null gate" else 1e-4)
    _lib.check_status()
