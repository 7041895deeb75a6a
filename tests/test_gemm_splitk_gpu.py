"""Split-K GEMM (csrc/gemm_splitk.cu): layouts, ragged edges and epilogues against the fp32 statement."""
import importlib
import math

import pytest
import torch

from teletron_b200.ops import _lib

G = importlib.import_module("teletron_b200.ops.gemm")
pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 1), (1, 0)])
@pytest.mark.parametrize("M,N,K", [(256, 1536, 1536), (256, 1536, 8960), (1, 72, 512), (130, 136, 1032), (512, 264, 5000)])
def test_splitk_layouts(a_mn, b_mn, M, N, K):
    torch.manual_seed(1)
    M += (-M) % 8 if a_mn else 0
    a = torch.randn((K, M) if a_mn else (M, K), device="cuda", dtype=BF16)
    b = torch.randn((K, N) if b_mn else (N, K), device="cuda", dtype=BF16)
    bias = torch.randn(N, device="cuda", dtype=BF16)
    kw = dict(a_mn=bool(a_mn), b_mn=bool(b_mn), bias=bias, alpha=1 / math.sqrt(K))
    out, ref = G.gemm(a, b, **kw), G.gemm_ref(a, b, out_dtype=torch.float32, **kw)
    # bf16 rounding of the output: 2^-9 uniform is 1.7e-3 of the norm
    assert ((out.float() - ref).norm() / ref.norm()).item() < 2.5e-3
    assert torch.equal(out, G.gemm(a, b, **kw))     # the parts are added in a fixed order
    _lib.check_status()


@pytest.mark.parametrize("epi", [G.EPI_GELU, G.EPI_SILU, G.EPI_GATE_RES, G.EPI_ACCUM])
def test_splitk_epilogues(epi):
    torch.manual_seed(2)
    M, N, K = 260, 392, 2048
    a, b = torch.randn(M, K, device="cuda", dtype=BF16), torch.randn(N, K, device="cuda", dtype=BF16)
    kw = dict(bias=torch.randn(N, device="cuda", dtype=BF16), epi=epi, alpha=1 / math.sqrt(K))
    if epi == G.EPI_GATE_RES:
        kw.update(residual=torch.randn(M, N, device="cuda", dtype=BF16), gate=torch.randn(2, N, device="cuda"), rows_per_gate=130)
    if epi == G.EPI_ACCUM:
        base = torch.randn(M, N, device="cuda")
        out, ref = G.gemm(a, b, out=base.clone(), **kw), G.gemm_ref(a, b, out=base.clone(), **kw)
        # fp32 sums of 2048 products in another order
        assert ((out - ref).norm() / ref.norm()).item() < 1e-4
        return
    (out, aux), (ref, aux_ref) = G.gemm(a, b, want_aux=True, **kw), G.gemm_ref(a, b, want_aux=True, **kw)
    for y, r in ((out, ref), (aux, aux_ref)):
        assert ((y.float() - r.float()).norm() / r.float().norm()).item() < 4e-3   # two bf16 roundings
