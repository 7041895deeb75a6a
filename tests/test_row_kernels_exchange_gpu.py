"""Row kernels in the forms that the context-parallel exchanges use, on one GPU: the scattering store with local buffers
for peers (the kernels only store, they wait for nobody), and the backward pass in place on column blocks."""
import importlib
from types import SimpleNamespace

import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from teletron_b200.ops import _lib
from teletron_b200.parallel.fused_ulysses import _scatter_rows

N = importlib.import_module("teletron_b200.ops.norm")
pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _inputs(rows, C, per_head, freq_rows):
    torch.manual_seed(0)
    x = torch.randn(rows, 3 * C, device="cuda", dtype=BF16)[:, C:2 * C]          # a column block
    w = torch.rand(128 if per_head else C, device="cuda") + 0.5
    ang = torch.randn(freq_rows, 64, device="cuda")
    return x, w, torch.stack([ang.cos(), ang.sin()], -1).contiguous()


@pytest.mark.parametrize("C", [256, 384, 1536, 1920, 2304, 3072, 4096, 5120, 6144])
@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("B,S_l,extra", [(1, 37, 0), (2, 300, 24)])
def test_scattered_rows_equal_the_plain_store(C, per_head, B, S_l, extra):
    D, world, H = 128, 2, C // 128
    Hl, S_pad = (H + 1) // 2, 2 * S_l
    x, w, fr = _inputs(B * S_l, C, per_head, S_l)
    y, rstd = N.rmsrope_fwd_raw(x, w, fr, D, per_head)
    for rank in range(world):
        peers = [torch.zeros(B, S_pad + extra, Hl, D, device="cuda", dtype=BF16) for _ in range(world)]
        fu = SimpleNamespace(world=world, rank=rank)
        got = torch.empty_like(rstd)
        _scatter_rows(fu, x, w, fr, got, B * S_l, C, D, 1e-6, (_lib.c_ll * world)(*[p.data_ptr() for p in peers]), S_l, S_pad,
                      per_head=per_head, dst_rows=S_pad + extra if extra else 0)
        assert torch.equal(got, rstd)
        want = y.view(B, S_l, H, D)
        for p, peer in enumerate(peers):
            mine = want[:, :, p * Hl:(p + 1) * Hl]
            at = peer[:, rank * S_l:(rank + 1) * S_l]
            assert torch.equal(at[:, :, :mine.shape[2]], mine) and (at[:, :, mine.shape[2]:] == 0).all()
            at.zero_()
            assert (peer == 0).all()                                            # nothing outside the rank's rows
    _lib.check_status()


@pytest.mark.parametrize("C", [256, 1536, 2304, 3072, 5120])
@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("rows", [3, 1201])
def test_backward_in_place(C, per_head, rows):
    x, w, fr = _inputs(rows, C, per_head, 400)
    _, rstd = N.rmsrope_fwd_raw(x, w, fr, 128, per_head)
    d = torch.randn(rows, 3 * C, device="cuda", dtype=BF16)
    dx, dw = N.rmsrope_bwd_raw(d[:, C:2 * C].clone(), x, w, fr, rstd, 128, per_head)
    ref = d.clone()
    ref[:, C:2 * C] = dx
    _, dw2 = N.rmsrope_bwd_raw(d[:, C:2 * C], x, w, fr, rstd, 128, per_head, out=d[:, C:2 * C])
    assert torch.equal(d, ref) and torch.equal(dw2, dw)


@pytest.mark.parametrize("C", [256, 2048, 2304, 3072, 4096, 5120, 6144])
@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("rows", [1535, 1536])
def test_forward_on_both_sides_of_the_line(C, per_head, rows):
    """Few rows take a CTA each, many a warp each, which needs their count more than their width."""
    x, w, fr = _inputs(rows, C, per_head, 400)
    y, rstd = N.rmsrope_fwd_raw(x, w, fr, 128, per_head)
    ref = N.rmsnorm_rope_ref(x.float(), w, fr, 128, per_head)
    heads = x.double().view(rows, -1, 128 if per_head else C)
    rstd_ref = torch.rsqrt(heads.pow(2).mean(-1) + 1e-6).view(-1)
    # one bf16 rounding: 1.7e-3 of the norm; fp32 sums
    assert ((y.float() - ref).norm() / ref.norm()).item() < 2.5e-3
    torch.testing.assert_close(rstd.double(), rstd_ref, rtol=2e-6, atol=0)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        N.rmsrope_fwd_raw(x, w, fr, 128, per_head)
        torch.cuda.synchronize()
    warp = any("rmsrope_fwd_warp" in e.key for e in prof.key_averages())
    assert warp == ((rows >= 1536 and C != 2048) if per_head else (rows >= 1536 or C <= 2048))


@pytest.mark.parametrize("C", [8, 1024, 1032, 1536, 1544, 2048, 2056])
@pytest.mark.parametrize("rows,residual", [(1, True), (5, False), (1300, True)])
def test_adaln_backward_on_both_sides_of_the_lines(C, rows, residual):
    """Widths around each change of the number of threads and of what is kept in registers."""
    torch.manual_seed(2)
    x, dy, dr = (torch.randn(rows, C, device="cuda", dtype=BF16) for _ in range(3))
    e = torch.randn(1, 2, C, device="cuda")
    xg, eg = x.clone().requires_grad_(), e.clone().requires_grad_()
    y, xr = N.adaln_res(xg, eg[:, 1], eg[:, 0], rows)
    dx, de = torch.autograd.grad([y, xr] if residual else [y], [xg, eg], [dy, dr] if residual else [dy])
    xd, ed = x.double().requires_grad_(), e.double().requires_grad_()
    yd = torch.nn.functional.layer_norm(xd, (C,), eps=1e-6) * (1 + ed[:, 1]) + ed[:, 0]
    dxd, ded = torch.autograd.grad([yd, xd * 1.0] if residual else [yd], [xd, ed], [dy.double(), dr.double()] if residual else [dy.double()])
    # one bf16 rounding of the output (1.7e-3 of the norm, at most 2^-8); the column sums stay in fp32
    assert ((dx.double() - dxd).norm() / dxd.norm()).item() < (2.5e-3 if rows * C > 1000 else 2 ** -8)
    assert ((de.double() - ded).norm() / ded.norm()).item() < 1e-5
