"""Row kernels (csrc/norm.cu) at every width class, and the multi-tensor gradient fold, against plain torch."""
import importlib

import pytest
import torch

from teletron_b200.ops import _lib

N = importlib.import_module("teletron_b200.ops.norm")
pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
WIDTHS = [128, 1536, 1544, 2048, 2560, 3072, 5120, 6144]   # one per thread / vector split, 1544 and 128 with idle lanes


def _err(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


@pytest.mark.parametrize("C", WIDTHS)
@pytest.mark.parametrize("batch,rpb", [(1, 37), (3, 5), (2, 700)])
def test_adaln_backward_widths(C, batch, rpb):
    torch.manual_seed(0)
    rows = batch * rpb
    x = torch.randn(rows, C, device="cuda", dtype=BF16)
    e = torch.randn(batch, 6, C, device="cuda")
    dy, dr = torch.randn_like(x), torch.randn_like(x)
    xg, eg = x.clone().requires_grad_(), e.clone().requires_grad_()
    y, xr = N.adaln_res(xg, eg[:, 1], eg[:, 0], rpb)
    dx, de = torch.autograd.grad([y, xr], [xg, eg], [dy, dr])
    xd, ed = x.double().requires_grad_(), e.double().requires_grad_()
    sc, sh = (ed[:, i].repeat_interleave(rpb, dim=0) for i in (1, 0))
    yd = torch.nn.functional.layer_norm(xd, (C,), eps=1e-6) * (1 + sc) + sh
    dxd, ded = torch.autograd.grad([yd, xd * 1.0], [xd, ed], [dy.double(), dr.double()])
    # one bf16 rounding of the output (1.7e-3 of the norm); the column sums stay in fp32
    assert _err(y, yd) < 2.5e-3 and _err(dx, dxd) < 2.5e-3 and _err(de, ded) < 1e-5


@pytest.mark.parametrize("C", [w for w in WIDTHS if w % 128 == 0])
@pytest.mark.parametrize("per_head,norm,rope", [(False, True, True), (True, True, True), (True, True, False), (False, False, True)])
def test_rmsrope_widths(C, per_head, norm, rope):
    torch.manual_seed(1)
    rows, D = 1201, 128
    x = torch.randn(rows, C, device="cuda", dtype=BF16)
    w = torch.randn(D if per_head else C, device="cuda").to(BF16) if norm else None
    ang = torch.randn(400, D // 2, device="cuda")
    fr = torch.stack([ang.cos(), ang.sin()], -1).contiguous() if rope else None
    dy = torch.randn_like(x)
    xg = x.clone().requires_grad_()
    wg = w.clone().requires_grad_() if norm else None
    y = N.rmsnorm_rope(xg, wg, fr, D, per_head)
    grads = torch.autograd.grad(y, [xg] + ([wg] if norm else []), dy)
    xr = x.float().requires_grad_()
    wr = w.float().requires_grad_() if norm else None
    yr = N.rmsnorm_rope_ref(xr, wr, fr, D, per_head)
    ref = torch.autograd.grad(yr, [xr] + ([wr] if norm else []), dy.float())
    assert _err(y, yr) < 2.5e-3
    for g, r in zip(grads, ref):
        assert _err(g, r) < 2.5e-3
    _lib.check_status()


def test_multi_fold_pieces():
    torch.manual_seed(2)
    L = _lib.lib()
    sizes = [1, 7, 8, 8191, 8192, 8193, 3, 100003]
    src = [torch.randn(n + 1, device="cuda").to(BF16)[i % 2:][:n] for i, n in enumerate(sizes)]   # every other one unaligned
    dst = [torch.randn(n + 4, device="cuda") for n in sizes]
    ref = [d.clone() for d in dst]
    for s, r in zip(src, ref):
        r[:s.numel()] += s.float()
    k = len(sizes)
    _lib.check(L.tt_multi_fold((_lib.c_ll * k)(*[s.data_ptr() for s in src]), (_lib.c_ll * k)(*[d.data_ptr() for d in dst]),
                               (_lib.c_int * k)(*sizes), _lib.c_int(k), _lib.stream()), "tt_multi_fold")
    for d, r in zip(dst, ref):
        assert torch.equal(d, r)
