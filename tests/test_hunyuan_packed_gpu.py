"""HunyuanVideo single-stream blocks on packed rows (no gradients) against the two-stream form."""
import pytest
import torch

from teletron_b200.models.hunyuan import HunyuanVideoModel, SingleStreamBlock, hunyuan_config
from teletron_b200.ops import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames,h,w,text,keep", [(1, 4, 4, 8, 8), (2, 18, 22, 40, 7), (3, 32, 34, 256, 100), (1, 2, 2, 16, None)])
def test_packed_single_blocks(monkeypatch, frames, h, w, text, keep):
    torch.manual_seed(0)
    cfg = hunyuan_config("hunyuanvideo-13b-t2v", num_layers=1, num_single_layers=2)
    with torch.device("cuda"):
        m = HunyuanVideoModel(cfg).to(torch.bfloat16).eval()
    for blk in m.single_transformer_blocks:
        for n in (blk.attn.norm_q, blk.attn.norm_k):
            torch.nn.init.normal_(n.weight, 1.0, 0.1)
    x = torch.randn(1, 16, frames, h, w, device="cuda", dtype=torch.bfloat16)
    txt = torch.randn(1, text, cfg.text_embed_dim, device="cuda", dtype=torch.bfloat16)
    mask = None if keep is None else (torch.arange(text, device="cuda") < keep).long()[None]
    pooled = torch.randn(1, 768, device="cuda", dtype=torch.bfloat16)
    args = (x, torch.tensor([500.0], device="cuda"), txt, mask, pooled, torch.tensor([6000.0], device="cuda"))
    calls = []
    run = SingleStreamBlock.packed_infer
    monkeypatch.setattr(SingleStreamBlock, "packed_infer", lambda self, *a: calls.append(1) or run(self, *a))
    with torch.no_grad():
        out = m(*args)
        assert len(calls) == 2
        monkeypatch.setattr(SingleStreamBlock, "packs", lambda self, *a: False)
        ref = m(*args)
    assert len(calls) == 2
    # the same products with other tile shapes: fp32 sums in another order, rounded to bf16 in each of two layers
    assert ((out.float() - ref.float()).norm() / ref.float().norm()).item() < 8e-3
    _lib.check_status()


def test_packed_route():
    cfg = hunyuan_config("hunyuanvideo-13b-t2v", num_layers=1, num_single_layers=1)
    with torch.device("cuda"):
        m = HunyuanVideoModel(cfg).to(torch.bfloat16).eval()
    blk = m.single_transformer_blocks[0]
    x = torch.randn(24, cfg.hidden_size, device="cuda", dtype=torch.bfloat16)
    temb, fr = torch.randn(1, cfg.hidden_size, device="cuda"), torch.randn(16, 64, 2, device="cuda")
    assert not blk.packs(x, 16, temb, fr, 1, None)            # gradients on
    with torch.no_grad():
        assert blk.packs(x, 16, temb, fr, 1, None)
        assert not blk.packs(x, 16, temb, fr, 2, None) and not blk.packs(x, 24, temb, fr, 1, None)
        assert not blk.packs(x.float(), 16, temb, fr, 1, None) and not blk.packs(x.cpu(), 16, temb, fr, 1, None)
        handle = blk.attn.to_qkv.register_forward_hook(lambda *a: None)
        assert not blk.packs(x, 16, temb, fr, 1, None)
        handle.remove()
