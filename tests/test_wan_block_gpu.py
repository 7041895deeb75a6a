"""The block-level inference call (csrc/wan_block.cu) against the op layer."""
import pytest
import torch

from teletron_b200.models import WanModel, wan_config
from teletron_b200.ops import _lib

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("batch,frames,h,w,text", [(1, 1, 4, 4, 512), (2, 3, 18, 22, 40), (1, 2, 32, 32, 512), (3, 1, 2, 2, 8)])
@pytest.mark.parametrize("dim,heads", [(256, 2), (1536, 12)])
def test_wan_block_call_equals_op_layer(dim, heads, batch, frames, h, w, text):
    """The native block runs the op layer's kernels on the op layer's operands: the same bits."""
    torch.manual_seed(0)
    cfg = wan_config("wan2.1-1.3b-t2v", dim=dim, num_heads=heads, num_layers=2, ffn_dim=4 * dim + 128)
    with torch.device("cuda"):
        m = WanModel(cfg).to(BF16).eval()
    for blk in m.blocks:
        for n in (blk.norm3, blk.self_attn.norm_q, blk.cross_attn.norm_k):
            torch.nn.init.normal_(n.weight, 1.0, 0.1)
    x = torch.randn(batch, 16, frames, h, w, device="cuda", dtype=BF16)
    ctx = torch.randn(batch, text, cfg.text_dim, device="cuda", dtype=BF16)
    t = torch.linspace(3, 900, batch, device="cuda")
    ref = m(x, t, ctx).detach()                     # gradients on: the op layer
    with torch.no_grad():
        out = m(x, t, ctx)
        handle = m.blocks[0].ffn[0].register_forward_hook(lambda *a: None)
        hooked = m(x, t, ctx)                       # a hook inside a block: the op layer again
        handle.remove()
    assert torch.isfinite(ref).all() and torch.equal(out, ref) and torch.equal(hooked, ref)
    _lib.check_status()
