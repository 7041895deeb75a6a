"""Calls of the model parts that have to keep their results, on the CPU."""
import torch

from teletron_b200.models import WanModel, wan_config


def test_block_widens_its_timestep_modulation():
    """A bf16 timestep modulation is added to the bf16 table in fp32."""
    torch.manual_seed(0)
    cfg = wan_config("wan-tiny")
    blk = WanModel(cfg).to(torch.bfloat16).blocks[0]
    x, ctx = torch.randn(8, cfg.dim).bfloat16(), torch.randn(1, 4, cfg.dim).bfloat16()
    t_mod, freqs = torch.randn(1, 6, cfg.dim).bfloat16(), torch.randn(8, cfg.head_dim // 2, 2)
    a, b = (blk(x, ctx, t, freqs, 1, None) for t in (t_mod, t_mod.float()))
    assert torch.equal(a, b)


def test_feed_forward_hooks_run():
    """Hooks on the feed-forward branch of a dual-stream block and on its second projection, forward and backward."""
    from teletron_b200.models.hunyuan import HunyuanVideoModel, hunyuan_config

    torch.manual_seed(0)
    cfg = hunyuan_config("hunyuan-tiny", num_layers=1, num_single_layers=0)
    m = HunyuanVideoModel(cfg)
    blk = m.transformer_blocks[0]
    xv, xt = torch.randn(8, cfg.hidden_size, requires_grad=True), torch.randn(4, cfg.hidden_size)
    args = (xv, xt, torch.randn(1, cfg.hidden_size), m.rope((1, 2, 4), None), 1, None, None)
    ref = blk(*args)
    seen = []
    for mod in (blk.ff, blk.ff_context, blk.ff.net[2]):
        mod.register_forward_hook(lambda *a: seen.append("f"))
    blk.ff.register_full_backward_hook(lambda *a: seen.append("b"))
    out = blk(*args)
    assert seen == ["f"] * 3 and all(torch.equal(a, b) for a, b in zip(out, ref))
    out[0].sum().backward()
    assert seen == ["f"] * 3 + ["b"]
    doubled = blk.ff.register_forward_hook(lambda mod, i, o: o * 2)
    assert not torch.equal(blk(*args)[0], ref[0])
    doubled.remove()
