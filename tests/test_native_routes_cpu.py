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
