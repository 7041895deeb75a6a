"""umT5 kernels (csrc/t5.cu) against the module chain."""
import pytest
import torch

from teletron_b200.models.encoders import UMT5Encoder, encode_prompt
from teletron_b200.ops import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,n,masked", [(2, 64, True), (1, 13, True), (3, 40, False), (1, 512, True), (2, 1, True)])
def test_t5_kernels_match_modules(batch, n, masked):
    torch.manual_seed(3)
    enc = UMT5Encoder(vocab=500, dim=256, dim_attn=256, dim_ffn=640, num_heads=4, num_layers=3)
    enc = enc.to("cuda", torch.bfloat16).eval().requires_grad_(False)
    for name, p in enc.named_parameters():
        if "norm" in name:
            torch.nn.init.normal_(p, 1.0, 0.1)
    ids = torch.randint(1, 500, (batch, n), device="cuda")
    mask = torch.zeros(batch, n, dtype=torch.long, device="cuda")
    for i in range(batch):
        mask[i, :max(1, n - 5 * i - 3)] = 1

    def run():
        before = _lib.launch_count()
        return (encode_prompt(enc, ids, mask) if masked else enc(ids)), _lib.launch_count() - before

    out, launches = run()
    assert launches == 3 * 4 + 1
    enc._native = lambda *a: False
    old, launches = run()
    assert launches == 0
    enc.double()
    ref, _ = run()

    def err(a):
        return ((a.double() - ref).norm() / ref.norm()).item()

    assert err(out) < 1.2 * err(old) + 1e-3, (err(out), err(old))


def test_t5_route_to_modules():
    enc = UMT5Encoder(vocab=50, dim=64, dim_attn=64, dim_ffn=128, num_heads=4, num_layers=1).to("cuda", torch.bfloat16)
    ids = torch.randint(1, 50, (1, 8), device="cuda")
    assert not enc._native(ids, None)                 # gradients wanted
    with torch.no_grad():
        assert enc._native(ids, None) and not enc._native(ids, torch.ones(1, 8, 8, device="cuda"))
        handle = enc.blocks[0].attn.q.register_forward_hook(lambda *a: None)
        assert not enc._native(ids, None)
        handle.remove()
        assert not enc.float()._native(ids, None)
