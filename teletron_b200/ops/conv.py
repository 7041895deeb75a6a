"""Video-VAE convolutions on tcgen05 (csrc/conv.cu) over the channel-chunked layout ``[T, C / E, H, W, E]`` with E
elements of 16 bytes (8 bf16, 4 fp32).  Replaces cuDNN behind ``nn.Conv3d`` / ``nn.Conv2d`` in the reference VAE
(teletron/models/wan/encoder/wan_video_vae.py:34-52, 86-173).  fp32 tensors are multiplied as TF32, which is what
cuDNN does with them by default; the operands are rounded to nearest, not truncated.
"""
from __future__ import annotations

import torch

from . import _lib

CONV_SPATIAL, CONV_POINT, CONV_STRIDE2 = 0, 1, 2   # k_t x 3 x 3 (padding 1), k_t x 1 x 1, 3 x 3 stride 2


def _f32(dtype) -> int:
    return int(dtype == torch.float32)


def chunk_elems(dtype) -> int:
    return 4 if dtype == torch.float32 else 8


class PackedConv:
    """Weights and bias of one convolution in the order the kernel reads them; channels are padded to an even number of
    chunks (inputs) and to 16 (outputs).  ``size`` is the (frames, height, width) of the output that the split into
    output-channel tiles is made for; other sizes are computed with it too."""

    def __init__(self, weight: torch.Tensor, bias, kind: int, size):
        n, c = weight.shape[:2]
        self.kind, self.kt = kind, (weight.shape[2] if weight.dim() == 5 else 1)
        e = chunk_elems(weight.dtype)
        self.n_real, self.n, self.chunks = n, -(-n // 16) * 16, -(-c // (2 * e)) * 2
        L = _lib.lib()
        L.tt_conv_packed_bytes.restype = _lib.c_ll
        dims = (_lib.c_int(kind), _lib.c_int(self.kt))
        nbytes = L.tt_conv_packed_bytes(*dims, _lib.c_int(self.chunks), _lib.c_int(self.n))
        if nbytes < 0:
            raise ValueError(f"convolution outside the kernel's domain: weight {tuple(weight.shape)}")
        self.nt = L.tt_conv_tile_channels(_lib.c_int(self.n), *(_lib.c_int(v) for v in size), _lib.c_int(L.tt_num_sms()))
        self.data = torch.empty(nbytes, dtype=torch.uint8, device=weight.device)
        w = weight.detach().contiguous()
        b = None if bias is None else bias.detach().contiguous()
        assert b is None or (b.dtype == w.dtype and b.device == w.device and b.numel() == n)
        _lib.check(L.tt_conv_pack(_lib.ptr(w), _lib.ptr(b), _lib.c_int(_f32(w.dtype)), *dims, _lib.c_int(c), _lib.c_int(n),
                                  _lib.c_int(self.chunks), _lib.c_int(self.n), _lib.c_int(self.nt), _lib.ptr(self.data),
                                  _lib.stream()), "tt_conv_pack")


def conv(x: torch.Tensor, pk: PackedConv, frames: int, hw, *, t_stride=1, t_off=0, out=None, res=None, t_mul=1,
         planar=False):
    """``frames`` x ``hw`` outputs; output frame t reads input frames ``t * t_stride + t_off ..``, frames below zero
    are zeros.  ``t_mul`` m > 1 spreads the output channels over m frames (frame t * m + i takes the i-th part).
    ``planar`` returns dense [C, T, H, W] instead of chunks."""
    e, (h, w) = chunk_elems(x.dtype), hw
    c_out = pk.n // t_mul
    assert x.is_contiguous() and x.dim() == 5 and x.shape[4] == e
    assert x.shape[1] == pk.chunks * (4 if pk.kind == CONV_STRIDE2 else 1)
    if planar:
        out = torch.empty((pk.n_real, frames, h, w), dtype=x.dtype, device=x.device)
    elif out is None:
        out = torch.empty((frames * t_mul, c_out // e, h, w, e), dtype=x.dtype, device=x.device)
    if not planar:
        assert out.is_contiguous() and out.shape == (frames * t_mul, c_out // e, h, w, e) and pk.n == pk.n_real
    if res is not None:
        assert res.is_contiguous() and res.shape == out.shape and not planar
    _lib.check(_lib.lib().tt_conv(
        _lib.ptr(x), _lib.c_int(_f32(x.dtype)), _lib.c_int(pk.kind), _lib.c_int(pk.kt), _lib.c_int(x.shape[0]),
        _lib.c_int(x.shape[2]), _lib.c_int(x.shape[3]), _lib.c_int(pk.chunks), _lib.ptr(pk.data), _lib.c_int(pk.n),
        _lib.c_int(pk.nt), _lib.ptr(out), _lib.ptr(res), _lib.c_int(frames), _lib.c_int(h), _lib.c_int(w),
        _lib.c_int(t_stride), _lib.c_int(t_off), _lib.c_int(c_out), _lib.c_int(t_mul), _lib.c_int(int(planar)),
        _lib.c_int(pk.n_real), _lib.ptr(_lib.status_word(x.device)), _lib.stream()), "tt_conv")
    return out


def chan_norm(x: torch.Tensor, gamma: torch.Tensor, out: torch.Tensor, act: bool = True) -> torch.Tensor:
    """``silu(x / max(|x|, 1e-12) * sqrt(C) * gamma)`` over the channels of every pixel; gamma [C] in x's type."""
    t, chunks, h, w, e = x.shape
    assert x.is_contiguous() and out.is_contiguous() and out.shape == x.shape and gamma.numel() == chunks * e
    assert gamma.dtype == x.dtype and gamma.is_contiguous()
    _lib.check(_lib.lib().tt_chan_norm(_lib.ptr(x), _lib.ptr(out), _lib.ptr(gamma), _lib.c_int(_f32(x.dtype)),
                                       _lib.c_int(t), _lib.c_int(chunks), _lib.c_ll(h * w), _lib.c_int(int(act)),
                                       _lib.stream()), "tt_chan_norm")
    return out


def from_planar(x: torch.Tensor, round_tf32: bool = False) -> torch.Tensor:
    """[C, T, H, W] (any strides) -> chunks; channels are padded with zeros to an even number of chunks."""
    c, t, h, w = x.shape
    e = chunk_elems(x.dtype)
    chunks = -(-c // (2 * e)) * 2
    out = torch.empty((t, chunks, h, w, e), dtype=x.dtype, device=x.device)
    _lib.check(_lib.lib().tt_blk_from_planar(
        _lib.ptr(x), _lib.ptr(out), _lib.c_int(_f32(x.dtype)), _lib.c_int(c), _lib.c_int(chunks), _lib.c_int(t),
        _lib.c_int(h), _lib.c_int(w), *(_lib.c_ll(s) for s in x.stride()), _lib.c_int(int(round_tf32)), _lib.stream()),
        "tt_blk_from_planar")
    return out


def to_planar(x: torch.Tensor) -> torch.Tensor:
    t, chunks, h, w, e = x.shape
    assert x.is_contiguous()
    out = torch.empty((chunks * e, t, h, w), dtype=x.dtype, device=x.device)
    _lib.check(_lib.lib().tt_blk_to_planar(_lib.ptr(x), _lib.ptr(out), _lib.c_int(_f32(x.dtype)), _lib.c_int(chunks),
                                           _lib.c_int(t), _lib.c_ll(h * w), _lib.stream()), "tt_blk_to_planar")
    return out


def _move(x, mode, shape, out=None):
    t, n, h, w, _ = x.shape
    assert x.is_contiguous()
    out = torch.empty(shape, dtype=x.dtype, device=x.device) if out is None else out
    assert out.is_contiguous() and out.shape == shape
    _lib.check(_lib.lib().tt_blk_move(_lib.ptr(x), _lib.ptr(out), _lib.c_int(_f32(x.dtype)), _lib.c_int(mode),
                                      _lib.c_int(t), _lib.c_int(n), _lib.c_int(h), _lib.c_int(w), _lib.stream()),
               "tt_blk_move")
    return out


def enlarge2(x):
    """Nearest 2x enlargement of every frame."""
    t, n, h, w, e = x.shape
    return _move(x, 0, (t, n, 2 * h, 2 * w, e))


def phases2(x):
    """Pixel phases (y & 1, x & 1) as four channel groups, the input of a stride-2 convolution."""
    t, n, h, w, e = x.shape
    return _move(x, 1, (t, 4 * n, (h + 1) // 2, (w + 1) // 2, e))


def rounded(x, out=None):
    """The tensor as a convolution operand: fp32 rounded to TF32; bf16 as it is (copied only into a given ``out``)."""
    if out is None and x.dtype == torch.bfloat16:
        return x
    return _move(x, 2, tuple(x.shape), out)


def softmax_split(scores, n: int, parts: int = 2):
    """Row softmax of the first ``n`` columns of fp32 [rows, np] as bf16 [rows, parts * np] (zero past column n): the
    rounded values, then the rounded remainders.  Two parts keep 16 bits of a probability, three all of an fp32 one."""
    rows, padded = scores.shape
    assert scores.dtype == torch.float32 and scores.is_contiguous()
    out = torch.empty((rows, parts * padded), dtype=torch.bfloat16, device=scores.device)
    _lib.check(_lib.lib().tt_softmax_split(_lib.ptr(scores), _lib.ptr(out), _lib.c_ll(rows), _lib.c_int(n),
                                           _lib.c_int(padded), _lib.c_int(parts), _lib.stream()), "tt_softmax_split")
    return out
