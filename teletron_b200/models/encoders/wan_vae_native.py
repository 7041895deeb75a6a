"""The VAE's encoder and decoder on the library's convolution kernels (ops/conv.py), module by module the function
of ``wan_vae.Encoder3d`` / ``Decoder3d`` (teletron/models/wan/encoder/wan_video_vae.py:34-420 in the reference).

Activations stay in the channel-chunked layout from the first convolution to the last; norm + SiLU write straight into
the buffer that the following convolution reads, behind the history frames of a chunked pass; the residual is added in
the convolution's epilogue; temporal up-sampling stores its two channel halves into alternating frames.
"""
from __future__ import annotations

import torch
import torch.nn as nn

from ... import ops
from ...ops import conv as C
from ...ops._lib import plain_call
from ..native_route import plain_modules
from . import wan_vae as V


_MODULES = frozenset((V.CausalConv3d, V.RMS_norm, V.Resample, V.ResidualBlock, V.AttentionBlock, nn.Conv2d, nn.SiLU, nn.Dropout,
                      nn.Identity, nn.Upsample, nn.ZeroPad2d, nn.Sequential))


def usable(net: nn.Module, x: torch.Tensor) -> bool:
    """Whether this forward pass may take the native kernels: one clip on a GPU, bf16 or fp32 with TF32 convolutions
    allowed (torch's default), weights of the same type, no gradients, hooks or tracing, channel counts in multiples
    of 16 up to 384 behind the first convolution."""
    if not (x.is_cuda and x.dim() == 5 and x.shape[0] == 1 and x.numel() > 0):
        return False
    if x.dtype == torch.float32:
        # the per-operator setting: `allow_tf32` may not be read once a program uses it, and follows it otherwise
        if not (torch.backends.cudnn.enabled and torch.backends.cudnn.conv.fp32_precision == "tf32"):
            return False
    elif x.dtype != torch.bfloat16:
        return False
    if not plain_call(x.device) or type(x) is not torch.Tensor:
        return False
    mods = plain_modules(net, _MODULES)
    if mods is None:
        return False
    grad = torch.is_grad_enabled()
    if grad and x.requires_grad:
        return False
    first, last = net.conv1, net.head[2]
    for m in mods:
        if isinstance(m, nn.Dropout) and m.training and m.p > 0:
            return False
        if isinstance(m, (nn.Conv2d, nn.Conv3d)):
            if (m.in_channels % 16 and m is not first) or (m.out_channels % 16 and m is not last):
                return False
            if m is not first and m.in_channels > 384:
                return False
        for p in m._parameters.values():
            if p is not None and (p.device != x.device or p.dtype != x.dtype or type(p) is not nn.Parameter
                                  or (grad and p.requires_grad)):
                return False
    return True


def _gamma(norm: nn.Module) -> torch.Tensor:
    """The norm's weights as a vector that starts on 16 bytes, as the kernel reads it; parameters may be views into one
    flat buffer."""
    g = norm.gamma.detach().reshape(-1)
    return g if g.data_ptr() % 16 == 0 else g.clone()


def open_run(net: nn.Module, x: torch.Tensor):
    return Run() if usable(net, x) else None


# Attention scores that are held at a time: 1 GiB in fp32 and 1.5 GiB of probabilities, query rows in whole row tiles.  All
# 6,240 rows of a 480P frame fit; the library holds all scores of a frame and their softmax, 2 x 4.3 GB at 1080P.
SCORES = 1 << 28


class Run:
    """One encode / decode call: the packed weights, shared by its chunks and tiles."""

    def __init__(self):
        self.packs = {}

    def conv(self, m, kind, x, frames, hw, **kw):
        pk = self.packs.get(m)
        if pk is None:
            pk = self.packs[m] = C.PackedConv(m.weight, m.bias, kind, (frames, *hw))
        return C.conv(x, pk, frames, hw, **kw)

    # -------------------------------------------------------------------------------------------------- pieces
    def _with_history(self, m, shape, like):
        """Buffer for the input of causal convolution ``m`` (two frames of history), the view to fill and the frame
        offset of its first window."""
        st = V._STREAM
        hist = st.get(m) if st is not None else None
        n = 0 if hist is None else 2
        buf = torch.empty((shape[0] + n, *shape[1:]), dtype=like.dtype, device=like.device)
        if n:
            buf[:2].copy_(hist)
        return buf, buf[n:], n - 2

    @staticmethod
    def _keep_history(m, buf):
        st = V._STREAM
        if st is not None:
            tail = buf[-2:].clone()
            st[m] = tail if tail.shape[0] == 2 else torch.cat([torch.zeros_like(tail), tail])

    def norm_conv(self, norm, m, x, res=None, planar=False):
        buf, view, t_off = self._with_history(m, x.shape, x)
        C.chan_norm(x, _gamma(norm), view)
        self._keep_history(m, buf)
        return self.conv(m, C.CONV_SPATIAL, buf, x.shape[0], x.shape[2:4], t_off=t_off, res=res, planar=planar)

    def first_conv(self, m, x):
        """x: planar [C, T, H, W]."""
        x = C.from_planar(x, round_tf32=True)
        frames, t_off = x.shape[0], -2
        st = V._STREAM
        if st is not None and st.get(m) is not None:
            x, t_off = torch.cat([st[m], x]), 0
        self._keep_history(m, x)
        return self.conv(m, C.CONV_SPATIAL, x, frames, x.shape[2:4], t_off=t_off)

    def res_block(self, m, x):
        r = m.residual
        h = self.norm_conv(r[0], r[2], x)
        if isinstance(m.shortcut, nn.Identity):
            skip = x
        else:
            skip = self.conv(m.shortcut, C.CONV_POINT, C.rounded(x), x.shape[0], x.shape[2:4])
        return self.norm_conv(r[3], r[6], h, res=skip)

    def attention(self, m, x):
        """Single-head attention over the pixels of each frame (heads of up to 384 channels)."""
        t, chunks, h, w, e = x.shape
        n, c = h * w, chunks * e
        if x.dtype != torch.bfloat16:
            return C.from_planar(m(C.to_planar(x).unsqueeze(0)).squeeze(0))
        y = C.chan_norm(x, _gamma(m.norm), torch.empty_like(x), act=False)
        qkv = self.conv(m.to_qkv, C.CONV_POINT, y, t, (h, w))
        padded = -(-n // 8) * 8                            # keys in whole vectors; the softmax stops at n
        rows = qkv.new_zeros((t, padded, 3 * c))
        rows[:, :n].unflatten(1, (h, w)).unflatten(3, (3 * chunks, e)).copy_(qkv.permute(0, 2, 3, 1, 4))
        out = torch.empty((t, n, c), dtype=x.dtype, device=x.device)
        step = max(256, SCORES // padded // 256 * 256)
        for f in range(t):
            k, v = rows[f, :, c:2 * c], rows[f, :, 2 * c:]
            v = torch.cat([v, v, v])
            for i in range(0, n, step):
                scores = ops.gemm(rows[f, i:min(i + step, n), :c], k, out_dtype=torch.float32, alpha=c ** -0.5)
                ops.gemm(C.softmax_split(scores, n, 3), v, b_mn=True, out=out[f, i:i + step])
        o = C.from_planar(out.view(t, h, w, c).permute(3, 0, 1, 2))
        return self.conv(m.proj, C.CONV_POINT, o, t, (h, w), res=x)

    def down(self, m, x):
        st = V._STREAM
        first = st is None or ("seen", m) not in st
        if st is not None:
            st[("seen", m)] = True
        hw = (x.shape[2] // 2, x.shape[3] // 2)
        x = self.conv(m.resample[1], C.CONV_STRIDE2, C.phases2(x), x.shape[0], hw)
        if m.mode != "downsample3d":
            return x
        last = x[-1:].clone() if st is not None else None
        t = x.shape[0]
        if not first:
            x, t, keep = torch.cat([st[("last", m)], x]), t + 1, 0
        else:
            keep = 1
        if t > 1:
            n = (t - 3) // 2 + 1
            out = torch.empty((keep + n, *x.shape[1:]), dtype=x.dtype, device=x.device)
            if keep:
                out[0].copy_(x[0])
            self.conv(m.time_conv, C.CONV_POINT, C.rounded(x), n, hw, t_stride=2, out=out[keep:])
            x = out
        if st is not None:
            st[("last", m)] = last
        return x

    def up(self, m, x):
        st = V._STREAM
        first = st is None or ("seen", m) not in st
        if st is not None:
            st[("seen", m)] = True
        t, hw = x.shape[0], x.shape[2:4]
        if m.mode == "upsample3d":
            keep = 1 if first else 0
            if t > keep:
                rest = x[keep:]
                buf, view, t_off = self._with_history(m.time_conv, rest.shape, x)
                C.rounded(rest, out=view)
                self._keep_history(m.time_conv, buf)
                out = torch.empty((keep + 2 * (t - keep), *x.shape[1:]), dtype=x.dtype, device=x.device)
                if keep:
                    out[0].copy_(x[0])
                self.conv(m.time_conv, C.CONV_POINT, buf, t - keep, hw, t_off=t_off, out=out[keep:], t_mul=2)
                x = out
        return self.conv(m.resample[1], C.CONV_SPATIAL, C.enlarge2(x), x.shape[0], (2 * hw[0], 2 * hw[1]))

    # ------------------------------------------------------------------------------------------------- networks
    def _layers(self, layers, x):
        for m in layers:
            if isinstance(m, V.ResidualBlock):
                x = self.res_block(m, x)
            elif isinstance(m, V.AttentionBlock):
                x = self.attention(m, x)
            else:
                x = self.down(m, x) if m.mode.startswith("down") else self.up(m, x)
        return x

    def encoder(self, net, x):
        """[1, 3, T, H, W] -> [1, 2 z, T', H / 8, W / 8], the same as ``net(x)``."""
        h = self._layers(net.downsamples, self.first_conv(net.conv1, x[0]))
        h = self._layers(net.middle, h)
        return self.norm_conv(net.head[0], net.head[2], h, planar=True).unsqueeze(0)

    def decoder(self, net, z):
        """[1, z, T, H, W] -> [1, 3, T', 8 H, 8 W], the same as ``net(z)``."""
        h = self._layers(net.middle, self.first_conv(net.conv1, z[0]))
        h = self._layers(net.upsamples, h)
        return self.norm_conv(net.head[0], net.head[2], h, planar=True).unsqueeze(0)
