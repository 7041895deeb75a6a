"""Pointwise kernels of the umT5 text encoder (csrc/t5.cu); bf16 on a GPU, no gradients."""
from __future__ import annotations

import torch

from . import _lib


def add_norm(x, delta, weight, eps):
    """(x + delta, T5 layer norm of it); delta None: (x, norm of x)."""
    assert x.is_contiguous() and x.dtype == torch.bfloat16 and weight.is_contiguous()
    C = x.shape[-1]
    assert weight.shape == (C,)
    if delta is not None:
        assert delta.shape == x.shape and delta.is_contiguous() and delta.dtype == torch.bfloat16
    xo = x if delta is None else torch.empty_like(x)
    y = torch.empty_like(x)
    _lib.check(_lib.lib().tt_t5_add_norm(_lib.ptr(x), _lib.ptr(delta), _lib.ptr(xo), _lib.ptr(y), _lib.ptr(weight),
                                         _lib.c_ll(x.numel() // C), _lib.c_int(C), _lib.c_float(eps), _lib.stream()),
               "tt_t5_add_norm")
    return xo, y


def geglu(a, gate):
    """a * gelu_tanh(gate)."""
    assert a.shape == gate.shape and a.is_contiguous() and gate.is_contiguous() and a.dtype == gate.dtype == torch.bfloat16
    y = torch.empty_like(a)
    _lib.check(_lib.lib().tt_t5_geglu(_lib.ptr(a), _lib.ptr(gate), _lib.ptr(y), _lib.c_ll(a.numel()), _lib.stream()),
               "tt_t5_geglu")
    return y


def bias(emb, bucket, keep, batch, heads, n):
    """[batch, heads, n, n]: emb[bucket[j - i + n - 1], head], the lowest bf16 where keep[b, j] is 0."""
    assert emb.dtype == torch.bfloat16 and emb.is_contiguous() and emb.shape[1] == heads
    assert bucket.dtype == torch.int32 and bucket.is_contiguous() and bucket.numel() == 2 * n - 1
    out = torch.empty((batch, heads, n, n), dtype=torch.bfloat16, device=emb.device)
    _lib.check(_lib.lib().tt_t5_bias(_lib.ptr(emb), _lib.ptr(bucket), _lib.ptr(keep), _lib.ptr(out), _lib.c_int(batch),
                                     _lib.c_int(heads), _lib.c_int(n), _lib.stream()), "tt_t5_bias")
    return out
