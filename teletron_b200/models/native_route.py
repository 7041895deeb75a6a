"""Whether a native call may skip the modules whose work it does."""
from __future__ import annotations

import torch.nn as nn
from torch.nn.modules.module import _has_any_global_hook


def plain_modules(root: nn.Module, types, root_hooks: bool = True):
    """The modules of ``root`` when calling ``root`` would run the forward methods that the native call stands for, and nothing else: every
    module below it is of one of ``types`` itself (a wrapper or subclass computes something of its own), with the
    class' forward, without forward hooks.  Else None.  ``root_hooks``: root's own hooks count too (its ``__call__`` is
    skipped)."""
    if _has_any_global_hook():
        return None
    mods = list(root.modules())
    for m in mods:
        if (m._forward_hooks or m._forward_pre_hooks) and (m is not root or root_hooks):
            return None
        if "forward" in m.__dict__ or (type(m) not in types and m is not root):
            return None
    return mods


def unobserved(*modules: nn.Module) -> bool:
    """True when no hook, forward or backward, and no instance-level forward sits on any of the modules."""
    return not (_has_any_global_hook() or any(
        m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks or "forward" in m.__dict__
        for m in modules))
