"""Who listens to the call of a module."""
from __future__ import annotations

from torch.nn.modules.module import _has_any_global_hook


def watched(*modules) -> bool:
    """Whether a hook or a replaced ``forward`` hangs on the call of one of the modules."""
    return bool(_has_any_global_hook()) or any(m._forward_hooks or m._forward_pre_hooks or "forward" in m.__dict__ for m in modules)
