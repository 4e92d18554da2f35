"""When the arithmetic of a module may stand for a call of it.

Fused paths read a module's parameters instead of calling it.  That gives the same result only where a call would run its
class's own ``forward`` and nothing else: no subclass, no ``forward`` set on the instance or put in place of the class's, no
hooks on the module or on all modules, and parameters that are not computed on access (a parametrisation makes a subclass).
"""
from __future__ import annotations

from torch.nn.modules import module as _nn


def global_hooks() -> bool:
    """Hooks that every module call runs (``torch.nn.modules.module.register_module_*_hook``)."""
    return bool(_nn._global_forward_hooks or _nn._global_forward_pre_hooks or _nn._global_backward_hooks or _nn._global_backward_pre_hooks)


def own_forward(cls) -> bool:
    """Whether ``cls.forward`` is the one that the class was written with."""
    fwd = cls.forward
    return getattr(fwd, "__qualname__", "") == cls.__qualname__ + ".forward" and fwd.__module__ == cls.__module__


def own_call(module, cls) -> bool:
    """Whether calling ``module`` runs ``cls.forward`` as ``cls`` defines it and nothing else (apart from ``global_hooks``)."""
    if type(module) is not cls:
        return False
    d = module.__dict__
    return not (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"] or "forward" in d) \
        and own_forward(cls)
