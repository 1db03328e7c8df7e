"""The native call path of the short operators (``csrc/bind.cpp``): ``attention``, ``linear``, ``experts``, and ``layers`` and ``pointers``,
which look over the modules and the tensors of a whole model.  Each returns None for a call it does not take; the callers then go their Python way, which raises the
error or serves the call.  Without the built module they always do."""

from __future__ import annotations

try:
    import torch  # noqa: F401  (the module links against torch's libraries)

    from lemoq._bind import attention, experts, layers, linear, pointers
except ImportError:  # not built: same results through ctypes
    def _absent(*args: object) -> None:
        return None

    attention = experts = layers = linear = pointers = _absent

__all__ = ["attention", "experts", "layers", "linear", "pointers"]
