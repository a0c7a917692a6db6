"""irontensor_b200: the B200 (sm_100a) attention path for the IronTensor library.

Host-side mirror of the reference's attention interface (`flash_attention`, `attention`,
`attention_backward_recompute`, `Tensor`, `CommandBatch`) over the C ABI declared in
include/irontensor_b200.h.  Importing this package needs neither a GPU nor torch; using it does: the names below are
loaded with their module, and torch with it, when one of them is first asked for."""
import importlib

_MODULES = ("ops", "synth", "_lib")
__all__ = ["CommandBatch", "Precision", "Tensor", "attention", "attention_backward", "attention_backward_recompute", "attention_gqa",
           "attention_gqa_backward", "attention_decode", "attention_packed", "attention_packed_backward", "linear_backward",
           "linear_forward", "qkv_rope_forward", "rope", "rope_qk", "flash_attention", "context", "raw", "HostAttentionStep"]


def __getattr__(name):
    if name in _MODULES:
        return importlib.import_module("." + name, __name__)
    if name in __all__:
        value = globals()[name] = getattr(importlib.import_module(".ops", __name__), name)
        return value
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


def __dir__():
    return sorted({*globals(), *__all__, *_MODULES})
