"""The CUDA library's engine: ops, gradients and releases of tensors through the ``_fastcall`` extension instead of ctypes."""
import ctypes as C

from .frontend import Engine, Tensor

try:
    from . import _fastcall
except ImportError:  # not built yet; needs only a host compiler
    from ._build import build_fastcall

    build_fastcall()
    from . import _fastcall


class FastTensor(_fastcall.TensorBase, Tensor):
    """``engine``, ``handle`` and ``grad`` come from the extension's base; so does the release of the handle."""


class FastEngine(Engine):
    tensor_type = FastTensor

    def __init__(self, lib, prefix):
        super().__init__(lib, prefix)
        self._calls = _fastcall.Calls(*[C.cast(getattr(lib, f"{prefix}_{n}"), C.c_void_p).value
                                        for n in ("op", "tensor_free", "tensor_has_grad", "tensor_grad")])

    def op(self, name, inputs, ip=(), fp=()):
        return self._calls.op(FastTensor, self, name, inputs, ip, fp)
