"""Resources handle and tensor marshalling shared by the Python mirror of the C interface."""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from . import _lib as L

_TORCH_DL = {torch.float32: (L.kDLFloat, 32), torch.float16: (L.kDLFloat, 16),
             torch.int8: (L.kDLInt, 8), torch.uint8: (L.kDLUInt, 8), torch.int64: (L.kDLInt, 64),
             torch.uint32: (L.kDLUInt, 32), torch.int32: (L.kDLInt, 32)}
_NP_DL = {np.dtype(np.float32): (L.kDLFloat, 32), np.dtype(np.float16): (L.kDLFloat, 16),
          np.dtype(np.int8): (L.kDLInt, 8), np.dtype(np.uint8): (L.kDLUInt, 8),
          np.dtype(np.int64): (L.kDLInt, 64), np.dtype(np.uint32): (L.kDLUInt, 32),
          np.dtype(np.int32): (L.kDLInt, 32)}


# the raw handle of torch's current stream, without building a Stream object where torch offers that
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _current_stream() -> int:
    if _raw_stream is not None:
        return _raw_stream(torch.cuda.current_device())
    return torch.cuda.current_stream().cuda_stream


class Resources:
    """Mirror of ``cuvs.common.Resources``: owns a ``cuvsResources_t`` bound to the current device.

    Work is enqueued on ``stream`` (default: torch's current stream at call time); ``sync()`` waits
    for it.
    """

    def __init__(self, stream: int | None = None):
        self._lib = L.load()
        h = C.c_size_t(0)
        L.check(self._lib.cuvsResourcesCreate(C.byref(h)))
        self.handle = h.value
        self._fixed_stream = stream
        if stream is not None:
            L.check(self._lib.cuvsStreamSet(self.handle, C.c_void_p(stream)))

    def use_current_stream(self):
        if self._fixed_stream is None:
            L.check(self._lib.cuvsStreamSet(self.handle, _current_stream()))

    def stream_at_call(self, device: int) -> int:
        """The stream that a call made now uses: the fixed one, else torch's current one."""
        if self._fixed_stream is not None:
            return self._fixed_stream
        return _raw_stream(device) if _raw_stream is not None else _current_stream()

    def sync(self):
        L.check(self._lib.cuvsStreamSync(self.handle))

    def set_workspace_pool(self, nbytes: int):
        L.check(self._lib.cuvsResourcesSetWorkspacePool(self.handle, C.c_size_t(nbytes)))

    def __del__(self):
        try:
            if getattr(self, "handle", 0):
                self._lib.cuvsResourcesDestroy(self.handle)
                self.handle = 0
        except Exception:
            pass


_default_resources = {}


def default_resources(dev: int | None = None) -> Resources:
    if dev is None:
        dev = torch.cuda.current_device()
    r = _default_resources.get(dev)
    if r is None:
        r = _default_resources[dev] = Resources()
    return r


CUDA_DEVICES = [torch.device("cuda", i) for i in range(64)]
# (type code, bits) of vectors
ELEMENT_TYPES = {t: _TORCH_DL[t] for t in (torch.float32, torch.float16, torch.int8, torch.uint8)}


def is_cuda_matrix(t, dtype) -> bool:
    """A row-major matrix of `dtype` that native code can be given by its address."""
    return type(t) is torch.Tensor and t.dtype == dtype and t.is_cuda and t.dim() == 2 and t.is_contiguous()


# ndim | dtype code << 32 | bits << 40 | lanes << 48, as the words of a DLTensor hold them
_TORCH_WORD = {t: (code << 32) | (bits << 40) | (1 << 48) for t, (code, bits) in _TORCH_DL.items()}
_NP_WORD = {t: (code << 32) | (bits << 40) | (1 << 48) for t, (code, bits) in _NP_DL.items()}
_WORDS = {n: C.c_int64 * (8 + 2 * n) for n in range(5)}


class DLTensorRef:
    """A DLManagedTensor describing (not owning) a torch tensor or a numpy array.

    The structure, its shape and its strides are one array of 64-bit words, filled by one call: three of these are made
    for every search, and field-by-field ctypes assignments took longer than the launches."""

    __slots__ = ("_keep", "_words")

    def __init__(self, obj, strided: bool = False):
        """`strided`: describe a non-contiguous torch tensor by its strides (only entry points that
        say so accept one) instead of refusing it."""
        strides = ()
        if isinstance(obj, torch.Tensor):
            if not obj.is_contiguous():
                if not strided:
                    raise ValueError("Expected a row-major matrix")
                strides = tuple(obj.stride())
            word = _TORCH_WORD[obj.dtype]
            if obj.is_cuda:
                dev = L.kDLCUDA | ((obj.get_device() or 0) << 32)
            else:
                dev = L.kDLCUDAHost if obj.is_pinned() else L.kDLCPU
            ptr, shape = obj.data_ptr(), tuple(obj.shape)
        elif isinstance(obj, np.ndarray):
            if not obj.flags.c_contiguous:
                raise ValueError("Expected a row-major matrix")
            word = _NP_WORD[obj.dtype]
            dev, ptr, shape = L.kDLCPU, obj.ctypes.data, obj.shape
        else:
            raise TypeError(f"unsupported array type {type(obj)}")
        n = len(shape)
        self._keep = obj
        words = (_WORDS.get(n) or C.c_int64 * (8 + 2 * n))(ptr, dev, word | n, 0, 0, 0, 0, 0, *shape, *strides)
        at = C.addressof(words)
        words[3] = at + 64
        if strides:
            words[4] = at + 64 + 8 * n
        self._words = words

    @property
    def managed(self):
        return L.DLManagedTensor.from_buffer(self._words)

    def ref(self):
        return C.byref(L.DLManagedTensor.from_buffer(self._words))


_TYPESTR = {(L.kDLFloat, 32): "<f4", (L.kDLUInt, 32): "<u4", (L.kDLInt, 64): "<i8",
            (L.kDLUInt, 8): "|u1"}


class _CudaView:
    def __init__(self, ptr, shape, typestr, strides_bytes):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False),
                                         "version": 2, "strides": strides_bytes}


def view_to_torch(mt: L.DLManagedTensor) -> torch.Tensor:
    """Copy a device view returned by a getter into an owning torch tensor, then free the view's
    shape arrays through its deleter."""
    t = mt.dl_tensor
    shape = tuple(int(t.shape[i]) for i in range(t.ndim))
    typestr = _TYPESTR[(t.dtype.code, t.dtype.bits)]
    itemsize = t.dtype.bits // 8
    strides = None
    if t.strides:
        strides = tuple(int(t.strides[i]) * itemsize for i in range(t.ndim))
    n = 1
    for s in shape:
        n *= s
    if n == 0:
        out = torch.empty(shape, dtype={"<f4": torch.float32, "<u4": torch.uint32,
                                        "<i8": torch.int64, "|u1": torch.uint8}[typestr],
                          device="cuda")
    else:
        out = torch.as_tensor(_CudaView(t.data, shape, typestr, strides), device="cuda").clone()
    if mt.deleter:
        mt.deleter(C.pointer(mt))
    return out
