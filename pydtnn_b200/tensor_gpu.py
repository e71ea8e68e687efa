"""Device tensor handle with the attributes the reference's ``TensorGPU`` exposes
(pydtnn/backends/gpu/tensor_gpu.py:31-66): ``.ary`` (device array with ``shape``, ``size``,
``get()``, ``set()``, ``reshape()``, ``gpudata``), ``.ptr`` (``ctypes.c_void_p``), ``.size`` and a
``.shape`` promoted to 4-D.  Storage comes from ``torch.empty``; torch is used for allocation and
host<->device copies only.
"""
import ctypes

import numpy as np
import torch

from . import _lib
from .utils import PYDTNN_TENSOR_FORMAT_NCHW

_TORCH_DTYPE = {np.dtype(np.float32): torch.float32, np.dtype(np.float64): torch.float64,
                np.dtype(np.int32): torch.int32, np.dtype(np.int64): torch.int64}


class Storage:
    #: counts, over the process, the times a tensor handle that is no model's (or several models') came to stand for other
    #: memory: recorded launches are only valid while this has not moved.  Handles of one model count as its layers' edits.
    moves = 0


class _Owned:
    owner = None

    def owned_by(self, model):
        """Says whose recorded passes read or write this memory; a handle of two models is nobody's."""
        object.__setattr__(self, "owner", model if self.__dict__.get("owner", model) is model else None)

    def _moved(self):
        if self.owner is not None:
            self.owner.layer_edits += 1
        else:
            Storage.moves += 1

    def _hand_on(self, other):
        if "owner" in self.__dict__:
            other.owned_by(self.owner)


class DeviceArray(_Owned):
    """Stands in for ``pycuda.gpuarray.GPUArray`` for the members the layer code touches."""

    def __init__(self, tensor: torch.Tensor):
        assert tensor.is_contiguous()
        self.t = tensor

    def __setattr__(self, name, value):
        if name in self.__dict__:
            self._moved()
        object.__setattr__(self, name, value)

    @property
    def shape(self):
        return tuple(self.t.shape)

    @property
    def size(self):
        return self.t.numel()

    @property
    def dtype(self):
        return {v: k for k, v in _TORCH_DTYPE.items()}[self.t.dtype]

    @property
    def gpudata(self):
        return self.t.data_ptr()

    def get(self):
        return self.t.detach().cpu().numpy()

    def set(self, host):
        src = torch.from_numpy(np.ascontiguousarray(host, dtype=self.dtype)).reshape(self.t.shape)
        self.t.copy_(src, non_blocking=True)

    def set_async(self, host, stream=None):
        self.set(host)

    def reshape(self, shape):
        return DeviceArray(self.t.view(*shape))

    def fill(self, value):
        self.t.fill_(value)
        return self


def empty(shape, dtype, device=None):
    device = device or torch.device("cuda", torch.cuda.current_device())
    return DeviceArray(torch.empty(tuple(int(s) for s in shape), dtype=_TORCH_DTYPE[np.dtype(dtype)], device=device))


def zeros(shape, dtype, device=None):
    return empty(shape, dtype, device).fill(0)


def to_gpu(host, device=None):
    a = empty(host.shape, host.dtype, device)
    a.set(host)
    return a


class TensorGPU(_Owned):
    def __init__(self, gpu_arr: DeviceArray, tensor_format, cudnn_dtype=None, tensor_type="tensor", desc=None,
                 gpudirect=False, cublas=False):
        if len(gpu_arr.shape) == 2:
            if tensor_format == PYDTNN_TENSOR_FORMAT_NCHW:
                self.shape = (*gpu_arr.shape, 1, 1)
            else:
                self.shape = (gpu_arr.shape[0], 1, 1, gpu_arr.shape[1])
        else:
            self.shape = gpu_arr.shape
        self.size = gpu_arr.size
        self.ary = gpu_arr
        self.tensor_format = tensor_format
        self.tensor_type = tensor_type
        self.desc = desc

    def __setattr__(self, name, value):
        if name == "ary":
            if "ary" in self.__dict__:
                self._moved()
            self._hand_on(value)
        object.__setattr__(self, name, value)

    def owned_by(self, model):
        super().owned_by(model)
        for array in map(self.__dict__.get, ("ary", "_cl", "_nchw")):
            if array is not None:
                array.owned_by(model)

    @property
    def ptr(self):
        return ctypes.c_void_p(self.ary.gpudata)

    def reshape(self, shape):
        self.ary = self.ary.reshape(shape)
        return self

    # -- what the layers' kernels read and write (see ChannelLastTensor) --------------------------------------
    @property
    def dims(self):
        """Shape without the promotion to 4-D."""
        return self.ary.shape

    def channel_last(self):
        """Address of the values with the channel axis last, or None where they are stored otherwise."""
        t = self.ary.t
        if self.tensor_format == PYDTNN_TENSOR_FORMAT_NCHW and t.dim() == 4:
            _, c, h, w = t.shape
            if c != 1 and h * w != 1:
                return None
        return t.data_ptr()

    @property
    def out(self):
        """Address a layer's kernel writes to; ``written()`` follows the call."""
        return self.ary.gpudata

    def written(self):
        pass


def transpose_inner(src, dst, n, rows, cols):
    """dst[n][cols][rows] = src[n][rows][cols] (device arrays), on the current stream."""
    _lib.check(_lib.lib().b2c_transpose(_lib.dtype_code(src.dtype), n, rows, cols, src.gpudata, dst.gpudata,
                                        torch.cuda.current_stream(src.t.device).cuda_stream))


class ChannelLastTensor(TensorGPU):
    """An (n, c, h, w) activation of an NCHW model whose values are kept channel-last between the layers: every kernel
    of this package runs channel-last, and in a network all neighbours of an activation are such kernels, so copying
    each tensor to NCHW and back around every layer would be most of the step (measured on a ResNet-50 step, batch 32:
    27.8 ms with NCHW storage).

    Whoever looks at the tensor (``ary``, ``ptr``) gets a real NCHW buffer: it is made at the first look and from then
    on the tensor is an NCHW buffer to everyone -- a layer that writes it brings the buffer up to date in the same call,
    a layer that reads it takes what the buffer holds, so the caller may also write to it."""

    def __init__(self, dims, dtype, tensor_format, tensor_type="tensor"):
        n, c, h, w = dims
        self._dims = self.shape = tuple(int(d) for d in dims)
        self.size = n * c * h * w
        self.tensor_format, self.tensor_type, self.desc = tensor_format, tensor_type, None
        self._cl = empty((n, h, w, c), dtype)
        self.same_order = c == 1 or h * w == 1              # both orders are the same bytes
        self._nchw = DeviceArray(self._cl.t.view(self._dims)) if self.same_order else None

    @property
    def ary(self):
        if self._nchw is None:
            n, c, h, w = self._dims
            self._nchw = empty(self._dims, self._cl.dtype, self._cl.t.device)
            self._hand_on(self._nchw)
            self._moved()
            transpose_inner(self._cl, self._nchw, n, h * w, c)
        return self._nchw

    @property
    def dims(self):
        return self._dims

    def channel_last(self):
        if self._nchw is not None and not self.same_order:
            n, c, h, w = self._dims
            transpose_inner(self._nchw, self._cl, n, c, h * w)
        return self._cl.gpudata

    @property
    def out(self):
        return self._cl.gpudata

    def written(self):
        if self._nchw is not None and not self.same_order:
            n, c, h, w = self._dims
            transpose_inner(self._cl, self._nchw, n, h * w, c)

    def reshape(self, shape):
        return TensorGPU(self.ary.reshape(shape), self.tensor_format, tensor_type=self.tensor_type)
