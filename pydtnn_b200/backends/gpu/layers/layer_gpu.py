"""Base of the GPU layers: buffer attributes and the gradient-exchange hooks
(pydtnn/backends/gpu/layers/layer_gpu.py:36-204).

The reference all-reduces every gradient tensor separately after a host synchronisation
(:78-82).  Here a layer only tells the model's gradient bucketer that its gradients are written;
the bucketer launches one NCCL all-reduce per contiguous bucket, ordered after the producing
kernels by a stream event, so no host synchronisation happens inside a step."""
from abc import ABC

from .... import tracer
from ....layers.base import Layer
from ....tensor_gpu import ChannelLastTensor, TensorGPU, empty, transpose_inner


class LayerGPU(Layer, ABC):

    def __init__(self, *args, **kwargs):
        super().__init__(*args, **kwargs)
        self.y = None
        self.weights_cpu = None
        self.biases_cpu = None
        self.x = None
        self.dx = None
        self.dw = None
        self.db = None
        self._copies = {}

    def initialize(self, prev_shape, need_dx, x):
        self.x = x  # must be set before super().initialize()
        super().initialize(prev_shape, need_dx)

    # -- activations ---------------------------------------------------------------------
    def _activation(self, dims):
        """A buffer for an activation or its gradient (``dims`` in the model's tensor format)."""
        m = self.model
        if m.channels_last and len(dims) == 4:
            return ChannelLastTensor(dims, m.dtype, m.tensor_format)
        return TensorGPU(empty(dims, m.dtype), m.tensor_format)

    def _in(self, t, slot):
        """Address of a tensor's values in the order this layer's kernels read (channel last).  A plain NCHW tensor
        (the network's input, or one the caller made) is copied into a buffer this layer keeps per ``slot``."""
        p = t.channel_last()
        if p is None:
            n, c, h, w = t.ary.shape
            buf = self._copies.get(slot)
            if buf is None or buf.shape != (n, h, w, c):
                buf = self._copies[slot] = empty((n, h, w, c), t.ary.dtype, t.ary.t.device)
            transpose_inner(t.ary, buf, n, c, h * w)
            p = buf.gpudata
        return p

    # -- gradient exchange ---------------------------------------------------------------
    def _grad_tensors(self):
        return [getattr(self, dw_) for dw_ in self.grad_vars.values()]

    def reduce_weights_async(self):
        if self.model.comm is None or not self.grad_vars:
            return
        with self.model.tracer.op_region(self, tracer.PYDTNN_OPS_ALLREDUCE_DW):
            self.model.bucketer.mark_ready(self)

    def wait_allreduce_async(self):
        if self.model.comm is None or not self.grad_vars:
            return
        self.model.bucketer.wait_for(self)

    def reduce_weights_sync(self):
        if self.model.comm is None or not self.grad_vars:
            return
        self.model.bucketer.mark_ready(self)
        self.model.bucketer.wait_for(self)
