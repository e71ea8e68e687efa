"""GPU layers either side of the convolution: Input, BatchNormalization, Relu, Softmax, pooling,
AdditionBlock, Flatten, Dropout(identity in evaluation).  Each mirrors the attributes and hook
behaviour of its reference counterpart under pydtnn/backends/gpu/{layers,activations}/ with the
cuDNN call replaced by a call through the C ABI."""
import numpy as np

from .... import _lib
from ....layers import (AdditionBlock, AveragePool2D, BatchNormalization, Dropout, Flatten, Input, MaxPool2D, Relu,
                        Softmax)
from ....tensor_gpu import ChannelLastTensor, TensorGPU, empty, to_gpu
from ....utils import EVALUATE_MODE, TRAIN_MODE
from .. import memory_allocation as wsp
from .layer_gpu import LayerGPU


# Activations are channel-last in either tensor format (ChannelLastTensor), so the library is always called with that
# layout; a (batch, features) tensor is the case h = w = 1.

class InputGPU(LayerGPU, Input):
    """pydtnn/backends/gpu/layers/input_gpu.py:28-40"""

    def initialize(self, prev_shape, need_dx, x):
        super().initialize(prev_shape, need_dx, x)
        self.y = TensorGPU(empty((self.model.batch_size, *self.shape), self.model.dtype), self.model.tensor_format)

    def forward(self, x):
        pass

    def backward(self, dy):
        pass


class BatchNormalizationGPU(LayerGPU, BatchNormalization):
    """pydtnn/backends/gpu/layers/batch_normalization_gpu.py:36-163; arithmetic of
    pydtnn/backends/cpu/layers/batch_normalization_cpu.py:59-129."""

    def initialize(self, prev_shape, need_dx, x):
        super().initialize(prev_shape, need_dx, x)
        m = self.model
        c = self.ci
        g_arr, dg_arr = m.arena.alloc_param(np.full((c,), self.gamma_init_val, m.dtype))
        b_arr, db_arr = m.arena.alloc_param(np.full((c,), self.beta_init_val, m.dtype))
        self.gamma, self.dgamma = TensorGPU(g_arr, m.tensor_format), TensorGPU(dg_arr, m.tensor_format)
        self.beta, self.dbeta = TensorGPU(b_arr, m.tensor_format), TensorGPU(db_arr, m.tensor_format)
        self.running_mean = TensorGPU(to_gpu(self.moving_mean_initializer((c,), m.dtype)), m.tensor_format)
        self.running_var = TensorGPU(to_gpu(self.moving_variance_initializer((c,), m.dtype)), m.tensor_format)
        self.save_mean = TensorGPU(empty((c,), m.dtype), m.tensor_format)
        self.save_inv_var = TensorGPU(empty((c,), m.dtype), m.tensor_format)
        self._inv_std = empty((c,), m.dtype)
        wsp.require_reduction_scratch(c)
        self.y = self._activation(x.dims)
        if self.need_dx:
            self.dx = self._activation(x.dims)
        self.fuse_relu = False           # set by the model's fusion pass (BN followed by ReLU)
        self.prestats = None             # (buffer, bytes) left by the preceding convolution's forward pass of this step
        self.residual = None             # (other branch, output) while an addition block folds its sum + ReLU in here
        self._dt = _lib.dtype_code(m.dtype)
        self._hw = self.hi * self.wi if self.spatial else 1
        self.updated_running_var = True
        self._inv_std_step = 0           # replayed training steps of the model when _inv_std was computed

    def forward(self, x):
        m = self.model
        L = _lib.lib()
        self.x = x
        x_ptr = self._in(x, "x")
        if m.mode == TRAIN_MODE and self.prestats is not None:
            # the convolution that wrote x already summed it per channel: statistics from those sums, one pass over x
            st, nbytes = self.prestats
            self.prestats = None
            addend, out, relu = (self.residual[0], self.residual[1], 1) if self.residual is not None else (None, self.y, int(self.fuse_relu))
            _lib.check(L.b2c_bn_train_forward_prestats(
                m.batch_size, self.ci, self._hw, x_ptr, st.data_ptr(), nbytes, self.gamma.ptr, self.beta.ptr,
                self.running_mean.ptr, self.running_var.ptr, float(self.momentum), float(self.epsilon), relu,
                self._in(addend, "addend") if addend is not None else None, out.out, self.save_mean.ptr, self.save_inv_var.ptr,
                wsp.reduction_scratch().data_ptr(), wsp.reduction_scratch().numel() * 8, m.stream_handle))
            out.written()
            self.updated_running_var = True
            return out
        if m.mode == TRAIN_MODE and self.residual is not None:
            # last batch norm of a residual branch: out = relu(bn(x) + other branch), written to the block's ReLU
            addend, out = self.residual
            _lib.check(L.b2c_bn_train_forward_residual(
                self._dt, _lib.LAYOUT_NHWC, m.batch_size, self.ci, self._hw, x_ptr, self.gamma.ptr, self.beta.ptr,
                self.running_mean.ptr, self.running_var.ptr, float(self.momentum), float(self.epsilon), self._in(addend, "addend"), 1,
                out.out, self.save_mean.ptr, self.save_inv_var.ptr, wsp.reduction_scratch().data_ptr(),
                wsp.reduction_scratch().numel() * 8, m.stream_handle))
            out.written()
            self.updated_running_var = True
            return out
        if m.mode == TRAIN_MODE:
            _lib.check(L.b2c_bn_train_forward(self._dt, _lib.LAYOUT_NHWC, m.batch_size, self.ci, self._hw, x_ptr,
                                              self.gamma.ptr, self.beta.ptr, self.running_mean.ptr,
                                              self.running_var.ptr, float(self.momentum), float(self.epsilon),
                                              int(self.fuse_relu), self.y.out, self.save_mean.ptr,
                                              self.save_inv_var.ptr, wsp.reduction_scratch().data_ptr(),
                                              wsp.reduction_scratch().numel() * 8, m.stream_handle))
            self.updated_running_var = True
        elif m.mode == EVALUATE_MODE:
            _lib.check(L.b2c_bn_inference(self._dt, _lib.LAYOUT_NHWC, m.batch_size, self.ci, self._hw, x_ptr,
                                          self.running_mean.ptr, self.inference_inv_std().gpudata, self.gamma.ptr,
                                          self.beta.ptr, int(self.fuse_relu), self.y.out, m.stream_handle))
        else:
            raise ValueError("Unexpected model mode")
        self.y.written()
        return self.y

    def inference_inv_std(self):
        """1 / sqrt(running_var + eps) on the device, recomputed (one small kernel, no host round trip) only after
        the running variance changed: a training step or a checkpoint load
        (pydtnn/backends/cpu/layers/batch_normalization_cpu.py:92-94 refreshes it under the same flag)."""
        if self.updated_running_var or self._inv_std_step != self.model.replayed_steps:
            _lib.check(_lib.lib().b2c_bn_inv_std(self._dt, self.ci, self.running_var.ptr, float(self.epsilon),
                                                 self._inv_std.gpudata, self.model.stream_handle))
            self.updated_running_var = False
            self._inv_std_step = self.model.replayed_steps
        return self._inv_std

    def backward(self, dy):
        m = self.model
        _lib.check(_lib.lib().b2c_bn_train_backward(
            self._dt, _lib.LAYOUT_NHWC, m.batch_size, self.ci, self._hw,
            self._in(self.x, "x"), self._in(dy, "dy"),
            self._in(self.y, "y") if self.fuse_relu else None, self.beta.ptr if self.fuse_relu else None, self.gamma.ptr,
            self.save_mean.ptr, self.save_inv_var.ptr,
            self.dgamma.ptr, self.dbeta.ptr, self.dx.out if self.need_dx else None,
            wsp.reduction_scratch().data_ptr(), wsp.reduction_scratch().numel() * 8, m.stream_handle))
        if self.need_dx:
            self.dx.written()
            return self.dx


class ReluGPU(LayerGPU, Relu):
    """pydtnn/backends/gpu/activations/relu_gpu.py:40-68"""

    def initialize(self, prev_shape, need_dx, x):
        super().initialize(prev_shape, need_dx, x)
        m = self.model
        self.y = self._activation(x.dims)
        if self.need_dx:
            self.dx = self._activation(x.dims)
        self._dt = _lib.dtype_code(m.dtype)
        self.absorbed = False            # True when the preceding BatchNormalization applies the ReLU itself
        self.fed_by_block = False        # True when the preceding AdditionBlock writes max(sum, 0) into self.y
        self.bwd_by_block = False        # True when the following AdditionBlock writes the masked gradient into self.dx

    def forward(self, x):
        if self.absorbed:
            return x
        if self.fed_by_block:
            return self.y
        _lib.check(_lib.lib().b2c_relu_forward(self._dt, self.y.size, self._in(x, "x"), self.y.out, self.model.stream_handle))
        self.y.written()
        return self.y

    def backward(self, dy):
        if self.absorbed:
            return dy
        if self.bwd_by_block and self.model.mode == TRAIN_MODE:
            return self.dx
        if self.need_dx:
            _lib.check(_lib.lib().b2c_relu_backward(self._dt, self.y.size, self._in(dy, "dy"), self._in(self.y, "y"), self.dx.out,
                                                    self.model.stream_handle))
            self.dx.written()
            return self.dx


class SoftmaxGPU(LayerGPU, Softmax):
    """pydtnn/backends/gpu/activations/softmax_gpu.py:40-64"""

    def initialize(self, prev_shape, need_dx, x):
        super().initialize(prev_shape, need_dx, x)
        m = self.model
        self.y = TensorGPU(empty(x.dims, m.dtype), m.tensor_format)
        if self.need_dx:
            self.dx = TensorGPU(empty(x.dims, m.dtype), m.tensor_format)
        self._dt = _lib.dtype_code(m.dtype)
        self.backward_done = False       # the loss of this step has written dx already
        self._rows, self._cols = int(x.dims[0]), int(np.prod(x.dims[1:]))

    def forward(self, x):
        self.backward_done = False       # of a step that never reached this layer's backward
        _lib.check(_lib.lib().b2c_softmax_forward(self._dt, self._rows, self._cols, x.ptr, self.y.ptr,
                                                  self.model.stream_handle))
        return self.y

    def backward(self, dy):
        if self.backward_done:
            self.backward_done = False
            return self.dx
        if self.need_dx:
            _lib.check(_lib.lib().b2c_softmax_backward(self._dt, self._rows, self._cols, dy.ptr, self.y.ptr,
                                                       self.dx.ptr, self.model.stream_handle))
            return self.dx


class DropoutGPU(LayerGPU, Dropout):
    """Identity in evaluation (the only mode the supported configurations use it in)."""

    def initialize(self, prev_shape, need_dx, x):
        super().initialize(prev_shape, need_dx, x)
        self.y = x

    def forward(self, x):
        if self.model.mode == TRAIN_MODE:
            raise NotImplementedError("training-mode dropout is outside the supported path")
        return x

    def backward(self, dy):
        raise NotImplementedError("training-mode dropout is outside the supported path")


class FlattenGPU(LayerGPU, Flatten):
    """pydtnn/backends/gpu/layers/flatten_gpu.py:33-52 -- views, no copies, where the flattened order is the stored one;
    the (c, h, w) order of an NCHW model's features is copied out of the channel-last activation otherwise."""

    def initialize(self, prev_shape, need_dx, x):
        super().initialize(prev_shape, need_dx, x)
        m = self.model
        self._copied = isinstance(x, ChannelLastTensor) and not x.same_order
        if self._copied:
            self.y = TensorGPU(empty((m.batch_size, *self.shape), m.dtype), m.tensor_format)
            if self.need_dx:
                self.dx = self._activation(x.dims)
        else:
            self.y = TensorGPU(x.ary.reshape((m.batch_size, *self.shape)), m.tensor_format)

    def _chw(self):
        c, h, w = self.prev_shape
        return c, h * w

    def forward(self, x):
        m = self.model
        if self._copied:
            c, hw = self._chw()
            _lib.check(_lib.lib().b2c_transpose(_lib.dtype_code(m.dtype), m.batch_size, hw, c, self._in(x, "x"), self.y.ptr,
                                                m.stream_handle))
            return self.y
        self.y = self._view(self.y, x, (m.batch_size, *self.shape))
        return self.y

    @staticmethod
    def _view(last, t, dims):
        """``t`` with other dimensions; the handle of the last call where that still is the same memory."""
        a = t.ary
        if last is not None and last.ary.gpudata == a.gpudata and last.ary.shape == dims:
            return last
        return TensorGPU(a.reshape(dims), t.tensor_format)

    def backward(self, dy):
        m = self.model
        if self.need_dx:
            if self._copied:
                c, hw = self._chw()
                _lib.check(_lib.lib().b2c_transpose(_lib.dtype_code(m.dtype), m.batch_size, c, hw, dy.ptr, self.dx.out,
                                                    m.stream_handle))
                self.dx.written()
            else:
                self.dx = self._view(self.dx, dy, (m.batch_size, *self.prev_shape))
            return self.dx


class _Pool2DGPU(LayerGPU):
    """pydtnn/backends/gpu/layers/abstract_pool_2d_layer_gpu.py:36-102"""
    _is_max = 0

    def initialize(self, prev_shape, need_dx, x):
        super().initialize(prev_shape, need_dx, x)
        m = self.model
        self.y = self._activation((m.batch_size, *self.shape))
        if self._is_max:
            self.idx_max = empty((m.batch_size, self.ho, self.wo, self.co), np.int32)
        if self.need_dx:
            self.dx = self._activation(x.dims)
        self._dt = _lib.dtype_code(m.dtype)

    def _geom(self):
        return (self.model.batch_size, self.hi, self.wi, self.ci, self.kh, self.kw, self.vpadding, self.hpadding,
                self.vstride, self.hstride, self.vdilation, self.hdilation)

    def forward(self, x):
        m = self.model
        _lib.check(_lib.lib().b2c_pool_forward(self._dt, _lib.LAYOUT_NHWC, self._is_max, *self._geom(),
                                               self._in(x, "x"), self.y.out,
                                               # the winning taps are for backward only
                                               self.idx_max.gpudata if self._is_max and m.mode != EVALUATE_MODE else None,
                                               m.stream_handle))
        self.y.written()
        return self.y

    def backward(self, dy):
        if self.need_dx:
            m = self.model
            _lib.check(_lib.lib().b2c_pool_backward(self._dt, _lib.LAYOUT_NHWC, self._is_max, *self._geom(),
                                                    self._in(dy, "dy"), self.idx_max.gpudata if self._is_max else None,
                                                    self.dx.out, m.stream_handle))
            self.dx.written()
            return self.dx


class MaxPool2DGPU(_Pool2DGPU, MaxPool2D):
    _is_max = 1


class AveragePool2DGPU(_Pool2DGPU, AveragePool2D):
    _is_max = 0


class AdditionBlockGPU(LayerGPU, AdditionBlock):
    """pydtnn/backends/gpu/layers/addition_block_gpu.py:30-85: run every path on the block input,
    sum the outputs into the first path's output; backward mirrors it."""

    def initialize(self, prev_shape, need_dx, x):
        super().initialize(prev_shape, need_dx, x)
        m = self.model
        self.out_shapes = []
        for p_i, p in enumerate(self.paths):
            shape, cur = self.prev_shape, self.x
            for i, layer in enumerate(p):
                layer.set_model(m)
                layer.initialize(shape, self.need_dx, cur)
                cur = layer.y
                shape = layer.shape
                self.nparams += layer.nparams
                if layer.act:
                    raise NotImplementedError("activation arguments inside block paths are not supported")
            self.out_shapes.append(shape)
        assert all(o == self.out_shapes[0] for o in self.out_shapes)
        self.shape = self.out_shapes[0]
        if len(self.paths[0]) == 0:
            raise NotImplementedError("the first path of an AdditionBlock must not be empty")
        self.y = self.paths[0][-1].y
        self._dt = _lib.dtype_code(m.dtype)
        self.relu_after = None           # set by the model: the Relu layer that directly follows this block
        self.fold_sum = True             # let the first branch's last batch norm do the sum and that ReLU
        self.relu_before = None          # set by the model: the Relu layer whose output is this block's input

    def _fold_sum_into_last_bn(self):
        """Training step, two branches, the block feeds a ReLU and the first branch ends in a plain batch norm:
        that batch norm can add the other branch and apply the ReLU while it writes (one pass less over the block's
        largest tensors, and the batch-norm output itself is never stored)."""
        if self.model.mode != TRAIN_MODE or self.relu_after is None or len(self.paths) != 2 or not self.fold_sum:
            return None
        bn = self.paths[0][-1]
        if type(bn).__name__ != "BatchNormalizationGPU" or bn.fuse_relu:
            return None
        return bn

    def _add(self, acc, other):
        """acc += other, in the buffer ``acc`` is kept in."""
        if acc.channel_last() is not None:
            _lib.check(_lib.lib().b2c_add_inplace(self._dt, acc.size, acc.out, self._in(other, "other"), self.model.stream_handle))
            acc.written()
        else:
            _lib.check(_lib.lib().b2c_add_inplace(self._dt, acc.size, acc.ptr, other.ptr, self.model.stream_handle))

    def forward(self, x):
        L = _lib.lib()
        bn = self._fold_sum_into_last_bn()
        if bn is not None:
            other = x
            for layer in self.paths[1]:
                other = layer.forward(other)
            bn.residual = (other, self.relu_after.y)
            y = x
            for layer in self.paths[0]:
                y = layer.forward(y)
            bn.residual = None
            self.y = y
            return self.y
        last = len(self.paths) - 1
        for i, p in enumerate(self.paths):
            y_i = x
            for layer in p:
                y_i = layer.forward(y_i)
            if i == 0:
                self.y = y_i
            elif i == last and self.relu_after is not None:
                # residual sum and the ReLU that follows in one pass: relu.y = max(y + y_i, 0)
                _lib.check(L.b2c_add_relu(self._dt, self.y.size, self._in(self.y, "y"), self._in(y_i, "other"),
                                          self.relu_after.y.out, self.model.stream_handle))
                self.relu_after.y.written()
            else:
                self._add(self.y, y_i)
        return self.y

    def backward(self, dy):
        L = _lib.lib()
        dx0 = None
        for i, p in enumerate(self.paths):
            dx_i = dy
            for layer in reversed(p):
                dx_i = layer.backward(dx_i)
            if i == 0:
                dx0 = dx_i
            elif i == len(self.paths) - 1 and self.relu_before is not None:
                # the sum of the branch gradients and the backward of the ReLU that feeds this block in one pass
                r = self.relu_before
                _lib.check(L.b2c_add_relu_backward(self._dt, dx0.size, self._in(dx0, "dx0"), self._in(dx_i, "other"),
                                                   self._in(r.y, "relu"), r.dx.out, self.model.stream_handle))
                r.dx.written()
            else:
                self._add(dx0, dx_i)
        self.dx = dx0
        return dx0

    def update_weights(self, optimizer):
        for layer in self.children:
            layer.update_weights(optimizer)

    def reduce_weights_async(self):
        for layer in self.children:
            layer.reduce_weights_async()

    def wait_allreduce_async(self):
        for layer in self.children:
            layer.wait_allreduce_async()

    def reduce_weights_sync(self):
        for layer in self.children:
            layer.reduce_weights_sync()
