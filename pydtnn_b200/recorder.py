"""Replays a pass over the layers as one CUDA graph.

A step issues the same launches with the same arguments every time: all buffers are allocated once, and what does change
from step to step (inputs, labels, the optimiser's scalars) lives in device memory or is issued outside.  From Python
that costs 5 to 20 us of host time per launch (a ResNet-50 step: 11.5 ms, a three-layer classifier: 0.3 ms, longer
than its kernels run), so after ``WARM`` passes the model records one pass and replays it from then on.

What a recording depends on is summed up in its key.  A changed key (an attribute of a layer, a flag of the model, a grown
workspace, a first look at an activation) drops the recording, and the passes that follow are issued one by one until
the new key has been seen often enough.  Only the model's own pass is recorded; hooks called one by one are not."""
import warnings

import torch

from . import _lib

WARM = 2                 # passes issued one by one before a key is recorded


class Recorder:
    def __init__(self, model):
        self.model = model
        self.key, self.seen = None, 0
        self.graph, self.result, self.keep, self.launches = None, None, None, 0
        self.off = False

    def run(self, key, keep, issue):
        """``issue()``, or the replay of an earlier call of it with this key.  ``keep``: tensors the launches read or write
        that nothing else may own for as long as the recording lives."""
        if torch.cuda.is_current_stream_capturing():         # a caller's own recording takes the launches themselves
            return issue()
        if self.graph is not None and key == self.key:
            self.graph.replay()
            _lib.lib().b2c_note_launches(self.launches)
            return self.result
        if self.off:
            return issue()
        if key != self.key:
            self.key, self.seen, self.graph, self.result, self.keep = key, 0, None, None, None
        self.seen += 1
        if self.seen <= WARM:
            return issue()
        return self._record(keep, issue)

    def _record(self, keep, issue):
        m = self.model
        parts = [*m.get_all_layers(), *([m.loss_func] if m.loss_func is not None else [])]
        if not all(type(p).__module__.startswith(__package__ + ".") and "forward" not in p.__dict__ and "backward" not in p.__dict__
                   for p in parts):
            self.off = True              # a caller's own layer may do anything on the host
            return issue()
        L, dev = _lib.lib(), m.device
        graph, before = torch.cuda.CUDAGraph(), L.b2c_launch_count()
        stream = _capture_stream(dev)
        stream.wait_stream(torch.cuda.current_stream(dev))
        try:
            with torch.cuda.stream(stream):
                graph.capture_begin(capture_error_mode="thread_local")
                try:
                    result = issue()
                finally:
                    graph.capture_end()
        except RuntimeError as e:
            # a pass that cannot be captured (a layer that allocates or synchronises) is issued one by one for good
            self.off = True
            m._side_pending = None       # an event of the recording that never was
            warnings.warn(f"passes of this model are not recorded: {e.__context__ or e}", RuntimeWarning, stacklevel=2)
            return issue()
        self.graph, self.result, self.keep, self.launches = graph, result, keep, L.b2c_launch_count() - before
        graph.replay()
        return result


_streams = {}


def _capture_stream(device):
    """One stream per device to record on: kernels of one stream share the library's hand-over flags, and recordings of
    different models that are replayed one after the other may share them too, as they share the workspaces."""
    if device not in _streams:
        _streams[device] = torch.cuda.Stream(device=device)
    return _streams[device]
