"""Which operands a kernel may read before its predecessor on the stream has ended.

The kernels of the decoding path are launched while their predecessor drains. Some ask for operands ahead of their wait for it:
the linears for their first weights, the decoding attentions for positions and cached keys. That is right if the operand was
complete before the predecessor STARTED, which nothing but the order of the launches says: the weight of a linear is any tensor
of a graph, and a gather or another linear may have written it in the launch before. A `LaunchOrder` follows that order for the
ops that a session executes: an operand may be read ahead if, since the last op that had it among its inputs or outputs, at
least one kernel of this library was launched on the same stream. (Each of them starts after all earlier work of its stream has
ended, or waits for it before it lets its successor start.) Without a `LaunchOrder`, in direct calls of a kernel, nothing is
read ahead.

A captured graph keeps what was decided when it was captured. It starts when all that was queued before it has ended, so only
the order inside it counts. Work on other streams is joined by events, which a launch waits for in full.
"""
import threading
from contextlib import contextmanager
from typing import Dict, Tuple

import torch

# Ops whose kernels read ahead, and the inputs among those that they only read: such an op does not hold up the next reader.
READERS: Dict[str, Tuple[int, ...]] = {
    "linear_rows": (1,), "linear_swiglu": (1,), "linear_split_glu": (1,), "linear_residual_dyt_": (2,), "linear_residual_rms_": (2,),
    "min_gru_": (1,), "linear_gq": (1, 2, 3), "linear_gq_window": (1, 2, 3), "linear_gq_window_t": (1, 2),
    "diff_attention_": (), "window_attention_": (), "rotary_attention_decode_into_": (),
}

_THREAD = threading.local()


def _storages(values):
    """Storages of tensors in nested lists."""
    for v in values:
        if isinstance(v, torch.Tensor):
            yield v.untyped_storage().data_ptr()
        elif isinstance(v, (list, tuple)):
            yield from _storages(v)


class LaunchOrder:
    """What ops had in hand since this library's latest launch on one stream (CUDA handle; 0 on the CPU)."""

    def __init__(self, stream: int = 0):
        self.stream, self.launches = stream, 0
        self._recent: list = []  # values of ops, as they came: most launches forget them unseen

    def launched(self, stream: int) -> None:
        if stream == self.stream:
            self.launches += 1
            self._recent.clear()

    def touch(self, *values) -> None:
        """An op that has just run had `values` (tensors, or lists of them) among its inputs and outputs."""
        self._recent.extend(values)
        if len(self._recent) > 64:  # a long row of ops without a launch: do not keep their tensors
            self._recent = [frozenset(_storages(self._recent)).union(*(v for v in self._recent if isinstance(v, frozenset)))]

    def complete(self, t: torch.Tensor) -> bool:
        if self.launches == 0:  # what was queued before this run may be the writer
            return False
        if t.is_cuda and torch.cuda.current_stream(t.device).cuda_stream != self.stream:
            return False
        at = t.untyped_storage().data_ptr()
        return not any(at in v for v in self._recent if isinstance(v, frozenset)) and at not in _storages(self._recent)


@contextmanager
def following(order):
    """Kernels launched by this thread are counted by `order`, and ask it what they may read ahead (None: nothing)."""
    before = getattr(_THREAD, "order", None)
    _THREAD.order = order
    try:
        yield order
    finally:
        _THREAD.order = before


def current():
    return getattr(_THREAD, "order", None)


def allowed(*tensors) -> bool:
    """Whether the next kernel of this thread may read all of `tensors` before its predecessor has ended."""
    order = current()
    return order is not None and all(order.complete(t) for t in tensors if t is not None)
