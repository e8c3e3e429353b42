"""``inv`` and ``cholesky`` with the signatures of torchsso/utils/inv_cupy.py:27-34 and
torchsso/utils/cholesky_cupy.py:9-14, executed by the tile-task engine of libsso_b200.

``inv(m)`` returns a new tensor holding the inverse of the SPD matrix ``m`` (input untouched);
``cholesky(m, upper=True)`` returns the upper factor U with U^T U = m (or the lower factor).
Both are one-matrix conveniences; the optimizers invert all layers in one batched plan."""
from __future__ import annotations

import threading
from collections import OrderedDict

import torch

from .. import _native as nat

_cache = OrderedDict()      # a plan for each size, device and direction, the one that was used longest ago first
_LIMIT = 34                 # inverses and factors of 17 sizes
_captured = {}              # plans that graphs run: these stay, and calls outside of graphs get others
_lock = threading.Lock()


class _Turns:
    """Runs of a plan share its scratch and its counters: each waits for the one before, whatever stream that is on."""

    def __init__(self, device, buffers):
        self.stream, self.raw = torch.cuda.current_stream(device), nat._stream()
        self.done, self.buffers = torch.cuda.Event(), buffers

    def begin(self, raw: int):
        if raw == self.raw:
            return
        if not self.raw:
            self.done.record(self.stream)
        self.stream, self.raw = torch.cuda.current_stream(), raw
        self.stream.wait_event(self.done)
        for b in self.buffers:
            b.record_stream(self.stream)      # their memory is not another tensor's before this run has ended

    def end(self):
        if self.raw:      # the default stream can still be asked when it matters (an event is 2 us); others may be gone then
            self.done.record(self.stream)


def _solo(d: int, device, upper: bool):
    key = (d, device.index, upper)      # a plan that can factor inverts in reverse order, which an inverse alone need not pay for
    ent = _cache.get(key)
    if ent is not None:
        _cache.move_to_end(key)
        return ent
    zero = torch.zeros(1, dtype=torch.float32, device=device)
    info = torch.zeros(2, dtype=torch.int32, device=device)
    direct = not nat.kron_plan_uses_work()
    src = dst = std = work = None
    if direct:
        # every run brings its matrix and its result (_run): the plan has none of its own, and these addresses are not used
        none = [zero.data_ptr()]
        plan = nat.kron_plan([d], none, none, None, none if upper else None, [-1], [0], device, lds=[d])
    else:
        src, dst, work = (torch.empty((d, d), dtype=torch.float32, device=device) for _ in range(3))
        std = torch.empty_like(src) if upper else None
        plan = nat.kron_plan([d], [src], [dst], [work], [std] if upper else None, [-1], [0], device)
    buffers = [t for t in (plan._dev_mem, zero, info, src, dst, std, work) if t is not None]
    ent = (plan, src, dst, std, zero, info, _Turns(device, buffers))
    while len(_cache) >= _LIMIT:
        _cache.popitem(last=False)
    _cache[key] = ent
    return ent


def _graph_plan(m: torch.Tensor, upper: bool):
    key = (m.shape[0], m.device.index, upper)
    ent = _captured.get(key)
    if ent is None:
        ent = _captured[key] = _solo(m.shape[0], m.device, upper)
        del _cache[key]
    return ent


def _run(m: torch.Tensor, upper: bool) -> torch.Tensor:
    m = m.detach()
    raw = nat._stream()
    capturing = raw != 0 and torch.cuda.is_current_stream_capturing()
    with _lock:
        plan, src, dst, std, zero, info, turns = _graph_plan(m, upper) if capturing else _solo(m.shape[0], m.device, upper)
        if not capturing:      # a graph's runs follow one another where it is replayed
            turns.begin(raw)
        if src is None:
            # read where it lies, if the kernel can read it as fast as a copy
            aligned = m.data_ptr() % 16 == 0 and m.stride(0) % 4 == 0 or m.shape[0] % 4 != 0
            if m.dtype != torch.float32 or m.is_neg() or m.stride(1) != 1 or not m.shape[0] <= m.stride(0) < 1 << 31 or not aligned:
                m = torch.empty(m.shape, dtype=torch.float32, device=m.device).copy_(m)
            out = torch.empty_like(m)
            nat.kron_plan_run_at(plan, zero, info, not upper, m, out)
        else:
            (dst if upper else src).copy_(m)      # the factorisation stage reads the "inverse" slot
            nat.kron_plan_run(plan, zero, info, not upper, upper)
            out = (std if upper else dst).clone()
        if not capturing:
            turns.end()
    return out


def inv(m: torch.Tensor) -> torch.Tensor:
    if not m.is_cuda:
        raise RuntimeError('torchsso.utils.inv needs a CUDA tensor (no CPU path in this build)')
    assert m.dim() == 2 and m.shape[0] == m.shape[1]
    return _run(m, False)


def cholesky(m: torch.Tensor, upper: bool = True) -> torch.Tensor:
    if not m.is_cuda:
        raise RuntimeError('torchsso.utils.cholesky needs a CUDA tensor (no CPU path in this build)')
    assert m.dim() == 2 and m.shape[0] == m.shape[1]
    out = _run(m, True)
    return out if upper else out.t()
