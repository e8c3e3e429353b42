"""``inv`` and ``cholesky`` with the signatures of torchsso/utils/inv_cupy.py:27-34 and
torchsso/utils/cholesky_cupy.py:9-14, executed by the tile-task engine of libsso_b200.

``inv(m)`` returns a new tensor holding the inverse of the SPD matrix ``m`` (input untouched);
``cholesky(m, upper=True)`` returns the upper factor U with U^T U = m (or the lower factor).
Both are one-matrix conveniences; the optimizers invert all layers in one batched plan."""
from __future__ import annotations

import torch

from .. import _native as nat

_cache = {}


def _solo(d: int, device, upper: bool):
    key = (d, device.index, upper)      # a plan that can factor inverts in reverse order, which an inverse alone need not pay for
    ent = _cache.get(key)
    if ent is None:
        src, dst = (torch.empty((d, d), dtype=torch.float32, device=device) for _ in range(2))
        std = torch.empty_like(src) if upper else None
        direct = not nat.kron_plan_uses_work()
        work = None if direct else [torch.empty_like(src)]
        plan = nat.kron_plan([d], [src], [dst], work, [std] if upper else None, [-1], [0], device)
        zero = torch.zeros(1, dtype=torch.float32, device=device)
        info = torch.zeros(2, dtype=torch.int32, device=device)
        ent = (plan, src, dst, std, zero, info, direct)
        if len(_cache) > 16:
            _cache.clear()
        _cache[key] = ent
    return ent


def _run(m: torch.Tensor, upper: bool) -> torch.Tensor:
    m = m.detach()
    plan, src, dst, std, zero, info, direct = _solo(m.shape[0], m.device, upper)
    if not direct:
        (dst if upper else src).copy_(m)      # the factorisation stage reads the "inverse" slot
        nat.kron_plan_run(plan, zero, info, not upper, upper)
        return (std if upper else dst).clone()
    # read where it lies, if the kernel can read it as fast as a copy
    aligned = m.data_ptr() % 16 == 0 and m.stride(0) % 4 == 0 or m.shape[0] % 4 != 0
    if m.dtype != torch.float32 or m.stride(1) != 1 or not m.shape[0] <= m.stride(0) < 1 << 31 or not aligned:
        m = src.copy_(m)
    out = torch.empty_like(src)
    nat.kron_plan_run_at(plan, zero, info, not upper, m, out)
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
