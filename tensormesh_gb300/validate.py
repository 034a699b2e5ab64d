"""Host-side input validation with clear errors.

The reference indexes its tensors with the connectivity directly and fails
deep inside torch (or silently reads another row) when an element lists a
node that does not exist; non-finite coefficients flow through to NaN
matrices.  Here both are rejected before any kernel launch:

* connectivity: every index in [0, n_points), checked once per mesh when the
  pattern is built (``IndexError``);
* floating inputs of a call (points, per-element / per-point / per-quadrature
  coefficients): all finite (``ValueError`` naming the input).  This check
  reads the inputs on the device (one launch, tm_check_finite) and waits for
  the answer (one host synchronisation per call, after the call's own kernels
  are queued); ``set_input_checks(False)`` turns it off for callers that
  pipeline many calls and validate their data elsewhere.
"""
from __future__ import annotations

import threading
from typing import Iterable, Optional, Tuple

import torch

_CHECK_FINITE = True


def set_input_checks(enabled: bool) -> None:
    """Turn the per-call finiteness check on or off (on by default)."""
    global _CHECK_FINITE
    _CHECK_FINITE = bool(enabled)


def input_checks_enabled() -> bool:
    return _CHECK_FINITE


def check_connectivity(elements: torch.Tensor, n_points: int) -> None:
    if elements.numel() == 0:
        return
    lo, hi = int(elements.min()), int(elements.max())
    if lo < 0 or hi >= n_points:
        bad = lo if lo < 0 else hi
        row = int(torch.nonzero((elements < 0) | (elements >= n_points), as_tuple=True)[0][0])
        raise IndexError(f"element {row} refers to node {bad}, outside [0, {n_points}) "
                         f"(the mesh has {n_points} points)")


_KERNEL_DTYPES = {torch.float32: 0, torch.float64: 1}   # TM_F32, TM_F64
_LOCAL = threading.local()


def _flag_buffers(device) -> list:
    """This thread's idle (pinned flags, their numpy view, event) for
    ``device``.  A check takes one until its answer has been read: the body
    may run further checks (a saved-tensor hook that calls an assembler), and
    those take another."""
    return _LOCAL.__dict__.setdefault("flags", {}).setdefault(str(device), [])


class finite_check:
    """Context that checks named inputs while the body queues its kernels: the
    check is launched on entry, the answer is waited for on exit (ValueError
    naming the first input that holds a nan or inf).

        with finite_check(("points", points), ("the coefficient", coef)):
            launch(...)
    """

    def __init__(self, *items: Tuple[str, Optional[torch.Tensor]]):
        self.items, self.pending = items, None

    def __enter__(self):
        if not _CHECK_FINITE:
            return self
        named = [(n, t.detach()) for n, t in self.items
                 if t is not None and torch.is_tensor(t) and t.is_floating_point() and t.numel()]
        if not named:
            return self
        dev = named[0][1].device
        if (dev.type != "cuda" or len(named) > 2 or
                any(t.device != dev or t.dtype not in _KERNEL_DTYPES or not t.is_contiguous() for _, t in named)):
            check_finite(self.items)
            return self
        from . import _lib
        idle = _flag_buffers(dev)
        if idle:
            buffer = idle.pop()
        else:
            pinned = torch.zeros(2, dtype=torch.int32, pin_memory=True)
            buffer = (pinned, pinned.numpy(), torch.cuda.Event())
        flags, view, event = buffer
        view[:] = 0
        (_, a), (_, b) = named[0], (named[1] if len(named) > 1 else (None, None))
        _lib.call("tm_check_finite", _KERNEL_DTYPES[a.dtype], a.numel(), a.data_ptr(),
                  _KERNEL_DTYPES[a.dtype if b is None else b.dtype], 0 if b is None else b.numel(),
                  0 if b is None else b.data_ptr(), flags.data_ptr(), _lib.stream_handle(dev))
        event.record(torch.cuda.current_stream(dev))
        self.pending = (named, buffer, idle)
        return self

    def __exit__(self, kind, *_):
        if self.pending is None:
            return
        named, buffer, idle = self.pending
        view, event = buffer[1:]
        event.synchronize()   # also when the body raised: the flags serve another check next
        bad = [bool(v) for v in view]
        idle.append(buffer)
        if kind is None and any(bad):
            raise ValueError(f"{named[0 if bad[0] else 1][0]} holds a non-finite value (nan or inf)")


def check_finite(items: Iterable[Tuple[str, Optional[torch.Tensor]]]) -> None:
    if not _CHECK_FINITE:
        return
    named = [(n, t) for n, t in items if t is not None and torch.is_tensor(t) and t.is_floating_point() and t.numel()]
    if not named:
        return
    flags = torch.stack([torch.isfinite(t.detach()).all() for _, t in named])
    if bool(flags.all()):
        return
    first = int(torch.nonzero(~flags, as_tuple=True)[0][0])
    raise ValueError(f"{named[first][0]} holds a non-finite value (nan or inf)")
