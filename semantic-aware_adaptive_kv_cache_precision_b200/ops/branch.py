"""Two pieces of a captured decode step side by side.

The kernels of a step of few tokens fill a small part of the GPU each, and in plain stream order each of
them waits for the one before, needed or not. Inside a CUDA graph a piece of work whose result is read
later can be a branch of its own: it is captured on another stream, which joins the first one where the
result is read."""

from __future__ import annotations

import threading

import torch

_local = threading.local()      # `streams`: a thread's own, by device; `open`: its branches not yet joined


def _other_stream(main: torch.cuda.Stream) -> torch.cuda.Stream:
    """A stream for work beside `main`'s: the first of this thread's and device's, or if `main` is one of
    them (a branch inside a branch) the one after it."""
    kept = getattr(_local, "streams", None)
    if kept is None:
        kept = _local.streams = {}
    streams = kept.setdefault(main.device, [])
    at = next((i + 1 for i, s in enumerate(streams) if s == main), 0)
    if at == len(streams):
        streams.append(torch.cuda.Stream(main.device))
    return streams[at]


def apart() -> bool:
    """Whether what this thread launches now may run at the same time as another piece of its step (a
    branch that is not joined yet). Scratch memory that calls share, one after another in stream order,
    is not to be used then."""
    return getattr(_local, "open", 0) > 0


class Aside:
    """What `aside` started; `join()` lets the stream it started from wait for it and gives its result."""

    __slots__ = ("result", "main", "stream")

    def __init__(self, result, main=None, stream=None):
        self.result, self.main, self.stream = result, main, stream

    def join(self):
        if self.stream is not None:
            _local.open -= 1
            stream, self.stream = self.stream, None
            self.main.wait_stream(stream)
        return self.result


def goes_aside(step, tokens: int) -> bool:
    """Whether `aside` gives work of this step a branch of its own: a decode step of few tokens that is
    being captured."""
    from .linear import TC_MAX_TOKENS
    return bool(getattr(step, "is_decode", False)) and tokens <= TC_MAX_TOKENS \
        and torch.cuda.is_current_stream_capturing()


def aside(work, step, tokens: int) -> Aside:
    """Start `work()` beside what the caller launches from here to `join()`; where it has no branch of its
    own (`goes_aside`), run it here and now.

    Memory: the caller keeps whatever `work` reads until it has joined. `work`'s launches come before the
    main path's, so what the main path gives back meanwhile can only be given to a later branch, which
    begins after it; what the branch itself made is given to later branches only, which begin after
    whoever read it. Neither side uses memory that calls share (`apart`)."""
    if not goes_aside(step, tokens):
        return Aside(work())
    main = torch.cuda.current_stream()
    stream = _other_stream(main)
    stream.wait_stream(main)
    _local.open = getattr(_local, "open", 0) + 1
    try:
        with torch.cuda.stream(stream):
            result = work()
    except BaseException:
        _local.open -= 1
        raise
    return Aside(result, main, stream)
