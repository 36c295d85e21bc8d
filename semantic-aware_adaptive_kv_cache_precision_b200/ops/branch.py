"""Two pieces of a captured decode step side by side.

The kernels of a step of few tokens fill a small part of the GPU each, and in plain stream order each of
them waits for the one before, needed or not. Inside a CUDA graph a piece of work whose result is read
later can be a branch of its own: it is captured on another stream, which joins the first one where the
result is read."""

from __future__ import annotations

import ctypes
import threading

import torch

from ._lib import KernelError, plain_function

_local = threading.local()      # `streams`: a thread's own; `open`: its branches not yet joined
_idle: dict = {}                # streams of threads that have ended, by device
_idle_lock = threading.Lock()


class _Streams:
    """One thread's streams for branches, by device, outermost first. They are not from PyTorch's pool, which
    deals its streams out again: what another thread launched on such a stream while this one captures on
    it would be captured with it. A thread that ends leaves them to the next."""

    def __init__(self):
        self.of: dict = {}

    def beside(self, main: torch.cuda.Stream) -> torch.cuda.Stream:
        """The first of `main`'s device, or if `main` is one of them (a branch inside a branch) the one
        after it."""
        streams = self.of.setdefault(main.device, [])
        at = next((i + 1 for i, s in enumerate(streams) if s.cuda_stream == main.cuda_stream), 0)
        if at == len(streams):
            with _idle_lock:
                idle = _idle.setdefault(main.device, [])
                stream = idle.pop() if idle else None
            streams.append(stream if stream is not None else self._make(main.device))
        return streams[at]

    @staticmethod
    def _make(device) -> torch.cuda.Stream:
        handle = ctypes.c_void_p()
        with torch.cuda.device(device):
            code = plain_function("sakv_stream_create")(ctypes.addressof(handle))
        if code != 0:
            raise KernelError(f"could not make a stream (CUDA error {code})")
        return torch.cuda.ExternalStream(handle.value, device)

    def __del__(self):
        with _idle_lock:
            for device, streams in self.of.items():
                _idle.setdefault(device, []).extend(streams)


def _other_stream(main: torch.cuda.Stream) -> torch.cuda.Stream:
    kept = getattr(_local, "streams", None)
    if kept is None:
        kept = _local.streams = _Streams()
    return kept.beside(main)


def apart() -> bool:
    """Whether what this thread launches now may run at the same time as another piece of its step (a
    branch that is not joined yet). Scratch memory that calls share, one after another in stream order,
    is not to be used then."""
    return getattr(_local, "open", 0) > 0


class Aside:
    """What `aside` started. As a context: the stream it started from waits for it at the end (also when
    something fails in between: what is captured then can still be ended, and the failure is what the
    caller sees); from there on `result` may be read."""

    __slots__ = ("result", "main", "stream")

    def __init__(self, main=None, stream=None):
        self.result, self.main, self.stream = None, main, stream

    def __enter__(self):
        return self

    def __exit__(self, kind, value, trace):
        if self.stream is not None:
            _local.open -= 1
            stream, self.stream = self.stream, None
            try:
                self.main.wait_stream(stream)
            except Exception:
                if kind is None:           # (else the capture itself has failed, and `value` says why)
                    raise
        return False


def goes_aside(step, tokens: int) -> bool:
    """Whether `aside` gives work of this step a branch of its own: a decode step of few tokens that is
    being captured."""
    from .linear import TC_MAX_TOKENS
    return bool(getattr(step, "is_decode", False)) and tokens <= TC_MAX_TOKENS \
        and torch.cuda.is_current_stream_capturing()


def aside(work, step, tokens: int) -> Aside:
    """`with aside(work, step, tokens) as beside: ...`: start `work()` beside what is launched in the
    context; where it has no branch of its own (`goes_aside`), run it here and now. `work` None: nothing.

    Memory: the caller keeps whatever `work` reads until the context ends. `work`'s launches come before the
    main path's, so what the main path gives back meanwhile can only be given to a later branch, which
    begins after it; what the branch itself made is given to later branches only, which begin after
    whoever read it. Neither side uses memory that calls share (`apart`)."""
    if work is None or not goes_aside(step, tokens):
        beside = Aside()
        beside.result = work() if work is not None else None
        return beside
    main = torch.cuda.current_stream()
    stream = _other_stream(main)
    stream.wait_stream(main)
    _local.open = getattr(_local, "open", 0) + 1
    beside = Aside(main, stream)
    try:
        with torch.cuda.stream(stream):
            beside.result = work()
    except BaseException as failure:
        beside.__exit__(type(failure), failure, None)
        raise
    return beside
