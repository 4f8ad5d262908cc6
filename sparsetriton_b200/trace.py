"""Per-stage device timing of the hot path.

    with trace.recording() as rec:
        ... run convolutions ...
    rec.summary()  -> {stage: {"calls": n, "ms": total, "launches": n_kernels, "work": flops or bytes}}

Each C-ABI call site is wrapped in `trace.stage(name)`.  When no recording is active the wrapper
does nothing; when one is, it brackets the call with CUDA events on the current stream (the stream
the kernels are launched on) and reads the library's own launch counter before and after, so
"launches" is the number of kernels the library really enqueued.  The native host side brackets its own calls the
same way while a recording is open.
"""
import contextlib

import torch

from sparsetriton_b200 import _lib

_active = None


class Recording:
    def __init__(self):
        self.spans = []          # (name, start_event, end_event, launches, algorithmic work, tag)
        self.native = None       # spans of the native host side, once the recording is closed

    def _all(self):
        """[(name, ms, launches, work, tag)] of both sides."""
        torch.cuda.synchronize()
        native = _lib.host().trace_spans() if self.native is None else self.native
        return [(name, a.elapsed_time(b), launches, work, tag) for name, a, b, launches, work, tag in self.spans] + \
            [(name, ms, launches, work, (ta, tb) if ta else None) for name, ms, launches, work, ta, tb in native]

    def summary(self):
        out = {}
        for name, ms, launches, work, _tag in self._all():
            e = out.setdefault(name, {"calls": 0, "ms": 0.0, "launches": 0, "work": 0.0})
            e["calls"] += 1
            e["ms"] += ms
            e["launches"] += launches
            e["work"] += work
        return out

    def by_tag(self):
        """{(stage, tag): {"calls", "ms", "work"}} over the spans that carry a tag (the products tag their channel widths)."""
        out = {}
        for name, ms, _launches, work, tag in self._all():
            if tag is None:
                continue
            e = out.setdefault((name, tag), {"calls": 0, "ms": 0.0, "work": 0.0})
            e["calls"] += 1
            e["ms"] += ms
            e["work"] += work
        return out

    def total_launches(self):
        return sum(s[2] for s in self._all())


@contextlib.contextmanager
def recording():
    global _active
    assert _active is None, "a recording is open already"
    rec = _active = Recording()
    host = _lib.host()
    host.trace_start()
    try:
        yield rec
    finally:
        _active = None
        torch.cuda.synchronize()
        rec.native = host.trace_spans()
        host.trace_stop()


def active():
    """True while a recording is open (call sites use it to skip bookkeeping that costs a sync)."""
    return _active is not None


_NULL_CONTEXT = contextlib.nullcontext()


def stage(name, launches=None, work=0.0, tag=None):
    """Context manager around one C-ABI call site: nothing when no recording is open."""
    if _active is None:
        return _NULL_CONTEXT
    return _recorded_stage(name, launches, work, tag)


@contextlib.contextmanager
def _recorded_stage(name, launches, work, tag):
    rec = _active
    counter = _lib.lib().st_launch_count
    a = torch.cuda.Event(enable_timing=True)
    b = torch.cuda.Event(enable_timing=True)
    before = counter()
    a.record()
    try:
        yield
    finally:
        b.record()
        rec.spans.append((name, a, b, counter() - before, float(work), tag))
