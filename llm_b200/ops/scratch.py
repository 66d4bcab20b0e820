"""Scratch memory of the kernels that work in parts: partial sums, and counters that a call finds and leaves at zero.

Two calls may have the same scratch only if one runs behind the other. So scratch belongs to a line of work:

* an engine's steps (a `StepScope`, entered with `with`): plain, recorded and captured ones share the engine's arena too,
  and so run one after the other whatever stream they are on;
* every other call belongs to its stream. The last STREAMS streams of a device that asked keep theirs; what an older one
  held goes back to the allocator, which reuses it behind that stream's work;
* a call under capture outside a `StepScope` has its own, inside its graph (with a kernel that zeroes the counters).
"""
from __future__ import annotations

import threading

import torch

STREAMS = 8
_LEAST = {"products": (148 * 2 * 128 * 256, 1 << 14),     # what a product on pairs of SMs asks for at most; tile counters
          "attention": (1 << 23, 0)}

generation = 0                            # grows with that of every scope and stream
_line = threading.local()                 # .entered: the scopes that this thread is inside of
_lock = threading.Lock()
_of_stream: dict = {}                     # (device, stream) -> StepScope, the one that was asked last at the end


def _new(device, floats: int, counters: int) -> tuple:
    return (torch.empty(floats, dtype=torch.float32, device=device),
            torch.zeros(counters, dtype=torch.int32, device=device) if counters else None)


class StepScope:
    """The scratch of one line of work, an engine's steps for instance. Inside `with scope:` the calls of this thread use it,
    on any stream and under capture, and products and norms take the matrices and gains that they are given for weights, which
    no kernel inside the scope writes (ops.linear, ops.norm_add_). It grows when a call needs more; what was outgrown is kept, because captured and
    recorded steps may hold its address. `generation` counts that."""

    def __init__(self):
        self._held, self._outgrown, self.generation = {}, [], 0

    def __enter__(self):
        if not hasattr(_line, "entered"):
            _line.entered = []
        _line.entered.append(self)
        return self

    def __exit__(self, *error):
        _line.entered.pop()

    def room(self, device, kind: str, floats: int, counters: int, capturing: bool) -> tuple:
        global generation
        held = self._held.get((device, kind))
        if held is not None and held[0].numel() >= floats and (held[1].numel() if held[1] is not None else 0) >= counters:
            return held
        if capturing:                     # what a capture allocates belongs to its graph
            return _new(device, floats, counters)
        least = _LEAST[kind]
        grown = _new(device, max(floats, least[0], held[0].numel() if held else 0),
                     max(counters, least[1], held[1].numel() if held and held[1] is not None else 0))
        if held is not None:
            self._outgrown.append(held)
            self.generation += 1
            generation += 1
        self._held[(device, kind)] = grown
        return grown


def inside() -> bool:
    """Whether this thread is inside a StepScope."""
    return bool(getattr(_line, "entered", None))


def of_call(device, stream: int, capturing: bool, kind: str, floats: int, counters: int = 0) -> tuple:
    """(float32 [>= floats], int32 [>= counters], zero, or None) for a call that is launched on `stream`."""
    entered = getattr(_line, "entered", None)
    if entered:
        return entered[-1].room(device, kind, floats, counters, capturing)
    if capturing:
        return _new(device, floats, counters)
    with _lock:
        scope = _of_stream.pop((device, stream), None)
        if scope is None:
            scope = StepScope()
            for key in [key for key in _of_stream if key[0] == device][:1 - STREAMS]:
                del _of_stream[key]
        _of_stream[(device, stream)] = scope
        found = scope.room(device, kind, floats, counters, False)
        scope._outgrown.clear()           # nothing but records points at it, and those keep it themselves
        return found
