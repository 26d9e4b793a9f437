"""Independent pieces of a layer side by side in a captured step.

A step of a few tokens is a chain of short kernels, each of which leaves most of the chip idle at its ends.  Where a layer
has two chains that only meet at an addition or an output projection (a mixer and a feed-forward that read the same stream,
two mixers of one layer, a shared expert and the routed ones), the second one is recorded on a stream of its own, and the
step's graph has two branches.  What a step computes does not depend on it, and neither do its kernels.  Parts of a layer are
recorded so only where they say that they may be (``Part.alone``).

Replays of decode steps of 8 requests, us, one branch and two: Ruvurax 4096 wide 851 and 802 (its experts' weights alone take
400 at the copy bandwidth), Lilulix 2048 wide 335 and 298; Ruvurax 2048 wide, one request, 277 and 210.  With the mixer's
branch on a stream of higher priority 821, 318 and 238: its kernels, launched ahead of their inputs, then hold the SMs
while they wait.  Steps that are launched kernel by kernel stay one chain: they are bound by the host (two prompt steps of Ruvurax
with two branches 4.9 ms where one takes 4.0), and so nothing is allocated on one stream and freed on another outside a capture.
What it costs: a branch takes memory of its graph's pool for itself, and its result is not used again before the capture ends; a
captured batch size holds 8 MB where one chain holds 2 (Ruvurax 4096 wide), 24 where it holds 22 (Lilulix 2048 wide).
"""

from __future__ import annotations

import copy

import torch

from ..csrc import ops

# The streams beside each stream that steps are recorded on, one per block that is open at a time, and how many are open; per
# device (from the library's pool of a few dozen).
_beside: dict[tuple[int, int], list[torch.cuda.Stream]] = {}
_open: dict[tuple[int, int], int] = {}


class beside:
    """``with beside() as side:``  ``result = side.run(f)`` launches what ``f()`` launches on a stream beside the
    current one, behind everything launched before; ``result()`` is what ``f`` returned (a tensor or None), and what is
    launched after that call, or after the block, starts behind ``f``'s kernels.  In between neither ``f`` nor the rest touches
    what the other writes.

    The caller keeps every tensor that ``f`` reads alive until the block's end.  Only a captured step has the second
    stream, and under ``ops.kept_sums`` not even that: ``gemm_tma``, which runs the products there, has one workspace per device
    (``ops`` raises where both sides of a block ask for such a workspace)."""

    def __init__(self) -> None:
        self.joined = True
        self.on = torch.cuda.is_initialized() and torch.cuda.is_current_stream_capturing() and not ops.sums_kept()
        if self.on:
            self.here = torch.cuda.current_stream()
            self.key = (self.here.device_index, self.here.cuda_stream)

    def __enter__(self) -> "beside":
        if self.on:       # (only one thread records on a stream at a time)
            depth = _open.get(self.key, 0)
            streams = _beside.setdefault(self.key, [])
            if depth == len(streams):
                streams.append(torch.cuda.Stream(self.here.device))
            self.stream = streams[depth]
            _open[self.key] = depth + 1
            ops.open_branches().append(self)
            self.second, self.workspaces = False, {}
        return self

    def run(self, f):
        if not self.on:
            value = f()
            return lambda: value
        self.stream.wait_stream(self.here)
        self.joined = False
        self.second = True
        try:
            with torch.cuda.stream(self.stream):
                value = f()
        finally:
            self.second = False

        def result():
            self._join()
            if value is not None:
                value.record_stream(self.here)      # its memory belongs to the stream beside
            return value
        return result

    def _join(self) -> None:
        if not self.joined:
            self.joined = True
            self.here.wait_stream(self.stream)

    def __exit__(self, *error) -> None:
        try:
            self._join()               # behind an error as well: a capture ends with one stream
        finally:
            if self.on:
                _open[self.key] -= 1
                ops.open_branches().remove(self)


def pair(ctx, part, run, other, run_other, position=None):
    """``(run(ctx), run_other(ctx))`` of a layer's two parts (tensors or None), the second one beside the first in a captured step
    where both, and the ``position`` part they may call, say that they can.  It then has a ``ctx.scratch`` of its own, as it was
    in front of both; what it leaves there, and the first one does not, is the layers' behind them when both are through."""
    parts = (part, other) if position is None else (part, other, position)
    if not all(getattr(p, "alone", False) for p in parts) or part.device_scratch & other.device_scratch:
        return run(ctx), run_other(ctx)
    with beside() as side:
        if not side.on:
            mine = run(ctx)
            return mine, side.run(lambda: run_other(ctx))()
        own = copy.copy(ctx)
        own.scratch = dict(ctx.scratch)
        theirs = side.run(lambda: run_other(own))
        both = run(ctx), theirs()
    for key, value in own.scratch.items():
        ctx.scratch.setdefault(key, value)
    return both
