"""A layer's two parts in order or side by side (``parts/streams.py``), on the host: who runs first, what each finds in the
step's shared dictionary, and which scratch memory both may ask for."""

from types import SimpleNamespace

import pytest
import torch

from mini_infer_b200.csrc import ops
from mini_infer_b200.parts import streams
from mini_infer_b200.parts.base import FeedForward, Mixer
from mini_infer_b200.parts.builtin import ParallelBlock, SameNorm
from mini_infer_b200.parts.mixers import ProjectedMixer, SideBySide
from mini_infer_b200.parts.spec import PartSpec


class FakeStream:
    device_index, device = 0, None

    def __init__(self, *_):
        self.cuda_stream, self.waits = id(self), []

    def wait_stream(self, other):
        self.waits.append(other)


class Recording:
    """``torch.cuda`` as ``beside`` sees it while a step is recorded."""

    def __init__(self, monkeypatch):
        self.now = [FakeStream()]
        cuda = torch.cuda
        monkeypatch.setattr(streams, "_beside", {})
        monkeypatch.setattr(streams, "_open", {})
        monkeypatch.setattr(cuda, "is_initialized", lambda: True)
        monkeypatch.setattr(cuda, "is_current_stream_capturing", lambda: True)
        monkeypatch.setattr(cuda, "current_stream", lambda: self.now[-1])
        monkeypatch.setattr(cuda, "Stream", FakeStream)
        monkeypatch.setattr(cuda, "stream", self.stream)
        monkeypatch.setattr(torch.Tensor, "record_stream", lambda *_: None)

    def stream(self, s):
        outer = self

        class Scope:
            def __enter__(self):
                outer.now.append(s)

            def __exit__(self, *_):
                outer.now.pop()
        return Scope()


class ToyMixer(Mixer):
    def forward(self, x, ctx, cache, position):
        ctx.scratch.setdefault("order", []).append("mixer")
        ctx.scratch["left_by_mixer"] = 7
        return x + 1


class ToyFeedForward(FeedForward):
    found = None

    def forward(self, x, ctx):
        ctx.scratch.setdefault("order", []).append("feed_forward")
        type(self).found = ctx.scratch.get("left_by_mixer")
        ctx.scratch["left_by_feed_forward"] = 8
        return x + 2


class AloneMixer(ToyMixer):
    alone = True


class AloneFeedForward(ToyFeedForward):
    alone = True


class DerivedFeedForward(AloneFeedForward):
    """Does not say it again."""


class StreamNorm:
    def forward(self, x, residual):
        return x, residual


def block(mixer, feed_forward):
    b = ParallelBlock.__new__(ParallelBlock)
    b.mixer, b.feed_forward, b.position = mixer(PartSpec("toy")), feed_forward(PartSpec("toy")), None
    b.mixer_norm, b.feed_forward_norm = StreamNorm(), SameNorm(PartSpec("same_norm"))
    return b


def run(b):
    type(b.feed_forward).found = None
    ctx = SimpleNamespace(scratch={"before": 1})
    (m, f), _ = b.forward(torch.zeros(2, 3), torch.zeros(2, 3), ctx, None)
    assert torch.equal(m, torch.ones(2, 3)) and torch.equal(f, torch.full((2, 3), 2.0))
    return ctx.scratch


@pytest.mark.parametrize("recorded", [False, True])
@pytest.mark.parametrize("mixer,feed_forward", [(ToyMixer, ToyFeedForward), (AloneMixer, ToyFeedForward),
                                                (ToyMixer, AloneFeedForward), (AloneMixer, DerivedFeedForward)])
def test_parts_that_do_not_stand_alone_run_in_order_and_share(mixer, feed_forward, recorded, monkeypatch):
    if recorded:
        Recording(monkeypatch)
    b = block(mixer, feed_forward)
    scratch = run(b)
    assert scratch["order"] == ["mixer", "feed_forward"] and b.feed_forward.found == 7
    assert scratch["left_by_mixer"] == 7 and scratch["left_by_feed_forward"] == 8


@pytest.mark.parametrize("recorded", [False, True])
def test_parts_that_stand_alone_run_in_order_outside_a_capture_and_apart_inside(recorded, monkeypatch):
    if recorded:
        Recording(monkeypatch)
    b = block(AloneMixer, AloneFeedForward)
    scratch = run(b)
    assert b.feed_forward.found == (None if recorded else 7)
    assert scratch["order"] == (["mixer"] if recorded else ["mixer", "feed_forward"])
    assert scratch["left_by_mixer"] == 7 and scratch["left_by_feed_forward"] == 8 and scratch["before"] == 1


class ToyProjected(ProjectedMixer):
    in_width = out_width = 3
    saw: list = []

    def mix(self, proj, out, out_scale, ctx, cache, position):
        self.saw.append((self.spec.kind, ctx.scratch.get("table")))
        ctx.scratch.setdefault("table", self.spec.kind)


class AloneProjected(ToyProjected):
    alone = True


class AttendingProjected(ToyProjected):
    alone = True
    device_scratch = frozenset({"decode_attention"})


@pytest.mark.parametrize("kinds,apart", [((ToyProjected, ToyProjected), False), ((AloneProjected, ToyProjected), False),
                                         ((AloneProjected, AttendingProjected), True),
                                         ((AttendingProjected, AttendingProjected), False)])
@pytest.mark.parametrize("recorded", [False, True])
def test_two_mixers_of_a_layer(kinds, apart, recorded, monkeypatch):
    if recorded:
        Recording(monkeypatch)
    s = SideBySide.__new__(SideBySide)
    s.children = [k(PartSpec(name)) for k, name in zip(kinds, ("left", "right"))]
    s.scales, s._in, s._out, s._in32 = [1.0, 1.0], lambda x: torch.zeros(2, 6), lambda o: o, None
    ToyProjected.saw.clear()
    ctx = SimpleNamespace(scratch={}, n_tokens=2)
    s.forward(torch.zeros(2, 3), ctx, None, None)
    second = None if apart and recorded else "left"
    assert sorted(ToyProjected.saw) == [("left", None), ("right", second)]
    assert ctx.scratch == {"table": "left"}
    if second == "left":
        assert ToyProjected.saw[0][0] == "left"


def test_one_workspace_per_device_is_one_branchs_alone(monkeypatch):
    Recording(monkeypatch)
    with streams.beside() as side:
        ops._claim_workspace("a")
        side.run(lambda: ops._claim_workspace("b"))
        ops._claim_workspace("a")
        with pytest.raises(ops.KernelError, match="a: both branches"):
            side.run(lambda: ops._claim_workspace("a"))
        with pytest.raises(ops.KernelError, match="b: both branches"):
            ops._claim_workspace("b")
        with streams.beside() as inner:       # an inner block's branches are one branch of the outer block
            inner.run(lambda: ops._claim_workspace("c"))
        ops._claim_workspace("c")
        with pytest.raises(ops.KernelError, match="c: both branches"):
            side.run(lambda: ops._claim_workspace("c"))
    assert not ops.open_branches()
    ops._claim_workspace("a")
    ops._claim_workspace("b")


def test_a_block_whose_join_fails_is_closed(monkeypatch):
    rec = Recording(monkeypatch)
    here = rec.now[-1]
    for _ in range(2):
        with pytest.raises(RuntimeError, match="capture"):
            with streams.beside() as side:
                side.run(lambda: None)

                def fail(other):
                    raise RuntimeError("capture")
                here.wait_stream = fail
        del here.wait_stream
        assert not any(streams._open.values()) and not ops.open_branches()
    assert len(streams._beside[(0, here.cuda_stream)]) == 1
