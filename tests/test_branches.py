"""A layer's two parts side by side (``parts/streams.py``), on the host."""

import pytest
import torch

from mini_infer_b200.parts import streams


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
        assert not any(streams._open.values())
    assert len(streams._beside[(0, here.cuda_stream)]) == 1
