"""The order of the events of ``sageattn_host``, on fake streams: copies run at once, in the order in
which they are issued."""
import contextlib

import pytest
import torch

from sageattention_rdna3_b200 import host_pipeline


class _Event:
    def __init__(self):
        self.stream = None

    def record(self, stream):
        self.stream = stream
        stream.log.append(("record", self))

    def synchronize(self):
        assert self.stream is not None


class _Stream:
    def __init__(self, name):
        self.name, self.log = name, []

    def wait_event(self, event):
        assert event.stream is not None, "waits for an event that has not been recorded"
        self.log.append(("wait", event))


@pytest.mark.parametrize("layout,chunks", [("HND", 16), ("HND", 2), ("NHD", 16)])
def test_events_of_the_pipeline(monkeypatch, layout, chunks):
    """Every chunk: copy in -> compute -> copy back, each behind an event of the stage before; the copy back of
    a chunk also behind the copy in of the next one (it must not start somewhere within it)."""
    s_in, s_run, s_out, cur = (_Stream(n) for n in ("in", "run", "out", "current"))
    monkeypatch.setattr(host_pipeline, "_streams", lambda dev: (s_in, s_run, s_out))
    monkeypatch.setattr(torch.cuda, "Event", _Event)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: cur)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda self, s: None)
    calls = []

    def attention(q, k, v, **kw):
        calls.append(kw)
        return q * 2 + k.mean() + v.mean()

    monkeypatch.setattr(host_pipeline, "sageattn", attention)
    shape = (2, 4, 8, 64) if layout == "HND" else (2, 8, 4, 64)
    q, k, v = (torch.randn(shape) for _ in range(3))
    out = host_pipeline.sageattn_host(q, k, v, out=torch.empty_like(q), tensor_layout=layout, device=torch.device("cpu"),
                                      chunks=chunks)
    n = len(calls)
    assert n == (2 if layout == "NHD" else min(8, chunks))
    per = (lambda t: [t[b:b + 1] for b in range(2)]) if n == 2 else (lambda t: [t[b:b + 1, h:h + 1] for b in range(2) for h in range(4)])
    for o, a, b, c in zip(*(per(t) for t in (out, q, k, v))):
        assert torch.equal(o, a * 2 + b.mean() + c.mean())
    of = lambda s, what: [e for w, e in s.log if w == what]
    copied, computed = of(s_in, "record"), of(s_run, "record")
    assert of(s_run, "wait")[1:] == copied and of(cur, "wait") == of(s_out, "record")
    want = []
    for i in range(n):
        want += [computed[i]] + copied[i + 1:i + 2]
    assert of(s_out, "wait")[1:] == want
