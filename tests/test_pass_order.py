"""Forward passes of one device share scratch and caches: every one of them runs inside `turn`, which orders the callers' streams."""
import contextlib

import pytest
import torch


class _Stream:
    def __init__(self):
        self.log = []

    def wait_event(self, e):
        self.log.append(("wait", e.at))


class _Event:
    at = None

    def record(self, stream):
        self.at = stream


def test_turn_orders_streams(monkeypatch):
    from xfastertransformer_b200.ops import native as N
    ws = N.Workspace.__new__(N.Workspace)
    ws.device, ws.used, ws.event = torch.device("cuda", 0), None, None
    a, b = _Stream(), _Stream()
    monkeypatch.setattr(torch.cuda, "Event", _Event)
    for s in (a, b, a):
        monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None, s=s: s)
        with contextlib.suppress(KeyError), ws.turn():
            if s is b:
                raise KeyError                               # a pass that fails has launched work too
    assert a.log == [("wait", b)] and b.log == [("wait", a)]


def test_every_pass_takes_its_turn(monkeypatch, tmp_path):
    import xfastertransformer_b200 as xft
    from xfastertransformer_b200.runtime import engine, kv_cache
    from xfastertransformer_b200.tools.synthetic import preset, write_synthetic_checkpoint
    inside, grown = [], []

    @contextlib.contextmanager
    def turn(device):
        inside.append(device)
        yield
        inside.pop()
    monkeypatch.setattr(engine, "turn", turn)
    monkeypatch.setattr(kv_cache, "turn", turn)
    write_synthetic_checkpoint(str(tmp_path), preset("tiny-llama"), seed=3)
    m = xft.AutoModel.from_pretrained(str(tmp_path), dtype="bf16")
    forward, grow, passes = m.model.decoder.forward, m.model.cache._grow_pools, []
    monkeypatch.setattr(m.model.decoder, "forward", lambda *a: (passes.append(len(inside)), forward(*a))[1])
    monkeypatch.setattr(m.model.cache, "_grow_pools", lambda n: (grown.append(len(inside)), grow(n))[1])
    ids = m.set_input_cb([[3, 4, 5]], None, 100).tolist()
    m.forward_cb()
    m.set_input_cb([7], ids)
    m.forward_cb()
    m.set_input_cb([8], ids, greedy=True)
    m.forward_cb_greedy()
    m.free_seqs(ids)
    m(torch.tensor([[1, 2, 3]]))
    m.generate(torch.tensor([[1, 2, 3]]), max_length=6)
    assert len(passes) >= 7 and min(passes) >= 1 and grown and min(grown) >= 1


def test_shapes_leave_in_the_order_of_their_last_use():
    from xfastertransformer_b200.runtime.cuda_runner import CudaRunner
    r = CudaRunner.__new__(CudaRunner)
    r.graphs = {i: object() for i in range(1, 66)}
    assert r.worth_capturing(None, 1) and len(r.graphs) == 65
    assert not r.worth_capturing(None, 100)                  # a new shape: the one unused for longest makes room
    assert 1 in r.graphs and 2 not in r.graphs and len(r.graphs) == 64
