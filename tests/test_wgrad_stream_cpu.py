"""Order of weight-gradient products that share a buffer but not a stream (``ops/gemm.py:weight_grad``)."""
import contextlib

import pytest
import torch

from xorl_b200.ops import _lib, gemm as G, grad_sink


class _Rows:
    """What ``weight_grad`` looks at of a gradient or an activation on the GPU."""
    is_cuda = True
    device = torch.device("cuda", 0)

    def __init__(self, rows, cols):
        self.shape = (rows, cols)

    def record_stream(self, stream):
        pass


class _Stream:
    def __init__(self, name, log):
        self.name, self.log = name, log

    def wait_stream(self, other):
        self.log.append((self.name, "waits", other.name))


@pytest.fixture
def log(monkeypatch):
    events = []
    main, side = _Stream("main", events), _Stream("side", events)
    current = [main]

    @contextlib.contextmanager
    def on(stream):
        current.append(stream)
        yield
        current.pop()

    monkeypatch.setattr(_lib, "current_stream", lambda: current[-1])
    monkeypatch.setattr(torch.cuda, "stream", on)
    monkeypatch.setattr(G, "wgrad_stream", lambda device: side)
    monkeypatch.setattr(grad_sink, "_wgrad_stream", {0: side})
    monkeypatch.setattr(grad_sink, "_wgrad_pending", False)
    monkeypatch.setattr(G, "gemm", lambda a, b, accumulate=False, **kw:
                        events.append((current[-1].name, "adds" if accumulate else "writes", a.shape[0])))
    return events


def _weight():
    w = torch.nn.Parameter(torch.zeros(4096, 4096))
    w._xb_grad_buf, w._xb_grad_fresh = torch.zeros(4096, 4096), True
    return w


LONG, SHORT = 512, 8          # rows: 2^33 and 2^27 multiply-adds


def test_short_product_waits_for_a_long_one_of_its_weight(log):
    w = _weight()
    for rows in (LONG, SHORT, SHORT):
        G.weight_grad(_Rows(rows, 4096), _Rows(rows, 4096), w)
    assert log == [("side", "waits", "main"), ("side", "writes", LONG), ("main", "waits", "side"),
                   ("main", "adds", SHORT), ("main", "adds", SHORT)]


def test_other_orders_and_weights_need_no_wait(log):
    w, other = _weight(), _weight()
    G.weight_grad(_Rows(SHORT, 4096), _Rows(SHORT, 4096), w)
    for rows in (LONG, LONG):
        G.weight_grad(_Rows(rows, 4096), _Rows(rows, 4096), w)
    G.weight_grad(_Rows(SHORT, 4096), _Rows(SHORT, 4096), other)
    assert ("main", "waits", "side") not in log


def test_gradient_of_another_kind_waits_too(log):
    w = _weight()
    G.weight_grad(_Rows(LONG, 4096), _Rows(LONG, 4096), w)
    grad_sink.deliver_param_grad(w, torch.ones(4096, 4096))
    assert log[-1] == ("main", "waits", "side")
    before = len(log)
    grad_sink.deliver_param_grad(w, torch.ones(4096, 4096))       # joined already
    assert len(log) == before and float(w._xb_grad_buf[0, 0]) == 2.0
