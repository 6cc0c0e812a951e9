"""The outlier rate that the wrapper observes over fake-quant calls of several streams and threads, read between calls, and
with calls captured in a graph."""
import copy
import threading

import pytest
import torch

import hqmq_b200 as hqmq
from hqmq_b200 import _lib

pytestmark = pytest.mark.gpu
SHAPE = (2, 2, 1, 64)


def _quantizer(fold=None):
    q = hqmq.with_outlier_extraction(hqmq.HQMQ(1, SHAPE[1], 96, 4, device="cuda"), 3.0)
    for kv in (0, 1):
        q.inner.tables(0, kv, "cuda:0")
    if fold:
        q._stats._FOLD = fold
    return q


def _inputs(n):
    """n inputs with 0 .. 7 flagged chunks per call, and the share of each."""
    xs, rates = [], []
    for i in range(n):
        x = torch.ones(SHAPE)
        x.view(2, 2, 16, 4)[0, 0, :i % 8] *= 50.0
        xs.append(x.bfloat16().cuda())
        rates.append((i % 8) / 64)
    torch.cuda.synchronize()
    return xs, rates


def test_a_stream_that_starts_while_another_is_busy():
    q, (xs, rates) = _quantizer(), _inputs(16)
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(100_000_000)
        q.quantize_K(xs[0], 0)
    with torch.cuda.stream(other):
        for x in xs[1:]:
            q.quantize_K(x, 0)
    assert q._n_observations == 16 and abs(q._observed_outlier_rate - sum(rates) / 16) < 1e-9


def test_the_rate_is_read_between_a_call_and_its_launch(monkeypatch):
    q, (xs, rates) = _quantizer(), _inputs(20)
    L = _lib.lib()
    real = L.hqmq_fake_quant

    def fake_quant(*args):
        q._observed_outlier_rate            # what another thread may do at this moment
        held.append(torch.zeros(1024, dtype=torch.int32, device="cuda"))
        return real(*args)
    held = []
    monkeypatch.setattr(L, "hqmq_fake_quant", fake_quant)
    for x in xs:
        q.quantize_K(x, 0)
    assert q._n_observations == 20 and abs(q._observed_outlier_rate - sum(rates) / 20) < 1e-9
    assert not any(h.any() for h in held)


def test_a_copy_made_between_calls_goes_on_by_itself():
    q, (xs, rates) = _quantizer(), _inputs(8)
    want = [q.quantize_K(x, 0) for x in xs]
    c = copy.deepcopy(q)
    assert all(torch.equal(c.quantize_K(x, 0), w) for x, w in zip(xs, want))
    assert c._n_observations == 16 and q._n_observations == 8 and abs(c._observed_outlier_rate - sum(rates) / 8) < 1e-9


def test_threads_on_streams_of_their_own_and_a_reader():
    q, (xs, rates) = _quantizer(fold=16), _inputs(100)
    done = threading.Event()

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for x in xs:
                q.quantize_K(x, 0)

    def read():
        while not done.is_set():
            assert 0.0 <= q._observed_outlier_rate < 1.0
    threads = [threading.Thread(target=work) for _ in range(4)]
    reader = threading.Thread(target=read)
    for t in threads + [reader]:
        t.start()
    for t in threads:
        t.join()
    done.set()
    reader.join()
    assert q._n_observations == 400 and abs(q._observed_outlier_rate - sum(rates) / 100) < 1e-9


def test_captured_calls_own_their_counters():
    q, (xs, rates) = _quantizer(fold=8), _inputs(24)
    want = [q.quantize_K(x, 0) for x in xs]
    x = xs[0].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):           # more calls than a block has counters
        out = [q.quantize_K(x, 0) for _ in range(12)]
    for y in xs:                            # blocks of ordinary calls are used up and folded meanwhile
        q.quantize_K(y, 0)
    x.copy_(xs[5])
    graph.replay()
    assert q._n_observations == 60 and abs(q._observed_outlier_rate - (2 * sum(rates) + 12 * rates[5]) / 60) < 1e-9
    canaries = [torch.zeros(n, dtype=torch.int32, device="cuda") for n in (8, 128, 1024) for _ in range(64)]
    for i in (6, 7):
        x.copy_(xs[i])
        graph.replay()
        assert all(torch.equal(o, want[i]) for o in out)
    assert not any(c.any() for c in canaries) and q._n_observations == 60
