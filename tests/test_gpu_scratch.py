"""Calls that overlap have scratch of their own: on two streams, from two threads on one stream, and in two graphs that are replayed side by side."""
import threading

import pytest
import torch

from xn_b200 import synth
from xn_b200.dtypes import GgmlDType as D

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
# one row whose activations are quantized into scratch, the generic kernel, the integer kernel with split tiles, the fp16 kernel with whole ones: kernels that
# give the same bits every time
CASES = [(D.Q4_0, 300, 4096, 1, torch.float32), (D.Q4K, 512, 14336, 1, torch.float32), (D.Q5K, 2048, 2048, 7, torch.float32), (D.Q8_0, 1000, 4096, 33, torch.float32), (D.Q4K, 3000, 2048, 16, torch.float32),
         (D.Q6K, 640, 1024, 300, torch.bfloat16)]


def _pairs(dt, n, k, m, act):
    """One weight, two inputs, their results one after the other."""
    from xn_b200 import quantized as Q
    Q.init(DEV)
    layer = Q.QCudaLinear.new(Q.QCudaTensor.from_qtensor(Q.QTensor(synth.make_weight(dt, n, k, seed=n), (n, k), dt), DEV))
    xs = [torch.from_numpy(synth.make_activation(m, k, seed=s)).to(act).to(DEV) for s in (1, 2)]
    want = [layer.forward(x) for x in xs]
    torch.cuda.synchronize()
    assert not torch.equal(*want)
    return layer, xs, want


@pytest.mark.parametrize("dt,n,k,m,act", CASES)
def test_two_streams(dt, n, k, m, act):
    layer, xs, want = _pairs(dt, n, k, m, act)
    streams = [torch.cuda.Stream(DEV) for _ in xs]
    got = [[], []]
    for _ in range(50):
        for s, x, g in zip(streams, xs, got):
            with torch.cuda.stream(s):
                g.append(layer.forward(x))
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        assert all(torch.equal(y, w) for y in g)


@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("dt,n,k,m,act", CASES)
def test_two_threads_on_one_stream(dt, n, k, m, act, general):
    layer, xs, want = _pairs(dt, n, k, m, act)
    got = [[], []]

    def work(i):
        for _ in range(100):
            got[i].append(layer.weight._matmul_float(xs[i], None, None) if general else layer.forward(xs[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        assert len(g) == 100 and all(torch.equal(y, w) for y in g)


@pytest.mark.parametrize("dt,n,k,m,act", CASES)
def test_two_graphs_side_by_side(dt, n, k, m, act):
    layer, xs, want = _pairs(dt, n, k, m, act)
    graphs, ys = [], []
    for x in xs:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ys.append([layer.forward(x) for _ in range(4)])
        graphs.append(g)
    streams = [torch.cuda.Stream(DEV) for _ in xs]
    eager = []
    torch.cuda.synchronize()
    for _ in range(20):
        for s, g in zip(streams, graphs):
            with torch.cuda.stream(s):
                g.replay()
        eager.append(layer.forward(xs[0]))   # and beside calls that are not in a graph
    torch.cuda.synchronize()
    for out, w in zip(ys, want):
        assert all(torch.equal(y, w) for y in out)
    assert all(torch.equal(y, want[0]) for y in eager)


@pytest.mark.parametrize("dt,n,k,served", [(D.Q4_0, 300, 32, True), (D.Q8_0, 129, 4096, True), (D.Q4K, 64, 256, True), (D.Q6K, 1000, 4096, True), (D.Q4K, 64, 4352, False),
                                           (D.Q8_0, 64, 4128, False), (D.Q5K, 64, 256, False)])
def test_one_row_without_scratch(dt, n, k, served):
    """The entry that takes no scratch serves the rows that need none, with the other entry's bits, and leaves the others to it."""
    from xn_b200 import _lib, quantized as Q
    Q.init(DEV)
    L = _lib.lib()
    w = Q.QCudaTensor.from_qtensor(Q.QTensor(synth.make_weight(dt, n, k, seed=n), (n, k), dt), DEV)
    for act in (torch.float32, torch.float16, torch.bfloat16):
        x, bias = torch.from_numpy(synth.make_activation(1, k, seed=3)).to(act).to(DEV), torch.randn(n, device=DEV).to(act)
        for b in (None, bias):
            y = torch.full((n + 16,), 777.0, device=DEV, dtype=act)
            rc = L.xnq_matvec(w._h, x.data_ptr(), Q._XNQ_IDS[act], None if b is None else b.data_ptr(), y.data_ptr(), Q._XNQ_IDS[act], Q._raw_stream(0))
            assert rc == (0 if served else -8)
            want = w._matmul_float(x, None, b)
            assert torch.all(y[n if served else 0:] == 777.0) and (not served or torch.equal(y[:n], want[0]))
            assert torch.equal(Q.QCudaLinear.new(w, b).forward(x), want)
    if served:
        assert L.xnq_matvec(w._h, x.data_ptr(), Q._XNQ_IDS[act], None, None, Q._XNQ_IDS[act], None) == -1
        assert L.xnq_matvec(w._h, x.data_ptr(), Q._XNQ_IDS[act], None, y.data_ptr(), 2, None) == -2
        assert L.xnq_matvec(w._h, x.data_ptr() + 2, Q._XNQ_IDS[act], None, y.data_ptr(), Q._XNQ_IDS[act], None) == -4


def test_many_streams():
    """More streams than scratch is kept for, again after all weights are gone."""
    streams = [torch.cuda.Stream(DEV) for _ in range(24)]
    for _ in range(2):
        layer, xs, want = _pairs(D.Q5K, 2048, 2048, 7, torch.float32)
        got = []
        for _ in range(4):
            for i, s in enumerate(streams):
                with torch.cuda.stream(s):
                    got.append((i % 2, layer.forward(xs[i % 2])))
        torch.cuda.synchronize()
        assert all(torch.equal(y, want[i]) for i, y in got)
        del layer, got


def test_rows_of_changing_number():
    """Calls whose scratch differs in size and kind, in turn on one stream, scratch that is kept and scratch that is not."""
    layer, _, _ = _pairs(D.Q4K, 512, 2048, 2, torch.float32)
    other, _, _ = _pairs(D.Q5K, 512, 2048, 2, torch.float32)
    ms = (1, 2, 3, 7, 16, 64, 65, 300, 2000)
    xs = [torch.from_numpy(synth.make_activation(m, 2048, seed=m)).to(torch.bfloat16).to(DEV) for m in ms]
    want = []
    for x in xs:
        want.append([w.forward(x) for w in (layer, other)])
        torch.cuda.synchronize()
    got = [[w.forward(x) for w in (layer, other)] for _ in range(20) for x in xs]
    torch.cuda.synchronize()
    for i, ys in enumerate(got):
        assert all(torch.equal(y, v) for y, v in zip(ys, want[i % len(ms)])), ms[i % len(ms)]
