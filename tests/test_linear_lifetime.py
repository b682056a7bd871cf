"""The weight that a linear's call works on lives until the call returns, also when another thread gives the layer a new one meanwhile. No device: the
native call is replaced by one that does what happens while the real one waits for the device's queue with the interpreter's lock free."""
import threading
import weakref

import pytest
import torch

from xn_b200 import quantized as Q


class _Weight:
    """Stands for a QCudaTensor: `_native` is what the native call gets, and does not own the weight."""

    def __init__(self, n):
        self.n, self.device, self._native = n, torch.device("cpu"), object()

    def matmul_t(self, xs):
        return torch.zeros(xs.shape[:-1] + (self.n,))


@pytest.mark.parametrize("bias", [None, torch.zeros(4)])
def test_weight_outlives_the_call(monkeypatch, bias):
    layer = Q.QCudaLinear(_Weight(4), bias)
    ref = weakref.ref(layer.weight)
    seen = []

    def replace():
        layer.weight, layer.bias = _Weight(4), None

    def call(native, xs, b):
        t = threading.Thread(target=replace)
        t.start()
        t.join()
        w = ref()
        seen.append(w is not None and native is w._native)
        return torch.ones(xs.shape[:-1] + (4,))

    monkeypatch.setattr(Q, "_linear", call)
    assert torch.equal(layer.forward(torch.zeros(2, 8)), torch.ones(2, 4))
    assert seen == [True]
    assert ref() is None   # and no longer: the layer holds another one


def test_weight_outlives_the_general_path(monkeypatch):
    layer = Q.QCudaLinear(_Weight(4))
    first = layer.weight

    def call(native, xs, b):
        layer.weight = _Weight(5)
        return None   # not an ordinary call

    monkeypatch.setattr(Q, "_linear", call)
    assert layer.forward(torch.zeros(2, 8)).shape == (2, first.n)
