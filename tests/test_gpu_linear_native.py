"""Which calls of a linear the C++ path takes, and that it gives what the general path gives."""
import pytest
import torch
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

from xn_b200 import synth
from xn_b200.dtypes import GgmlDType as D

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
N, K = 200, 512


class Sub(torch.Tensor):
    pass


class Mode(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


@pytest.fixture(scope="module")
def weight():
    from xn_b200 import quantized as Q
    Q.init(DEV)
    return Q.QCudaTensor.from_qtensor(Q.QTensor(synth.make_weight(D.Q4K, N, K, seed=4), (N, K), D.Q4K), DEV)


def _rows(*shape, act=torch.float32):
    g = torch.Generator(device="cpu"); g.manual_seed(sum(shape))
    return torch.randn(shape, generator=g).to(act).to(DEV)


FORMS = {   # input -> whether the C++ path takes it
    "one row": (lambda a: _rows(1, K, act=a), True),
    "rows": (lambda a: _rows(7, K, act=a), True),
    "many rows": (lambda a: _rows(90, K, act=a), True),
    "no rows": (lambda a: _rows(0, K, act=a), True),
    "three dimensions": (lambda a: _rows(2, 3, K, act=a), True),
    "rows apart": (lambda a: _rows(5, 2 * K, act=a)[:, :K], True),
    "every other row": (lambda a: _rows(6, K, act=a)[::2], True),
    "one row of a wider matrix": (lambda a: _rows(3, 2 * K, act=a)[1:2, :K], True),
    "a parameter": (lambda a: torch.nn.Parameter(_rows(4, K, act=a)), True),
    "columns apart": (lambda a: _rows(K, 5, act=a).t(), False),
    "one row repeated": (lambda a: _rows(1, K, act=a).expand(4, K), False),
    "three dimensions, rows apart": (lambda a: _rows(2, 3, 2 * K, act=a)[:, :, :K], False),
    "one dimension": (lambda a: _rows(K, act=a), False),
    "a subclass": (lambda a: _rows(4, K, act=a).as_subclass(Sub), False),
}


@pytest.mark.parametrize("act", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("form", FORMS)
def test_same_results_on_both_paths(weight, form, act):
    from xn_b200 import quantized as Q
    make, native = FORMS[form]
    x = make(act)
    y = Q._linear(weight._native, x, None)
    assert (y is not None) == native
    want = weight._matmul_float(x, None, None)
    got = weight.matmul_t(x)
    assert got.dtype is act and got.shape == x.shape[:-1] + (N,) and got.is_contiguous() and not got.requires_grad
    assert torch.equal(got, want) and (y is None or torch.equal(y, want))


def test_calls_that_are_not_ordinary(weight):
    from xn_b200 import quantized as Q
    x = _rows(3, K)
    want = weight.matmul_t(x)
    with Mode():
        assert Q._linear(weight._native, x, None) is None and torch.equal(weight.matmul_t(x), want)
    with torch.inference_mode():
        assert torch.equal(weight.matmul_t(x), want)
    for bad in (x.double(), x.cpu(), x[:, : K - 32], x.int()):
        assert Q._linear(weight._native, bad, None) is None
        with pytest.raises(ValueError):
            weight.matmul_t(bad)
    odd = torch.zeros(3 * K + 1, device=DEV)[1:].view(3, K)      # rows that do not start on 16 bytes
    for call in (weight.matmul_t, Q.QCudaLinear.new(weight).forward, lambda t: weight._matmul_float(t, None, None)):
        with pytest.raises(Q.XnqError):
            call(odd)
    with pytest.raises(ValueError):
        Q.QCudaLinear.new(weight).forward(x[0])


def test_in_a_captured_graph(weight):
    x = _rows(20, K)
    want = weight.matmul_t(x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = weight.matmul_t(x)
    y.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)


def test_a_weight_on_a_device_without_an_index(weight):
    """It refuses rows of a device with an index, with and without `out`; images are taken, on the current device."""
    from xn_b200 import decoder_ops as ops, quantized as Q
    w = Q.QCudaTensor.from_qtensor(Q.QTensor(weight.data(), (N, K), D.Q4K), torch.device("cuda"))
    x = _rows(3, K)
    for call in (lambda: w.matmul_t(x), lambda: Q.QCudaLinear.new(w).forward(x), lambda: w.matmul_t(x, out=torch.empty(3, N, device=DEV))):
        with pytest.raises(ValueError, match="input on cuda:0, weight on cuda"):
            call()
    image = ops.quantize_act_image(x, ops.ActImage.for_weight(D.Q4K, 3, K, DEV))
    assert torch.equal(w.matmul_t(image), weight.matmul_t(image))
    assert w.workspace(3).device == DEV


class Recorder(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen.append(func.overloadpacket)
        return func(*args, **(kwargs or {}))


class FunctionRecorder(TorchFunctionMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.seen.append(getattr(func, "__name__", ""))
        return func(*args, **(kwargs or {}))


def test_modes_see_the_addition_of_a_bias(weight):
    from xn_b200 import quantized as Q
    x, bias = _rows(3, K), torch.randn(N, device=DEV)
    layer = Q.QCudaLinear.new(weight, bias)
    want = layer.forward(x)
    assert torch.equal(want, weight.matmul_t(x) + bias)
    with Recorder() as r:
        assert torch.equal(layer.forward(x), want)
    assert torch.ops.aten.add_ in r.seen
    with FunctionRecorder() as r:
        assert torch.equal(layer.forward(x), want)
    assert "add_" in r.seen
    assert torch.equal(layer.forward(x), want)


def test_transforms_and_tracers(weight):
    """What torch wraps has no memory that a kernel could read: such calls are refused, as the results of a call inside `grad` or `jvp` are."""
    from xn_b200 import quantized as Q
    x, biases = _rows(3, K), torch.randn(4, N, device=DEV)
    forward = lambda b: Q.QCudaLinear.new(weight, b).forward(x)
    want = forward(biases[0])
    for call in (lambda: torch.func.vmap(forward)(biases), lambda: torch.func.vmap(lambda r: weight.matmul_t(r[None]))(x),
                 lambda: torch.func.grad(lambda b: forward(b).sum())(biases[0]), lambda: torch.func.jvp(forward, (biases[0],), (biases[1],))):
        with pytest.raises(RuntimeError):
            call()
    assert torch.equal(forward(biases[0]), want)
    seen = []

    def look(t):
        seen.append(Q._linear(weight._native, t, None) is None)
        return forward(biases[0]) + t[0, 0]
    trace = torch.jit.trace(look, x, check_trace=False)
    assert seen == [True] and "add_" in str(trace.graph)
    assert Q._linear(weight._native, x, None) is not None
    with torch.inference_mode():
        assert Q._linear(weight._native, x, None) is not None
    with torch.autocast("cuda"):
        assert Q._linear(weight._native, x, None) is not None
