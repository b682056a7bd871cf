"""Calls of a linear from a torch program: biases, streams, strides and shapes."""
import pytest
import torch

from xn_b200 import synth
from xn_b200.dtypes import GgmlDType as D

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
N, K = 300, 1024


@pytest.fixture(scope="module")
def weight():
    from xn_b200 import quantized as Q
    Q.init(DEV)
    return Q.QCudaTensor.from_qtensor(Q.QTensor(synth.make_weight(D.Q4K, N, K, seed=4), (N, K), D.Q4K), DEV)


@pytest.mark.parametrize("act", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bias_type", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, K), (2, 3, K), (70, K), (0, K)])
def test_a_bias_is_added_in_the_type_of_the_result(weight, act, bias_type, shape):
    from xn_b200 import quantized as Q
    g = torch.Generator(device="cpu"); g.manual_seed(len(shape) + shape[0])
    x = torch.randn(shape, generator=g).to(act).to(DEV)
    bias = torch.randn(N, generator=g).to(bias_type).to(DEV)
    kept = bias.clone()
    plain = Q.QCudaLinear.new(weight)
    biased = Q.QCudaLinear.new(weight, bias)
    y, yb = plain.forward(x), biased.forward(x)
    assert yb.dtype is act and yb.shape == shape[:-1] + (N,)
    assert torch.equal(yb, y + bias.to(act)) and torch.equal(biased.forward(x), yb)
    assert torch.equal(bias, kept)


@pytest.mark.parametrize("m", [1, 3, 16, 70])
def test_a_call_runs_on_the_current_stream(weight, m):
    """The input is rewritten on a side stream that is still busy: only a call on that stream sees the new rows."""
    g = torch.Generator(device="cpu"); g.manual_seed(m)
    a, b = (torch.randn(m, K, generator=g).to(DEV) for _ in range(2))
    want = weight.matmul_t(b)
    x = a.clone()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
        x.copy_(b)
        got = weight.matmul_t(x)
    side.synchronize()
    assert torch.equal(got, want)


def test_rows_with_strides_and_views(weight):
    g = torch.Generator(device="cpu"); g.manual_seed(9)
    wide = torch.randn(6, 2 * K, generator=g).to(DEV)
    want = weight.matmul_t(wide[:, :K].contiguous())
    assert torch.equal(weight.matmul_t(wide[:, :K]), want)                                     # rows apart
    assert torch.equal(weight.matmul_t(wide[:, :K].t().contiguous().t()), want)                # columns apart
    assert torch.equal(weight.matmul_t(wide[:1, :K].expand(6, K)), weight.matmul_t(wide[:1, :K].repeat(6, 1)))  # one row six times
    assert torch.equal(weight.matmul_t(wide[:, :K].reshape(2, 3, K)), want.view(2, 3, N))
    assert torch.equal(weight.matmul_t(wide[::2, :K]), weight.matmul_t(wide[::2, :K].contiguous()))
    out = torch.full((6, N), 7.0, device=DEV)
    assert weight.matmul_t(wide[:, :K], out=out) is out and torch.equal(out, want)
    with pytest.raises(ValueError):
        weight.matmul_t(wide)
    with pytest.raises(ValueError):
        weight.matmul_t(wide[:, :K].double())
    with pytest.raises(ValueError):
        weight.matmul_t(wide[:, :K].cpu())
