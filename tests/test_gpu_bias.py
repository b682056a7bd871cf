"""A linear's bias in every kernel that adds it: bit for bit the plain result plus the bias in the result's type."""
import pytest
import torch

from xn_b200 import synth
from xn_b200.dtypes import GgmlDType as D

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
FAST = [D.Q4_0, D.Q8_0, D.Q4K, D.Q6K]


def _linears(dt, n, k, act):
    from xn_b200 import quantized as Q
    Q.init(DEV)
    weight = Q.QCudaTensor.from_qtensor(Q.QTensor(synth.make_weight(dt, n, k, seed=n + k), (n, k), dt), DEV)
    bias = torch.from_numpy(synth.make_activation(1, n, seed=7)[0]).to(act).to(DEV)
    return Q.QCudaLinear.new(weight), Q.QCudaLinear.new(weight, bias), bias


# one row (both ring depths, segments of a long row), the dp4a rows, the integer kernel with whole and split tiles, the fp16 kernel with one and
# two accumulators, whole, split and paired tiles; rows of y that take 16-byte stores and rows that do not
@pytest.mark.parametrize("act", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dt", FAST + [D.Q5K, D.Q5_1])
def test_bias_is_the_last_addition(dt, act):
    for n, k, ms in ((300, 1024, (1, 2, 3, 6, 17, 48, 70, 300)), (129, 8192, (1, 4, 16, 65)), (4096, 512, (1, 5, 64, 128, 257)), (3841, 2048, (881,))):
        if dt not in FAST and n == 3841:
            continue
        plain, biased, bias = _linears(dt, n, k, act)
        for m in ms:
            x = torch.from_numpy(synth.make_activation(m, k, seed=m)).to(act).to(DEV)
            y, yb = plain.forward(x), biased.forward(x)
            assert yb.dtype is act
            if act is torch.float32 and m > 16 and dt in FAST:   # split tiles: more than two parts (at most 64 here) meet in any order, one rounding each
                assert (yb - (y + bias)).abs().max() <= 64 * 2.0 ** -24 * 4 * float(y.abs().max()), (dt.name, n, k, m)
            else:
                assert torch.equal(yb, y + bias), (dt.name, n, k, m)


def test_bias_that_torch_has_to_see():
    plain, _, _ = _linears(D.Q4K, 300, 1024, torch.float32)
    from xn_b200 import quantized as Q
    x = torch.from_numpy(synth.make_activation(3, 1024, seed=1)).to(DEV)
    want = plain.forward(x)
    bias = torch.nn.Parameter(torch.randn(300, device=DEV))
    linear = Q.QCudaLinear.new(plain.weight, bias)
    y = linear.forward(x)
    y.sum().backward()
    assert torch.equal(y.detach(), want + bias.detach()) and torch.equal(bias.grad, torch.full((300,), 3.0, device=DEV))
    with torch.no_grad():
        assert torch.equal(linear.forward(x), want + bias)
    apart = torch.randn(600, device=DEV)[::2]
    assert torch.equal(Q.QCudaLinear.new(plain.weight, apart).forward(x), want + apart)
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(apart, torch.ones_like(apart))
        tangent = torch.autograd.forward_ad.unpack_dual(Q.QCudaLinear.new(plain.weight, dual).forward(x)).tangent
        assert torch.equal(tangent, torch.ones(3, 300, device=DEV))
