"""How far f32 results of the small-batch kernels are from the exact dot of the quantized operands: no further than the roundings of
the order in which they add."""
import numpy as np
import pytest
import torch

from xn_b200 import synth
from xn_b200.dtypes import GgmlDType as D

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
# rms error of one rounding to f32, relative to the value: uniform within half a unit in the last place, the mantissa's logarithm uniform
ROUNDING = 2.0 ** -24 * np.sqrt(0.75 / (2 * np.log(2)) / 3)


@pytest.fixture(scope="module")
def Q():
    from xn_b200 import quantized
    quantized.init(DEV)
    return quantized


def chain(terms, var, first):
    """Sum of the variances of the partial sums that a chain of `terms` terms of variance `var` rounds; first: whether the first one is."""
    return var * sum(range(1 if first else 2, terms + 1))


def runs(terms, var, first):
    """The same where the chain is cut after eight terms and the runs' sums are added in a second chain."""
    whole, rest = divmod(terms, 8)
    total = whole * chain(8, var, first) + chain(rest, var, first)
    return total + sum(var * min(8 * i, terms) for i in range(2, whole + (rest > 0) + 1))


def expected(dt, steps, per_cta):
    """Relative rms error: `steps` steps of 256 values (variance 1 each) of which a CTA adds `per_cta`; the parts of a tile are added in runs."""
    parts = steps // per_cta
    if dt is D.Q6K:     # one fused multiply-add per step, in runs; and the rounding of the two scales' product
        total = parts * runs(per_cta, 1.0, True) + steps
    else:               # eight block terms (fused; their scales' product is exact), then the step's sum
        total = steps * chain(8, 1 / 8, True) + parts * chain(per_cta, 1.0, False)
    return ROUNDING * np.sqrt((total + runs(parts, float(per_cta), False)) / steps)


# equal shares of two steps (every tile is in steps / 2 parts), and whole tiles
@pytest.mark.parametrize("dt", [D.Q4_0, D.Q8_0, D.Q6K])
@pytest.mark.parametrize("tiles,steps", [(8, 4), (5, 56), (0, 16)])
def test_integer_tensor_core_kernel(Q, O, dt, tiles, steps):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per_cta = 2 if tiles else steps
    tiles = tiles or sms
    assert tiles * steps // 2 <= sms if per_cta == 2 else tiles == sms
    n, k, m = 128 * tiles, 256 * steps, 8
    w = synth.make_weight(dt, n, k, seed=steps)
    x = np.random.default_rng(steps).standard_normal((m, k)).astype(np.float32)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    want = O.matmul(int(dt), x, w, n, order="f64", threads=O.hw_threads())
    got = t.matmul_t(torch.from_numpy(x).to(DEV)).cpu().numpy().astype(np.float64)
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err <= 1.06 * expected(dt, steps, per_cta), (dt.name, n, k, err, expected(dt, steps, per_cta))
