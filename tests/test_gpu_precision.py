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


def exact_dots(O, dt, w, x, n, k):
    """f64 dots of the quantized operands; the offset term of the Q8_1 formats is the stored product, as the CPU code has it."""
    f16 = lambda b: b.copy().view(np.float16).astype(np.float64)
    adt, wf = dt.vec_dot_type, O.to_float(int(dt), w, n * k).reshape(n, k).astype(np.float64)
    out = np.empty((len(x), n))
    for r, row in enumerate(x):
        b = O.from_float(int(adt), row).reshape(-1, adt.type_size)
        if adt is D.Q8K:
            out[r] = wf @ (b[:, 4:260].copy().view(np.int8) * b[:, :4].copy().view(np.float32).astype(np.float64)).reshape(-1)
        elif adt is D.Q8_0:
            out[r] = wf @ (b[:, 2:34].copy().view(np.int8) * f16(b[:, :2])).reshape(-1)
        else:
            mins = f16(w.reshape(n, -1, dt.type_size)[:, :, 2:4].reshape(-1, 2)).reshape(n, -1)
            out[r] = (wf - np.repeat(mins, 32, 1)) @ (b[:, 4:36].copy().view(np.int8) * f16(b[:, :2])).reshape(-1) + mins @ f16(b[:, 2:4])[:, 0]
    return out


@pytest.mark.parametrize("dt", [D.Q4_1, D.Q5_0, D.Q5_1, D.Q2K, D.Q3K, D.Q5K])
@pytest.mark.parametrize("k", [1024, 4096, 14336])
def test_formats_held_as_file_blocks(Q, O, dt, k):
    """No further from the exact dots than the CPU code's own f32 order (4 % for the sample: 16 x 500 results)."""
    n, m = 500, 16
    w = synth.make_weight(dt, n, k, seed=k)
    x = np.random.default_rng(k).standard_normal((m, k)).astype(np.float32)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    want = exact_dots(O, dt, w, x, n, k)
    cpu = np.linalg.norm(O.matmul(int(dt), x, w, n) - want) / np.linalg.norm(want)
    got = np.linalg.norm(t.matmul_t(torch.from_numpy(x).to(DEV)).cpu().numpy().astype(np.float64) - want) / np.linalg.norm(want)
    assert got <= 1.04 * cpu, (dt.name, k, got, cpu)
