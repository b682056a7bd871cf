"""A workspace that was once large enough for a call stays large enough: programs keep the size with their plans."""
import ctypes

import numpy as np
import pytest

from conftest import assert_close_ref

torch = pytest.importorskip("torch")
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

from xn_b200 import synth  # noqa: E402
from xn_b200.dtypes import GgmlDType as D  # noqa: E402

DEV = torch.device("cuda:0")
GUARD = 4096


def _up(v):
    return (v + 255) // 256 * 256


def earlier_answer(dt, m, k, n):
    """What xnq_matmul_workspace_bytes answered for m rows when the integer tensor-core kernel came in."""
    if dt not in (D.Q4_0, D.Q8_0, D.Q4K, D.Q6K):   # the canonical activation blocks
        block, size = {D.Q4_1: (32, 36), D.Q5_0: (32, 34), D.Q5_1: (32, 36)}.get(dt, (256, 292))
        return _up(m * (k // block) * size)
    rows, block = min(m, 16), 32 if dt in (D.Q4_0, D.Q8_0) else 256
    need = _up(rows * k) + _up(rows * (k // block) * 4) + _up(rows * (k // 16) * 2)
    if dt is not D.Q6K and m >= 2:
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        cols, steps, tiles = (16 if m <= 16 else 32 if m <= 32 else 64), -(-k // 256), -(-n // 128)
        need = max(need, _up(steps * 2 * cols * 128) + _up(steps * cols * 32) + _up(tiles * 4) + _up(2 * sms * cols * 512) + _up(sms * cols * 512) + 256)
    if m > 16:
        m16 = -(-m // 16) * 16
        tiles = -(-n // 128) * -(-m16 // 256)
        need = max(need, -(-k // 64) * m16 * 128 + _up(m16 * 4) + _up(8 * tiles) + 256)
    return need


@pytest.mark.parametrize("m", [1, 2, 5, 6, 11, 16, 17, 33, 48, 64, 65])
@pytest.mark.parametrize("dt", [D.Q4_0, D.Q8_0, D.Q4K, D.Q6K, D.Q4_1, D.Q5_0, D.Q5_1, D.Q2K, D.Q3K, D.Q5K], ids=lambda d: d.name)
def test_a_workspace_of_the_earlier_size_is_accepted_and_not_overrun(O, dt, m):
    from xn_b200 import _lib
    from xn_b200 import quantized as Q
    L = _lib.lib()
    n, k = 300, 1280
    blocks = synth.make_weight(dt, n, k, seed=m)
    x = synth.make_activation(m, k, seed=m + 1)
    w = Q.QCudaTensor.from_qtensor(Q.QTensor(blocks, (n, k), dt), DEV)
    size = earlier_answer(dt, m, k, n)
    if dt is not D.Q6K:
        assert L.xnq_matmul_workspace_bytes(w._h, m) <= size
    xd, y = torch.from_numpy(x).to(DEV), torch.full((m, n), 7.0, device=DEV)
    buf = torch.full((size + GUARD,), 0xA5, dtype=torch.uint8, device=DEV)
    assert buf.data_ptr() % 256 == 0
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    _lib.check(L.xnq_matmul_t(w._h, p(xd), int(D.F32), m, k, p(y), int(D.F32), n, p(buf), size, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert bool((buf[size:] == 0xA5).all())
    want = O.matmul(int(dt), x, blocks, n)
    if m <= (16 if dt is D.Q6K else 64) or dt not in (D.Q4_0, D.Q8_0, D.Q4K, D.Q6K):
        assert_close_ref(y.cpu().numpy(), want, 2e-3, f"{dt.name} m={m}")
    else:   # fp16 operands: 5e-3 of the outputs' rms
        assert np.abs(y.cpu().numpy() - want).max() <= 5e-3 * np.sqrt((want.astype(np.float64) ** 2).mean())


@pytest.mark.parametrize("dt", [D.Q4_0, D.Q8_0, D.Q4K, D.Q6K, D.Q5_0, D.Q5K], ids=lambda d: d.name)
def test_the_answer_for_more_rows_serves_fewer(dt):
    from xn_b200 import _lib
    from xn_b200 import quantized as Q
    n, k = 300, 1280
    w = Q.QCudaTensor.from_qtensor(Q.QTensor(synth.make_weight(dt, n, k, seed=3), (n, k), dt), DEV)
    sizes = [_lib.lib().xnq_matmul_workspace_bytes(w._h, m) for m in range(1, 300)]
    assert sizes == sorted(sizes)
    if dt is D.Q6K:   # rows that run on the dp4a kernel ask for its codes alone
        assert sizes[4] == _lib.lib().xnq_act_image_bytes(int(D.Q8K), 5, k) < sizes[5]
