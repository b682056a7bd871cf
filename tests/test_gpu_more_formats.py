"""Q4_1, Q5_0, Q5_1, Q2_K, Q3_K, Q5_K weights and the Q8_1 activation format on the GPU, through the C-ABI, against the CPU
oracle: upload / canonical bytes round trip, to_float bit for bit, the Q8_1 quantizer byte for byte, matmul within the
reference's metric |g - w| <= 2e-3 * max(|w|, 1) for one row, small batches and a prefill-sized batch."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from xn_b200 import synth
from xn_b200.dtypes import GgmlDType as D

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
FORMATS = [D.Q4_1, D.Q5_0, D.Q5_1, D.Q2K, D.Q3K, D.Q5K]


@pytest.fixture(scope="module", autouse=True)
def _init():
    from xn_b200 import quantized
    O.build()
    quantized.init(DEV)


def _upload(dt, n, k, seed=0, **kw):
    from xn_b200 import quantized as Q
    blocks = synth.make_weight(dt, n, k, seed=seed)
    return blocks, Q.QCudaTensor.from_qtensor(Q.QTensor(blocks, (n, k), dt), DEV, **kw)


@pytest.mark.parametrize("dt", FORMATS)
def test_upload_round_trip_and_to_float_bit_exact(dt):
    n, k = 37, 1024
    blocks, w = _upload(dt, n, k, seed=21)
    assert w.dtype() == dt and tuple(w.shape()) == (n, k)
    assert np.array_equal(w.data(), blocks)
    got = w.dequantize(torch.float32).cpu().numpy().reshape(-1)
    want = O.to_float(int(dt), blocks, n * k)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    for tdt in (torch.float16, torch.bfloat16):   # narrower outputs are the f32 values rounded once
        got16 = w.dequantize(tdt).float().cpu().numpy().reshape(-1)
        assert np.array_equal(got16, torch.from_numpy(want).to(tdt).float().numpy())


@pytest.mark.parametrize("dt", FORMATS)
@pytest.mark.parametrize("n,k,m", [(64, 256, 1), (333, 1024, 1), (200, 4096, 5), (96, 2048, 16), (130, 512, 40)])
def test_matmul_against_the_oracle(dt, n, k, m):
    blocks, w = _upload(dt, n, k, seed=22)
    x = synth.make_activation(m, k, seed=23)
    got = w.matmul_t(torch.from_numpy(x).to(DEV)).cpu().numpy()
    want = O.matmul(int(dt), x, blocks, n)
    err = np.abs(got - want) / np.maximum(np.abs(want), 1.0)
    assert got.shape == (m, n) and err.max() <= 2e-3, (dt.name, n, k, m, float(err.max()))


@pytest.mark.parametrize("xdt", [torch.float32, torch.float16, torch.bfloat16])
def test_q8_1_activation_blocks_byte_exact(xdt):
    from xn_b200.quantized import quantize_act
    g = torch.Generator().manual_seed(24)
    x = torch.randn(7, 512, generator=g)
    x[0] = 0
    x[1, :32] = torch.linspace(-127, 127, 32) * 0.5
    x[2, 5] = 1e4
    xd = x.to(xdt)
    got = quantize_act(xd.to(DEV), D.Q8_1).cpu().numpy()
    want = np.concatenate([O.from_float(int(D.Q8_1), xd[r].float().numpy()) for r in range(x.shape[0])])
    assert np.array_equal(got, want)


def test_half_outputs_sharded_upload_and_error_paths():
    from xn_b200 import quantized as Q
    from xn_b200._lib import XnqError
    dt, n, k = D.Q5K, 64, 512
    blocks, w = _upload(dt, n, k, seed=25)
    x = torch.from_numpy(synth.make_activation(3, k, seed=26)).to(DEV)
    y32 = w.matmul_t(x)
    for tdt in (torch.float16, torch.bfloat16):
        y = w.matmul_t(x.to(tdt))
        assert y.dtype is tdt
        want = torch.from_numpy(O.matmul(int(dt), x.to(tdt).float().cpu().numpy(), blocks, n)).to(DEV)
        assert torch.allclose(y.float(), want, rtol=1e-2, atol=2e-2)
    # an N-shard of two holds half of the rows and computes exactly those columns
    sh = Q.QCudaTensor.from_qtensor(Q.QTensor(blocks, (n, k), dt), DEV, shard_rank=1, shard_count=2)
    assert torch.equal(sh.matmul_t(x), y32[:, n // 2:])
    # the 32-element formats refuse an odd number of blocks, as the reference's dots do
    b96, w96 = _upload(D.Q4_1, 8, 96, seed=27)
    with pytest.raises(XnqError):
        w96.matmul_t(torch.zeros(1, 96, device=DEV))


# around the edges of the kernel's splits: one piece of 32 or one super-block, the k where more warps share a row (64 and 128 pieces) and a
# ragged last round of pieces; odd row counts; every tile of activation rows (1, 2, 4, 8, 16) with remainders
@pytest.mark.parametrize("dt", FORMATS)
@pytest.mark.parametrize("kb", [1, 7, 8, 15, 16, 21])
def test_matmul_row_and_tile_edges(dt, kb):
    k = 256 * kb if dt.block_size == 256 else 192 * kb - 64 * (kb == 1)
    for n, m in ((1, 2), (3, 3), (17, 8), (33, 9), (2, 35)):
        blocks, w = _upload(dt, n, k, seed=kb + n)
        x = synth.make_activation(m, k, seed=kb + m)
        xd = torch.from_numpy(x).to(DEV)
        got = w.matmul_t(xd)
        want = O.matmul(int(dt), x, blocks, n)
        # both sides add at most two rounded f32 terms per 32 elements to a running f32 sum: k / 16 roundings of partial sums that stay
        # below sum |w| |x| (doubled: the min terms do not cancel in it; the activations' own rounding is common to both sides)
        dense = np.abs(O.to_float(int(dt), blocks, n * k).reshape(n, k)).astype(np.float64)
        bound = 4 * (k / 16 + 8) * 2.0 ** -24 * (np.abs(x).astype(np.float64) @ dense.T + np.abs(x).max() * dense.max() * 32)
        assert (np.abs(got.cpu().numpy().astype(np.float64) - want) <= bound).all(), (dt.name, n, k, m)
        for r in (0, m - 1):   # the sum's order depends on k alone
            assert torch.equal(w.matmul_t(xd[r:r + 1]), got[r:r + 1])


# How many activation rows a warp takes, and whether a CTA walks over several groups of weight rows, depends on the shape (one, two and four warps
# to a row of k; many and few groups; tiles of eight, four, two rows and one): a row's bits do not.
@pytest.mark.parametrize("dt", FORMATS)
@pytest.mark.parametrize("n,k,ms", [(9001, 512, (5, 8, 9, 24)), (4097, 2048, (2, 7, 17)), (3001, 4096, (3, 8, 13)), (130, 1024, (2, 3, 4, 5, 10, 40)), (1, 512, (9,))])
def test_a_rows_bits_do_not_depend_on_the_batch(dt, n, k, ms):
    from xn_b200 import quantized as Q
    Q.init(DEV)
    w = synth.make_weight(dt, n, k, seed=n)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    x = torch.from_numpy(synth.make_activation(max(ms), k, seed=k)).to(DEV)
    alone = torch.cat([t.matmul_t(x[i:i + 1]) for i in range(max(ms))])
    for m in ms:
        buf = torch.full((m * n + 64,), 777.0, device=DEV)
        t.matmul_t(x[:m], out=buf[: m * n].view(m, n))
        assert torch.equal(buf[: m * n].view(m, n), alone[:m]) and torch.all(buf[m * n:] == 777.0), (dt.name, n, k, m)


# The same on both sides of the lines where eight rows are taken for four, and where a tile's CTAs walk or not.
@pytest.mark.parametrize("dt", FORMATS)
@pytest.mark.parametrize("n,k,ms", [(2710, 1280, (2, 3, 4, 6, 8)), (1430, 1024, (3, 4, 5, 8)), (4500, 1536, (6, 8)), (5000, 2816, (7,)), (2050, 8448, (5, 8, 9))])
def test_a_rows_bits_where_a_rule_turns(dt, n, k, ms):
    test_a_rows_bits_do_not_depend_on_the_batch(dt, n, k, ms)


# Many activation rows: how many CTAs share a tile's weight rows depends on the number of tiles (1200 rows: 150 tiles of eight; 2376: one more than there are
# places for CTAs; 2369: the last of one row). Every row has the bits it has alone, and every element is written, once and nowhere else.
@pytest.mark.parametrize("dt", FORMATS)
@pytest.mark.parametrize("n,k,m", [(300, 512, 1200), (67, 256, 2376), (1030, 256, 2369), (517, 2048, 600), (4097, 512, 100)])
def test_many_activation_rows(dt, n, k, m):
    from xn_b200 import quantized as Q
    Q.init(DEV)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(synth.make_weight(dt, n, k, seed=n), (n, k), dt), DEV)
    x = torch.from_numpy(synth.make_activation(m, k, seed=k)).to(DEV)
    buf = torch.full((m * n + 64,), 777.0, device=DEV)
    t.matmul_t(x, out=buf[: m * n].view(m, n))
    assert torch.all(buf[m * n:] == 777.0)
    got = buf[: m * n].view(m, n)
    assert torch.equal(got, torch.cat([t.matmul_t(part) for part in x.split(4)]))
    for i in (0, m // 2, m - 1):
        assert torch.equal(got[i], t.matmul_t(x[i:i + 1])[0])
