"""GPU parity of the tensor-core paths (more than one activation row) against the CPU oracle.

Two kernels serve these shapes. Up to 64 rows on Q4_0 / Q8_0 / Q4_K weights the integer kernel (tcgen05 kind::i8,
exact block sums, f32 scaling as the CPU code does it): it is held to the reference's own metric
|g - w| <= 2e-3 * max(|w|, 1). Above 64 rows, and for Q6_K, the fp16-operand kernel: its error is proportional
to the output scale, so it is held to 5e-3 of the output rms and to 1e-2 elementwise with the floor at the rms;
what it reaches under the reference's floor of 1 is printed, not asserted."""
import numpy as np
import pytest
import torch

from xn_b200 import synth
from xn_b200.dtypes import GgmlDType as D

pytestmark = pytest.mark.gpu
WEIGHT_TYPES = [D.Q4_0, D.Q8_0, D.Q4K, D.Q6K]
DEV = "cuda:0"
TOL_MMA = 1e-2


@pytest.fixture(scope="module")
def Q():
    from xn_b200 import quantized
    quantized.init(DEV)
    return quantized


def _integer_exact(dt, m):
    """Which (format, rows) the integer tensor-core kernel serves."""
    return dt in (D.Q4_0, D.Q8_0, D.Q4K) and 2 <= m <= 64


def _check(got, want, what, exact=False):
    """Bars of the tensor-core paths. exact: the integer kernel, judged by the reference's own metric at 2e-3.

    fp16 operand rounding gives an absolute error proportional to the output scale, so the unit of the
    comparison is the rms of the reference output: (1) max |g - w| / rms(w) <= 5e-3 (two times
    tighter than the 1e-2 the task allows an MMA path); (2) the reference's own elementwise metric
    |g - w| <= tol * max(|w|, floor) with tol = 1e-2 and the floor at rms(w) instead of the constant 1
    (a floor of 1 is only meaningful for outputs of order 1; it is printed for information)."""
    got = np.asarray(got, np.float64)
    want = np.asarray(want, np.float64)
    rms = max(float(np.sqrt((want ** 2).mean())), 1e-30)
    diff = np.abs(got - want)
    e_rms = diff.max() / rms
    e_floor_rms = (diff / np.maximum(np.abs(want), rms)).max()
    e_floor_one = (diff / np.maximum(np.abs(want), 1.0)).max()
    print(f"{what}: err/rms {e_rms:.2e}, elementwise (floor rms) {e_floor_rms:.2e}, elementwise (floor 1) {e_floor_one:.2e}, rms {rms:.3g}")
    if exact:
        assert e_floor_one <= 2e-3, f"{what}: reference metric {e_floor_one:.3e} on the integer-exact kernel"
    assert e_rms <= 5e-3, f"{what}: max error / rms {e_rms:.3e}"
    assert e_floor_rms <= TOL_MMA, f"{what}: elementwise {e_floor_rms:.3e}"
    return e_rms


@pytest.mark.parametrize("dt", WEIGHT_TYPES)
@pytest.mark.parametrize("m", [17, 32, 63, 64, 100, 256, 300])
def test_prefill_small_shapes(Q, O, dt, m):
    n, k = 200, dt.block_size * (4 if dt.block_size == 256 else 9)   # 32-blocks: k = 288 (not a multiple of 64)
    w = synth.make_weight(dt, n, k, seed=200)
    x = synth.make_activation(m, k, seed=200 + m)
    x[0, :] = 0.0
    x[1, :] *= 1e-4
    x[2, :] *= 3e3
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    got = t.matmul_t(torch.from_numpy(x).to(DEV)).cpu().numpy()
    want = O.matmul(int(dt), x, w, n)
    # Rows 1 and 2 are the same distribution at 1e-4 and 3e3 times the scale. The reference's metric
    # has an absolute floor (max(|w|, 1)) that only means something at the natural scale of the data,
    # so each row is judged in units where its activations are N(0,1).
    for rows, unit in ((slice(0, 1), 1.0), (slice(1, 2), 1e-4), (slice(2, 3), 3e3), (slice(3, m), 1.0)):
        if want[rows].size and np.abs(want[rows]).max() > 0:
            _check(got[rows] / unit, want[rows] / unit, f"{dt.name} m={m} rows {rows}", exact=_integer_exact(dt, m))
        else:
            assert not got[rows].any()


@pytest.mark.parametrize("dt", WEIGHT_TYPES)
@pytest.mark.parametrize("n", [1, 127, 128, 129, 385])
def test_prefill_ragged_n(Q, O, dt, n):
    k, m = 1024, 48
    w = synth.make_weight(dt, n, k, seed=210)
    x = synth.make_activation(m, k, seed=211)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    buf = torch.full((m * n + 128,), 777.0, device=DEV)
    out = buf[:m * n].view(m, n)
    t.matmul_t(torch.from_numpy(x).to(DEV), out=out)
    assert torch.all(buf[m * n:] == 777.0), "wrote past the output"
    _check(out.cpu().numpy(), O.matmul(int(dt), x, w, n), f"{dt.name} n={n}", exact=_integer_exact(dt, m))


@pytest.mark.parametrize("dt", WEIGHT_TYPES)
def test_prefill_half_precision_io_and_bias(Q, O, dt):
    n, k, m = 256, 2048, 40
    w = synth.make_weight(dt, n, k, seed=220)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    x = synth.make_activation(m, k, seed=221)
    for td in (torch.float16, torch.bfloat16):
        xh = torch.from_numpy(x).to(td)
        want = O.matmul(int(dt), xh.float().numpy(), w, n)
        got = t.matmul_t(xh.to(DEV))
        assert got.dtype == td
        rms = float(np.sqrt((want.astype(np.float64) ** 2).mean()))
        err = np.abs(got.float().cpu().numpy() - want) / np.maximum(np.abs(want), rms)   # floor at the output scale
        assert err.max() <= (1e-2 if td == torch.float16 else 2e-2), (dt.name, td, err.max())
    bias = synth.make_activation(1, n, seed=222)[0]
    host = t.forward_host(x, bias)
    _check(host, O.matmul(int(dt), x, w, n) + bias, f"{dt.name} forward_host m={m}")


FULL = [
    ("C2", D.Q8_0, 11008, 4096, (64, 128, 512)),
    ("C3", D.Q4K, 14336, 4096, (32, 64, 512)),
    ("C1", D.Q4_0, 4096, 4096, (48, 512)),
    ("C4", D.Q6K, 128256, 4096, (32,)),
]


@pytest.mark.parametrize("name,dt,n,k,ms", FULL)
def test_prefill_full_size_configs(Q, O, name, dt, n, k, ms):
    w = synth.make_weight(dt, n, k, seed=0)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    for m in ms:
        x = synth.make_activation(m, k, seed=0)
        got = t.matmul_t(torch.from_numpy(x).to(DEV)).cpu().numpy()
        _check(got, O.matmul(int(dt), x, w, n, threads=O.hw_threads()), f"{name} m={m}", exact=_integer_exact(dt, m))


def test_prefill_device_status_is_clean(Q):
    import ctypes
    from xn_b200 import _lib
    bits = ctypes.c_uint(123)
    _lib.check(_lib.lib().xnq_device_status(ctypes.byref(bits)))
    assert bits.value == 0, f"device status bits {bits.value:#x}"


def _f32_bound(O, dt, w, x, n, k):
    """What exact block sums that are scaled and added in f32 may differ by: at most two rounded terms per 32 elements on each side, of
    partial sums that stay below sum |w| |x| (doubled for min terms that do not cancel in it)."""
    dense = np.abs(O.to_float(int(dt), w, n * k).reshape(n, k)).astype(np.float64)
    return 4 * (k / 16 + 8) * 2.0 ** -24 * (np.abs(x).astype(np.float64) @ dense.T + np.abs(x).max() * dense.max() * 32)


# the integer kernel around its operand row counts (16, 32, 48, 64) and the row counts where other kernels take over, over one step, a
# partial step, tiles that several CTAs share, and rows of a last tile (a CTA has two steps here; the test behind it has the long runs)
@pytest.mark.parametrize("dt", WEIGHT_TYPES)
@pytest.mark.parametrize("m", [4, 5, 6, 16, 17, 32, 33, 48, 49, 64])
def test_integer_kernel_row_and_step_edges(Q, O, dt, m):
    if dt is D.Q6K and m > 16:
        pytest.skip("more than 16 rows of Q6_K run on fp16 operands")
    for n, k in ((3, 256), (130, 256 * 5), (129, 256 * 13)) if dt.block_size == 256 else ((3, 32), (130, 1312), (129, 3360)):
        w = synth.make_weight(dt, n, k, seed=m + n)
        x = synth.make_activation(m, k, seed=m + k)
        t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
        got = t.matmul_t(torch.from_numpy(x).to(DEV)).cpu().numpy().astype(np.float64)
        assert (np.abs(got - O.matmul(int(dt), x, w, n)) <= _f32_bound(O, dt, w, x, n, k)).all(), (dt.name, m, n, k)


# two to four rows of Q4_0 / Q8_0, on both sides of every line between the dp4a and the tensor-core kernel (k 256, 512, 3072, 4096, 5632, 8192;
# n 512, 3072, 6144, 8192), in every type of rows and with rows apart, against the kernel that the option imma = 0 leaves and the oracle
@pytest.mark.parametrize("dt", [D.Q4_0, D.Q8_0])
@pytest.mark.parametrize("n,k", [(511, 5632), (511, 5664), (512, 4096), (512, 3072), (512, 3104), (513, 8192), (513, 8224), (3071, 3104), (3072, 8224), (5, 512), (6144, 512),
                                 (6143, 512), (6144, 544), (6144, 256), (8191, 5664), (8192, 5664), (8192, 5632)])
def test_two_to_four_rows_on_either_kernel(Q, O, dt, n, k):
    from xn_b200 import _lib
    L = _lib.lib()
    w = synth.make_weight(dt, n, k, seed=n)
    x = synth.make_activation(4, 2 * k, seed=k)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    for act in (torch.float32, torch.float16, torch.bfloat16):
        xd = torch.from_numpy(x).to(act).to(DEV)[:, :k]
        rows = xd.float().cpu().numpy()
        want = O.matmul(int(dt), rows, w, n, threads=O.hw_threads())
        bound = _f32_bound(O, dt, w, rows, n, k) if act is torch.float32 else \
            2e-5 * np.abs(want).max() + np.abs(want) * 2.0 ** (-11 if act is torch.float16 else -8)   # and rounded to the result's type
        for m in (2, 3, 4):
            for imma in (1, 0):
                try:
                    _lib.check(L.xnq_set_option(b"imma", imma))
                    got = t.matmul_t(xd[:m])
                finally:
                    _lib.check(L.xnq_set_option(b"imma", 1))
                assert got.dtype is act
                assert (np.abs(got.float().cpu().numpy().astype(np.float64) - want[:m]) <= bound[:m]).all(), (dt.name, m, n, k, imma, act)


# Every CTA of the integer kernel takes an equal run of the (tile, step) space: here more steps than twice the stages of any of its rings
# but the two of eight (operand 2 or 3, activations 2 to 8, side 8), so every barrier is met in both parities, and the long rings wrap.
@pytest.mark.parametrize("dt", WEIGHT_TYPES)
def test_integer_kernel_long_runs_of_steps(Q, O, dt):
    n, k = 148 * 128 + 1, 256 * 13 - (0 if dt.block_size == 256 else 64)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert -(-n // 128) * 13 >= sms * 13
    w = synth.make_weight(dt, n, k, seed=31)
    x = synth.make_activation(64, k, seed=32)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    want, bound = O.matmul(int(dt), x, w, n, threads=O.hw_threads()), _f32_bound(O, dt, w, x, n, k)
    for m in (6, 16) if dt is D.Q6K else (5, 16, 17, 32, 33, 48, 64):
        got = t.matmul_t(torch.from_numpy(x[:m]).to(DEV)).cpu().numpy().astype(np.float64)
        assert (np.abs(got - want[:m]) <= bound[:m]).all(), (dt.name, m)


# the fp16 kernel: one and two accumulators, tiles that end with 1 and 16 rows, k-steps that do not fill a super-step or a stage ring,
# output types that are stored whole, a weight of less than a tile and one row more than a tile
@pytest.mark.parametrize("dt", WEIGHT_TYPES)
@pytest.mark.parametrize("m", [65, 128, 129, 257, 513])
def test_fp16_kernel_tile_and_step_edges(Q, O, dt, m):
    for n, k in ((3, 256), (129, 256 * 5)) if dt.block_size == 256 else ((3, 32), (129, 96), (40, 1312)):
        w = synth.make_weight(dt, n, k, seed=m + n)
        x = synth.make_activation(m, k, seed=m + k)
        t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
        xd = torch.from_numpy(x).to(DEV)
        want = O.matmul(int(dt), x, w, n)
        got = t.matmul_t(xd)
        _check(got.cpu().numpy(), want, f"{dt.name} m={m} n={n} k={k}")
        half = t.matmul_t(xd, out=torch.empty(m, n, dtype=torch.float16, device=DEV))
        assert torch.allclose(half.float(), got, rtol=2.0 ** -10, atol=1e-4 * float(got.abs().max()))   # rounded once; parts of a split tile may meet in another order


# 16-bit results of the fp16 kernel on pairs of CTAs: an odd number of row tiles and one row in the last, m-tiles of unequal halves, k-steps that
# do not fill a super-step; against the oracle, and against the f32 results of single CTAs
@pytest.mark.parametrize("dt", WEIGHT_TYPES)
@pytest.mark.parametrize("n,k,m", [(3841, 2048, 881), (3841, 2048, 1024), (14209, 4096, 209)])
def test_fp16_kernel_on_pairs(Q, O, dt, n, k, m):
    k -= 0 if dt.block_size == 256 else 32
    w = synth.make_weight(dt, n, k, seed=m)
    x = synth.make_activation(m, k, seed=m + k)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    xd = torch.from_numpy(x).to(DEV)
    got = t.matmul_t(xd)
    _check(got.cpu().numpy(), O.matmul(int(dt), x, w, n, threads=O.hw_threads()), f"{dt.name} m={m} n={n} k={k}")
    for out in (torch.float16, torch.bfloat16):
        buf = torch.full((m * n + 128,), 777.0, device=DEV, dtype=out)
        half = t.matmul_t(xd, out=buf[:m * n].view(m, n))
        assert torch.all(buf[m * n:] == 777.0), "wrote past the output"
        assert torch.allclose(half.float(), got, rtol=2.0 ** (-10 if out is torch.float16 else -7), atol=1e-4 * float(got.abs().max()))


# several tiles of unequal widths (256 and 192, 256 and 16 rows) on one CTA's single accumulator, whose halves are given back one by one; rows of y that
# start on 16 bytes (n a multiple of 8) and rows that do not
@pytest.mark.parametrize("dt", WEIGHT_TYPES)
@pytest.mark.parametrize("n,m", [(515, 700), (512, 700), (516, 528), (1029, 260)])
def test_fp16_kernel_unequal_tiles(Q, O, dt, n, m):
    k = 512 if dt.block_size == 256 else 352
    w = synth.make_weight(dt, n, k, seed=m + n)
    x = synth.make_activation(m, k, seed=m)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    xd = torch.from_numpy(x).to(DEV)
    got = t.matmul_t(xd)
    _check(got.cpu().numpy(), O.matmul(int(dt), x, w, n, threads=O.hw_threads()), f"{dt.name} m={m} n={n}")
    wide = torch.full((m, n + 7), 777.0, dtype=torch.bfloat16, device=DEV)   # rows apart
    t.matmul_t(xd, out=wide[:, :n]) if n % 8 else t.matmul_t(xd, out=wide.view(-1)[: m * n].view(m, n))
    half = wide[:, :n] if n % 8 else wide.view(-1)[: m * n].view(m, n)
    assert torch.allclose(half.float(), got, rtol=2.0 ** -7, atol=1e-4 * float(got.abs().max()))


# a tile's last super-step lacks some of its k-steps (k-steps not a multiple of two or four) while the CTA goes on to further tiles: the warps of a missing
# step must neither miss nor outrun a phase of a stage's barrier. f32 (ranges of k-steps) and 16-bit (whole tiles)
@pytest.mark.parametrize("dt", [d for d in WEIGHT_TYPES if d.block_size == 32])
@pytest.mark.parametrize("n,k,m", [(640, 8384, 814), (640, 8288, 814), (1029, 8512, 700), (300, 1312, 814), (4096, 352, 257), (2048, 96, 1100), (520, 4128, 100)])
def test_fp16_kernel_missing_steps(Q, O, dt, n, k, m):
    w = synth.make_weight(dt, n, k, seed=m + n)
    x = synth.make_activation(m, k, seed=m)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    xd = torch.from_numpy(x).to(DEV)
    want = O.matmul(int(dt), x, w, n, threads=O.hw_threads())
    for _ in range(20):
        got = t.matmul_t(xd)
    _check(got.cpu().numpy(), want, f"{dt.name} m={m} n={n} k={k}")
    half = t.matmul_t(xd, out=torch.empty(m, n, dtype=torch.bfloat16, device=DEV))
    assert torch.allclose(half.float(), got, rtol=2.0 ** -7, atol=1e-4 * float(got.abs().max()))


# tiles in more parts than are requested at once (28 of two steps; 16 and more rows), CTAs whose range starts in one tile and ends in another, and with both ends
# inside one; the parts are added in k order, so that every call has the same bits
@pytest.mark.parametrize("dt", WEIGHT_TYPES)
@pytest.mark.parametrize("n,k", [(129, 14336), (3 * 128, 256 * 5), (1000, 2048), (128 * 90, 1024)])
def test_integer_kernel_parts_of_tiles(Q, O, dt, n, k):
    w = synth.make_weight(dt, n, k, seed=n)
    x = synth.make_activation(64, k, seed=k)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    want, bound = O.matmul(int(dt), x, w, n, threads=O.hw_threads()), _f32_bound(O, dt, w, x, n, k)
    for m in (6, 16) if dt is D.Q6K else (5, 16, 20, 33, 48, 64):
        xd = torch.from_numpy(x[:m]).to(DEV)
        got = t.matmul_t(xd)
        assert (np.abs(got.cpu().numpy().astype(np.float64) - want[:m]) <= bound[:m]).all(), (dt.name, m)
        for _ in range(10):
            assert torch.equal(t.matmul_t(xd), got), (dt.name, m)


# 16-bit results take as many tiles of activation rows as finish first: 8 of 192 rows instead of 6 of 256, 10 of 64 instead of 3, 2 of 80 instead of 1, 7 of 256
# on single CTAs where pairs would take a round more; bits of a tile's sums do not depend on its width, so that f32 results rounded once are the same
@pytest.mark.parametrize("dt", WEIGHT_TYPES)
@pytest.mark.parametrize("n,m", [(3584, 1459), (1100, 600), (4100, 150), (2615, 1773)])
def test_fp16_kernel_number_of_tiles(Q, O, dt, n, m):
    k = 768 if dt.block_size == 256 else 736
    w = synth.make_weight(dt, n, k, seed=m + n)
    x = synth.make_activation(m, k, seed=m)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    xd = torch.from_numpy(x).to(DEV)
    got = t.matmul_t(xd)
    _check(got.cpu().numpy(), O.matmul(int(dt), x, w, n, threads=O.hw_threads()), f"{dt.name} m={m} n={n}")
    for out in (torch.float16, torch.bfloat16):
        buf = torch.full((m * n + 128,), 777.0, device=DEV, dtype=out)
        half = t.matmul_t(xd, out=buf[:m * n].view(m, n))
        assert torch.all(buf[m * n:] == 777.0), "wrote past the output"
        assert torch.allclose(half.float(), got, rtol=2.0 ** (-10 if out is torch.float16 else -7), atol=1e-4 * float(got.abs().max()))


# one tile of 176 rows on 70 CTAs instead of two on 140
@pytest.mark.parametrize("dt", WEIGHT_TYPES)
def test_fp16_kernel_keeps_off_sms(Q, O, dt):
    test_fp16_kernel_number_of_tiles(Q, O, dt, 8910, 165)


def _status_is_clean():
    import ctypes

    from xn_b200 import _lib
    bits = ctypes.c_uint(0)
    _lib.check(_lib.lib().xnq_device_status(ctypes.byref(bits)))
    assert bits.value == 0, f"device status {bits.value:#x}"


# Rows of a wider buffer: nothing past a row's end is written, between the rows or behind the last one, in 16-byte stores (n and the rows' distance are whole
# pieces of them) and in single ones
@pytest.mark.parametrize("dt", WEIGHT_TYPES)
@pytest.mark.parametrize("n,m,gap", [(515, 700, 7), (512, 700, 8), (516, 528, 12), (1029, 260, 3), (120, 70, 8), (1, 300, 1)])
def test_fp16_kernel_keeps_inside_its_rows(Q, dt, n, m, gap):
    k = 512 if dt.block_size == 256 else 352
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(synth.make_weight(dt, n, k, seed=m + n), (n, k), dt), DEV)
    x = torch.from_numpy(synth.make_activation(m, k, seed=m)).to(DEV)
    for out in (torch.float32, torch.float16, torch.bfloat16):
        want = t.matmul_t(x, out=torch.empty(m, n, dtype=out, device=DEV))
        wide = torch.full((m, n + gap), 777.0, dtype=out, device=DEV)
        t.matmul_t(x, out=wide[:, :n])
        assert torch.all(wide[:, n:] == 777.0), (dt.name, out)
        if out is torch.float32:   # parts of a split tile may meet in another order
            assert torch.allclose(wide[:, :n], want, rtol=0, atol=1e-5 * float(want.abs().max()))
        else:
            assert torch.equal(wide[:, :n], want)


# As test_fp16_kernel_missing_steps, each of the calls against the oracle, and no wait ran out
@pytest.mark.parametrize("dt", [d for d in WEIGHT_TYPES if d.block_size == 32])
@pytest.mark.parametrize("n,k,m", [(640, 8384, 814), (1029, 8512, 700), (300, 1312, 814), (2048, 96, 1100), (520, 4128, 100)])
def test_fp16_kernel_missing_steps_in_every_call(Q, O, dt, n, k, m):
    w = synth.make_weight(dt, n, k, seed=m + n)
    x = synth.make_activation(m, k, seed=m)
    t = Q.QCudaTensor.from_qtensor(Q.QTensor(w, (n, k), dt), DEV)
    xd = torch.from_numpy(x).to(DEV)
    want = O.matmul(int(dt), x, w, n, threads=O.hw_threads())
    for i in range(20):
        _check(t.matmul_t(xd).cpu().numpy(), want, f"{dt.name} m={m} n={n} k={k}, call {i}")
    _status_is_clean()
