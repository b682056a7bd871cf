// GGUF <-> device layout conversion, full-tensor dequantize, bias add.
//
// None of this is on the decode hot path: relayout runs once per weight at upload, dequantize is
// the API's counterpart of Q8Tensor::dequantize (xn-core/src/cuda_backend/q8.rs:94-113). What
// matters here is exactness: dequantize is bit-identical to GgmlType::to_float, so every float
// operation is an explicit round-to-nearest intrinsic the compiler may not contract into an FMA.
#include <algorithm>

#include "xnq_common.cuh"
#include "xnq_unpack.cuh"

namespace xnq {

namespace {

constexpr int TPB = 256;

// ---- GGUF blocks -> device layout, one thread per block ------------------------------------------
__global__ void relayout_q4_0(const uint8_t *__restrict__ src, uint8_t *__restrict__ qs, __half *__restrict__ d,
                              int64_t n, int64_t nblk, int64_t dstride) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n * nblk) return;
  const int64_t row = i / nblk, b = i % nblk;
  const uint16_t *s = reinterpret_cast<const uint16_t *>(src + i * 18); // blocks are 2-byte aligned
  reinterpret_cast<uint16_t *>(d)[row * dstride + b] = s[0];
  uint16_t *o = reinterpret_cast<uint16_t *>(qs + i * 16);
#pragma unroll
  for (int j = 0; j < 8; j++) o[j] = s[1 + j];
}

__global__ void relayout_q8_0(const uint8_t *__restrict__ src, uint8_t *__restrict__ qs, __half *__restrict__ d,
                              int64_t n, int64_t nblk, int64_t dstride) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n * nblk) return;
  const int64_t row = i / nblk, b = i % nblk;
  const uint16_t *s = reinterpret_cast<const uint16_t *>(src + i * 34);
  reinterpret_cast<uint16_t *>(d)[row * dstride + b] = s[0];
  uint16_t *o = reinterpret_cast<uint16_t *>(qs + i * 32);
#pragma unroll
  for (int j = 0; j < 16; j++) o[j] = s[1 + j];
}

// one thread per 2 bytes of a 210-byte super-block (105 threads of work per block)
__global__ void relayout_q6k(const uint8_t *__restrict__ src, uint8_t *__restrict__ ql, uint8_t *__restrict__ qh,
                             int8_t *__restrict__ sc, __half *__restrict__ d, int64_t n, int64_t nsb, int64_t dstride) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n * nsb * 105) return;
  const int64_t blk = t / 105;
  const int w = (int)(t % 105); // 16-bit word index inside the block
  const uint16_t v = reinterpret_cast<const uint16_t *>(src + blk * 210)[w];
  if (w < 64) {
    reinterpret_cast<uint16_t *>(ql + blk * 128)[w] = v;
  } else if (w < 96) {
    reinterpret_cast<uint16_t *>(qh + blk * 64)[w - 64] = v;
  } else if (w < 104) {
    reinterpret_cast<uint16_t *>(sc + blk * 16)[w - 96] = v;
  } else {
    const int64_t row = blk / nsb, b = blk % nsb;
    reinterpret_cast<uint16_t *>(d)[row * dstride + b] = v;
  }
}

// Q4_K: blocks stay where they are; one thread per super-block re-packs the 12 scale bytes
template <bool TO_DEVICE>
__global__ void repack_q4k(const uint8_t *__restrict__ src, uint8_t *__restrict__ dst, int64_t nblocks) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nblocks) return;
  const uint4 *s = reinterpret_cast<const uint4 *>(src + i * 144);
  uint4 *o = reinterpret_cast<uint4 *>(dst + i * 144);
  uint4 hdr = s[0];
  const uint32_t in[3] = {hdr.y, hdr.z, hdr.w};
  uint32_t out[3];
  if (TO_DEVICE) k4_fields_from_gguf(in, out);
  else k4_fields_to_gguf(in, out);
  hdr.y = out[0];
  hdr.z = out[1];
  hdr.w = out[2];
  o[0] = hdr;
#pragma unroll
  for (int j = 1; j < 9; j++) o[j] = s[j];
}

// ---- device layout -> GGUF blocks ----------------------------------------------------------------
__global__ void canonical_q4_0(uint8_t *__restrict__ dst, const uint8_t *__restrict__ qs, const __half *__restrict__ d,
                               int64_t n, int64_t nblk, int64_t dstride) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n * nblk) return;
  const int64_t row = i / nblk, b = i % nblk;
  uint16_t *o = reinterpret_cast<uint16_t *>(dst + i * 18);
  o[0] = reinterpret_cast<const uint16_t *>(d)[row * dstride + b];
  const uint16_t *s = reinterpret_cast<const uint16_t *>(qs + i * 16);
#pragma unroll
  for (int j = 0; j < 8; j++) o[1 + j] = s[j];
}

__global__ void canonical_q8_0(uint8_t *__restrict__ dst, const uint8_t *__restrict__ qs, const __half *__restrict__ d,
                               int64_t n, int64_t nblk, int64_t dstride) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n * nblk) return;
  const int64_t row = i / nblk, b = i % nblk;
  uint16_t *o = reinterpret_cast<uint16_t *>(dst + i * 34);
  o[0] = reinterpret_cast<const uint16_t *>(d)[row * dstride + b];
  const uint16_t *s = reinterpret_cast<const uint16_t *>(qs + i * 32);
#pragma unroll
  for (int j = 0; j < 16; j++) o[1 + j] = s[j];
}

__global__ void canonical_q6k(uint8_t *__restrict__ dst, const uint8_t *__restrict__ ql, const uint8_t *__restrict__ qh,
                              const int8_t *__restrict__ sc, const __half *__restrict__ d, int64_t n, int64_t nsb,
                              int64_t dstride) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n * nsb * 105) return;
  const int64_t blk = t / 105;
  const int w = (int)(t % 105);
  uint16_t v;
  if (w < 64) {
    v = reinterpret_cast<const uint16_t *>(ql + blk * 128)[w];
  } else if (w < 96) {
    v = reinterpret_cast<const uint16_t *>(qh + blk * 64)[w - 64];
  } else if (w < 104) {
    v = reinterpret_cast<const uint16_t *>(sc + blk * 16)[w - 96];
  } else {
    const int64_t row = blk / nsb, b = blk % nsb;
    v = reinterpret_cast<const uint16_t *>(d)[row * dstride + b];
  }
  reinterpret_cast<uint16_t *>(dst + blk * 210)[w] = v;
}

// ---- dequantize: one thread per element, exact to_float arithmetic --------------------------------
template <typename T>
__device__ __forceinline__ T cast_out(float v);
template <>
__device__ __forceinline__ float cast_out<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half cast_out<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 cast_out<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

template <typename T>
__global__ void dequantize_kernel(WeightView w, T *__restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= w.n * w.k) return;
  const int64_t row = i / w.k;
  const int col = (int)(i % w.k);
  float v;
  switch (w.dtype) {
    case XNQ_Q4_0: v = deq_q4_0(w, row, col); break;
    case XNQ_Q8_0: v = deq_q8_0(w, row, col); break;
    case XNQ_Q4K: v = deq_q4k(w, row, col); break;
    default: v = deq_q6k(w, row, col); break;
  }
  out[i] = cast_out<T>(v);
}

__global__ void max_abs_kernel(WeightView w, unsigned int *out) {
  float m = 0.f;
  const int64_t total = w.n * w.k;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / w.k;
    const int col = (int)(i % w.k);
    float v;
    switch (w.dtype) {
      case XNQ_Q4_0: v = deq_q4_0(w, row, col); break;
      case XNQ_Q8_0: v = deq_q8_0(w, row, col); break;
      case XNQ_Q4K: v = deq_q4k(w, row, col); break;
      default: v = deq_q6k(w, row, col); break;
    }
    v = fabsf(v);
    if (v < 3.0e38f) m = fmaxf(m, v); // ignore inf / nan scales
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m)); // non-negative floats order like their bit patterns
}

// VEC values a thread (what its 16 bytes hold, where y's rows allow that) of four rows, all requested before any is stored. Bound by y's traffic; with a row
// to a CTA odd rows were bound by the number of CTAs (with the matmul before it, Q4_K 1819 x 768, 360 rows: 23.6 us, with four 21.4; 1820 x 768 the
// same 22.4). It starts while the matmul before it drains.
constexpr int BIAS_ROWS = 4;
template <typename T, int VEC>
__global__ void __launch_bounds__(TPB) add_bias_kernel(T *__restrict__ y, const T *__restrict__ bias, int64_t m, int64_t n, int64_t ldy, int y_dtype) {
  constexpr int ROWS = BIAS_ROWS;
  const int64_t c = ((int64_t)blockIdx.x * TPB + threadIdx.x) * VEC;
  pdl_launch_dependents();
  pdl_wait();
  if (c >= n) return;
  float b[VEC];
#pragma unroll
  for (int i = 0; i < VEC; i++) b[i] = bias_at(bias, y_dtype, c + i);
  for (int64_t r0 = (int64_t)blockIdx.y * ROWS; r0 < m; r0 += (int64_t)gridDim.y * ROWS) {
    __align__(16) T v[ROWS][VEC];
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
      const T *p = y + min(r0 + r, m - 1) * ldy + c;
      if (VEC > 1) *reinterpret_cast<uint4 *>(v[r]) = *reinterpret_cast<const uint4 *>(p);
      else v[r][0] = p[0];
    }
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
      if (r0 + r >= m) break;
      T *p = y + (r0 + r) * ldy + c;
#pragma unroll
      for (int i = 0; i < VEC; i++) v[r][i] = cast_out<T>(__fadd_rn(bias_at(v[r], y_dtype, i), b[i]));
      if (VEC > 1) *reinterpret_cast<uint4 *>(p) = *reinterpret_cast<const uint4 *>(v[r]);
      else p[0] = v[r][0];
    }
  }
}

inline unsigned grid_for(int64_t work) { return (unsigned)((work + TPB - 1) / TPB); }

} // namespace

int make_weight_maps(const WeightView &v, WeightMaps *maps) {
  if (v.n == 0) return XNQ_OK;
  using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  void *fn = nullptr;
  cudaDriverEntryPointQueryResult found;
  XNQ_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found));
  if (found != cudaDriverEntryPointSuccess || !fn) return fail(XNQ_ERR_UNSUPPORTED, "weight_upload: the driver has no cuTensorMapEncodeTiled");
  auto encode = [&](CUtensorMap *m, const void *base, int64_t row_bytes, uint32_t box_bytes, CUtensorMapSwizzle swizzle) {
    const cuuint64_t dims[2] = {(cuuint64_t)row_bytes, (cuuint64_t)v.n}, strides[1] = {(cuuint64_t)row_bytes};
    const cuuint32_t box[2] = {box_bytes, 128}, steps[2] = {1, 1};
    const CUresult r = reinterpret_cast<Encode>(fn)(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? XNQ_OK : fail(XNQ_ERR_CUDA, "weight_upload: cuTensorMapEncodeTiled of [%lld, %lld bytes] failed: %d", (long long)v.n, (long long)row_bytes, (int)r);
  };
  int rc = XNQ_OK;
  switch (v.dtype) {
    case XNQ_Q4K: rc = encode(&maps->codes, v.qs, v.k / QK_K * 144, 144, CU_TENSOR_MAP_SWIZZLE_NONE); break;
    case XNQ_Q4_0: rc = encode(&maps->codes, v.qs, v.k / 2, 128, CU_TENSOR_MAP_SWIZZLE_128B); break;
    case XNQ_Q8_0: rc = encode(&maps->codes, v.qs, v.k, 128, CU_TENSOR_MAP_SWIZZLE_128B); break;
    case XNQ_Q6K:
      rc = encode(&maps->codes, v.qs, v.k / 2, 128, CU_TENSOR_MAP_SWIZZLE_128B);
      if (rc == XNQ_OK) rc = encode(&maps->high, v.qh, v.k / 4, 64, CU_TENSOR_MAP_SWIZZLE_64B);
      break;
  }
  return rc;
}

int launch_relayout(const WeightView &v, const uint8_t *src, cudaStream_t s) {
  if (v.n == 0) return XNQ_OK;
  const int64_t nblk = v.k / block_size(v.dtype);
  switch (v.dtype) {
    case XNQ_Q4_0:
      relayout_q4_0<<<grid_for(v.n * nblk), TPB, 0, s>>>(src, const_cast<uint8_t *>(v.qs), const_cast<__half *>(v.d), v.n, nblk, v.dstride);
      break;
    case XNQ_Q8_0:
      relayout_q8_0<<<grid_for(v.n * nblk), TPB, 0, s>>>(src, const_cast<uint8_t *>(v.qs), const_cast<__half *>(v.d), v.n, nblk, v.dstride);
      break;
    case XNQ_Q6K:
      relayout_q6k<<<grid_for(v.n * nblk * 105), TPB, 0, s>>>(src, const_cast<uint8_t *>(v.qs), const_cast<uint8_t *>(v.qh),
                                                              const_cast<int8_t *>(v.sc), const_cast<__half *>(v.d), v.n, nblk, v.dstride);
      break;
    case XNQ_Q4K: repack_q4k<true><<<grid_for(v.n * nblk), TPB, 0, s>>>(src, const_cast<uint8_t *>(v.qs), v.n * nblk); break;
    default: return fail(XNQ_ERR_DTYPE, "relayout: dtype %d", v.dtype);
  }
  XNQ_CUDA(cudaGetLastError());
  count_launch();
  return XNQ_OK;
}

int launch_to_canonical(const WeightView &v, uint8_t *dst, cudaStream_t s) {
  if (v.n == 0) return XNQ_OK;
  const int64_t nblk = v.k / block_size(v.dtype);
  switch (v.dtype) {
    case XNQ_Q4_0: canonical_q4_0<<<grid_for(v.n * nblk), TPB, 0, s>>>(dst, v.qs, v.d, v.n, nblk, v.dstride); break;
    case XNQ_Q8_0: canonical_q8_0<<<grid_for(v.n * nblk), TPB, 0, s>>>(dst, v.qs, v.d, v.n, nblk, v.dstride); break;
    case XNQ_Q6K: canonical_q6k<<<grid_for(v.n * nblk * 105), TPB, 0, s>>>(dst, v.qs, v.qh, v.sc, v.d, v.n, nblk, v.dstride); break;
    case XNQ_Q4K: repack_q4k<false><<<grid_for(v.n * nblk), TPB, 0, s>>>(v.qs, dst, v.n * nblk); break;
    default: return fail(XNQ_ERR_DTYPE, "to_canonical: dtype %d", v.dtype);
  }
  XNQ_CUDA(cudaGetLastError());
  count_launch();
  return XNQ_OK;
}

int launch_dequantize(const WeightView &w, int out_dtype, void *dst, cudaStream_t s) {
  if (w.n == 0) return XNQ_OK;
  const unsigned g = grid_for(w.n * w.k);
  switch (out_dtype) {
    case XNQ_F32: dequantize_kernel<float><<<g, TPB, 0, s>>>(w, static_cast<float *>(dst)); break;
    case XNQ_F16: dequantize_kernel<__half><<<g, TPB, 0, s>>>(w, static_cast<__half *>(dst)); break;
    case XNQ_BF16: dequantize_kernel<__nv_bfloat16><<<g, TPB, 0, s>>>(w, static_cast<__nv_bfloat16 *>(dst)); break;
    default: return fail(XNQ_ERR_DTYPE, "dequantize: output dtype %d is not f32/f16/bf16", out_dtype);
  }
  XNQ_CUDA(cudaGetLastError());
  count_launch();
  return XNQ_OK;
}

int launch_max_abs(const WeightView &w, float *dev_out, cudaStream_t s) {
  XNQ_CUDA(cudaMemsetAsync(dev_out, 0, sizeof(float), s));
  if (w.n == 0) return XNQ_OK;
  const int64_t total = w.n * w.k;
  const unsigned grid = (unsigned)std::min<int64_t>((total + TPB - 1) / TPB, 148 * 16);
  max_abs_kernel<<<grid, TPB, 0, s>>>(w, reinterpret_cast<unsigned int *>(dev_out));
  XNQ_CUDA(cudaGetLastError());
  count_launch();
  return XNQ_OK;
}

template <typename T>
static int add_bias_as(void *y, int y_dtype, const void *bias, int64_t m, int64_t n, int64_t ldy, cudaStream_t s) {
  constexpr int VEC = 16 / sizeof(T);
  const bool vec = (reinterpret_cast<uintptr_t>(y) & 15) == 0 && n % VEC == 0 && ldy % VEC == 0;
  const dim3 grid(grid_for(vec ? n / VEC : n), (unsigned)std::min<int64_t>((m + BIAS_ROWS - 1) / BIAS_ROWS, 65535));
  if (vec) XNQ_CUDA(launch_pdl(add_bias_kernel<T, VEC>, grid, dim3(TPB), 0, s, static_cast<T *>(y), static_cast<const T *>(bias), m, n, ldy, y_dtype));
  else XNQ_CUDA(launch_pdl(add_bias_kernel<T, 1>, grid, dim3(TPB), 0, s, static_cast<T *>(y), static_cast<const T *>(bias), m, n, ldy, y_dtype));
  count_launch();
  return XNQ_OK;
}
int launch_add_bias(void *y, int y_dtype, const void *bias, int64_t m, int64_t n, int64_t ldy, cudaStream_t s) {
  if (m == 0 || n == 0) return XNQ_OK;
  if (y_dtype == XNQ_F32) return add_bias_as<float>(y, y_dtype, bias, m, n, ldy, s);
  if (y_dtype == XNQ_F16) return add_bias_as<__half>(y, y_dtype, bias, m, n, ldy, s);
  return add_bias_as<__nv_bfloat16>(y, y_dtype, bias, m, n, ldy, s);
}

int layout_init(int) {
  cudaFuncAttributes fa;
  XNQ_CUDA(cudaFuncGetAttributes(&fa, relayout_q4_0));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, relayout_q8_0));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, relayout_q6k));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, canonical_q4_0));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, canonical_q8_0));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, canonical_q6k));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, repack_q4k<true>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, repack_q4k<false>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, dequantize_kernel<float>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, dequantize_kernel<__half>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, dequantize_kernel<__nv_bfloat16>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, add_bias_kernel<float, 1>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, add_bias_kernel<float, 4>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, add_bias_kernel<__half, 1>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, add_bias_kernel<__half, 8>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, add_bias_kernel<__nv_bfloat16, 1>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, add_bias_kernel<__nv_bfloat16, 8>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, max_abs_kernel));
  return XNQ_OK;
}

} // namespace xnq
