// The GGML formats beyond the four of the benchmark configurations: Q4_1, Q5_0, Q5_1, Q2_K, Q3_K, Q5_K as weight
// formats and Q8_1 as an activation format (xn-core/src/quantized/k_quants.rs:100-186 block layouts, 307-610 the
// 32-element formats, 834-878 Q8_1, 880-1316 Q2_K / Q3_K, 1507-1722 Q5_K).
//
// Real GGUF files mix types, so a handle must be able to hold any of them. These formats are kept on the device exactly as in the
// file (canonical blocks, no re-layout) and served by one kernel per operation:
//   to_float   one thread per element, the reference's arithmetic operation for operation (bit-identical results);
//   matmul     activations are quantized to the block format of the weight's VecDotType (Q8_0, Q8_1 or Q8_K) as planar codes,
//              scales and sums, then one kernel unpacks the file's blocks to int8 codes in registers and multiplies them with
//              dp4a: each block's integer sums are exact, scales are applied in f32 as in the reference, and only the order in
//              which block contributions are added differs from its serial sum (within 2e-3 under its own metric).
#include <algorithm>
#include <type_traits>

#include "xnq_common.cuh"
#include "xnq_quantize_act.cuh"
#include "xnq_unpack.cuh"

namespace xnq {
namespace {

constexpr int TPB = 256;

__device__ __forceinline__ uint32_t ld16(const uint8_t *p) { return *reinterpret_cast<const uint16_t *>(p); } // blocks are 2-byte aligned
__device__ __forceinline__ uint32_t ld32(const uint8_t *p) { return ld16(p) | (ld16(p + 2) << 16); }
__device__ __forceinline__ float ldh(const uint8_t *p) { return __half2float(__ushort_as_half((unsigned short)ld16(p))); }

// 6-bit (scale, min) pair j of the 12 packed bytes of a Q4_K / Q5_K block (utils.rs:53-63)
__device__ __forceinline__ void scale_min_k4(int j, const uint8_t *q, int &sc, int &mn) {
  if (j < 4) {
    sc = q[j] & 63;
    mn = q[j + 4] & 63;
  } else {
    sc = (q[j + 4] & 0xF) | ((q[j - 4] >> 6) << 4);
    mn = (q[j + 4] >> 4) | ((q[j] >> 6) << 4);
  }
}
// the sixteen 6-bit scales of a Q3_K block (k_quants.rs:1122-1127): scale s as an unsigned byte, before the -32
__device__ __forceinline__ int q3k_scale(const uint8_t *packed, int s) {
  const uint32_t a0 = ld32(packed), a1 = ld32(packed + 4), tmp = ld32(packed + 8);
  const uint32_t kmask1 = 0x03030303u, kmask2 = 0x0f0f0f0fu;
  uint32_t w;
  switch (s >> 2) {
    case 0: w = (a0 & kmask2) | (((tmp) & kmask1) << 4); break;
    case 1: w = (a1 & kmask2) | (((tmp >> 2) & kmask1) << 4); break;
    case 2: w = ((a0 >> 4) & kmask2) | (((tmp >> 4) & kmask1) << 4); break;
    default: w = ((a1 >> 4) & kmask2) | (((tmp >> 6) & kmask1) << 4); break;
  }
  return (int)(int8_t)((w >> (8 * (s & 3))) & 0xff);
}

// ---- to_float: element j of a block, the reference's expression with every operation rounded separately --------------
__device__ __forceinline__ float deq_q4_1(const uint8_t *b, int j) { // {f16 d; f16 m; u8 qs[16]}, k_quants.rs:379-399
  const int q = j < 16 ? (b[4 + j] & 0x0F) : (b[4 + j - 16] >> 4);
  return __fadd_rn(__fmul_rn((float)q, ldh(b)), ldh(b + 2));
}
__device__ __forceinline__ int code_q5(uint32_t qh, const uint8_t *qs, int j) { // 5-bit code of element j (k_quants.rs:489-497)
  return j < 16 ? ((qs[j] & 0x0F) | (((qh >> j) << 4) & 0x10)) : ((qs[j - 16] >> 4) | ((qh >> (j - 16 + 12)) & 0x10));
}
__device__ __forceinline__ float deq_q5_0(const uint8_t *b, int j) { // {f16 d; u8 qh[4]; u8 qs[16]}, k_quants.rs:478-502
  return __fmul_rn((float)(code_q5(ld32(b + 2), b + 6, j) - 16), ldh(b));
}
__device__ __forceinline__ float deq_q5_1(const uint8_t *b, int j) { // {f16 d; f16 m; u8 qh[4]; u8 qs[16]}, k_quants.rs:586-612
  return __fadd_rn(__fmul_rn((float)code_q5(ld32(b + 4), b + 8, j), ldh(b)), ldh(b + 2));
}
__device__ __forceinline__ float deq_q2k(const uint8_t *b, int j) { // {u8 scales[16]; u8 qs[64]; f16 d; f16 dmin}, k_quants.rs:1014-1056
  const int half = j >> 7, jj = j & 127, sh = jj >> 5, l = jj & 31;
  const int sc = b[8 * half + 2 * sh + (l >> 4)];
  const float dl = __fmul_rn(ldh(b + 80), (float)(sc & 0xF)), ml = __fmul_rn(ldh(b + 82), (float)(sc >> 4));
  const int q = (b[16 + 32 * half + l] >> (2 * sh)) & 3;
  return __fsub_rn(__fmul_rn(dl, (float)q), ml);
}
__device__ __forceinline__ int code_q3k(const uint8_t *b, int j) { // signed code of element j (k_quants.rs:1290-1300)
  const int half = j >> 7, jj = j & 127, sh = jj >> 5, l = jj & 31;
  const int q = (b[32 + 32 * half + l] >> (2 * sh)) & 3;
  return q - ((b[l] & (1 << (4 * half + sh))) ? 0 : 4);
}
__device__ __forceinline__ float deq_q3k(const uint8_t *b, int j) { // {u8 hmask[32]; u8 qs[64]; u8 scales[12]; f16 d}, k_quants.rs:1260-1313
  const float dl = __fmul_rn(ldh(b + 108), __fsub_rn((float)q3k_scale(b + 96, j >> 4), 32.0f));
  return __fmul_rn(dl, (float)code_q3k(b, j));
}
__device__ __forceinline__ int code_q5k(const uint8_t *b, int j) { // 5-bit code of element j (k_quants.rs:1700-1709)
  const int c = j >> 6, jj = j & 63, l = jj & 31, hi = jj >> 5;
  const int q = hi ? (b[48 + 32 * c + l] >> 4) : (b[48 + 32 * c + l] & 0xF);
  return q + ((b[16 + l] & (1 << (2 * c + hi))) ? 16 : 0);
}
__device__ __forceinline__ float deq_q5k(const uint8_t *b, int j) { // {f16 d; f16 dmin; u8 scales[12]; u8 qh[32]; u8 qs[128]}, k_quants.rs:1684-1718
  int sc, mn;
  scale_min_k4(j >> 5, b + 4, sc, mn);
  const float d1 = __fmul_rn(ldh(b), (float)sc), m1 = __fmul_rn(ldh(b + 2), (float)mn);
  return __fsub_rn(__fmul_rn(d1, (float)code_q5k(b, j)), m1); // (ql + 16) is exact in f32, as in the reference's (ql as f32 + to_add)
}

template <typename T>
__device__ __forceinline__ T cast_to(float v);
template <>
__device__ __forceinline__ float cast_to<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half cast_to<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 cast_to<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

template <typename T>
__global__ void __launch_bounds__(TPB) generic_dequantize_kernel(int dtype, const uint8_t *blocks, int64_t total, int bs, int ts, T *out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= total) return;
  const uint8_t *b = blocks + (i / bs) * ts;
  const int j = (int)(i % bs);
  float v;
  switch (dtype) {
    case XNQ_Q4_1: v = deq_q4_1(b, j); break;
    case XNQ_Q5_0: v = deq_q5_0(b, j); break;
    case XNQ_Q5_1: v = deq_q5_1(b, j); break;
    case XNQ_Q2K: v = deq_q2k(b, j); break;
    case XNQ_Q3K: v = deq_q3k(b, j); break;
    default: v = deq_q5k(b, j); break;
  }
  out[i] = cast_to<T>(v);
}

// ---- Q8_1 activation quantizer (k_quants.rs:847-873): one thread per 32-element block -------------------------------
template <typename XT>
__global__ void __launch_bounds__(TPB) quantize_q8_1_kernel(const XT *x, int64_t m, int64_t k, int64_t ldx, uint8_t *dst) {
  const int64_t nb_row = k / 32, i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= m * nb_row) return;
  const int64_t r = i / nb_row, bi = i % nb_row;
  float v[32];
#pragma unroll
  for (int c = 0; c < 4; c++) load8(x + r * ldx + bi * 32 + 8 * c, v + 8 * c);
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 32; j++) amax = fmaxf(amax, fabsf(v[j])); // fmaxf ignores a NaN operand, as f32::max does
  const float d = __fdiv_rn(amax, 127.0f), id = d != 0.f ? __fdiv_rn(1.0f, d) : 0.f;
  const __half dh = __float2half_rn(d);
  uint8_t *b = dst + i * 36;
  int sum = 0;
#pragma unroll
  for (int j = 0; j < 32; j++) {
    const int q = round_away_sat_i8(__fmul_rn(v[j], id));
    b[4 + j] = (uint8_t)(int8_t)q;
    sum += q;
  }
  // s = f16(sum) * d as f16 values: both widened to f32, multiplied, the product rounded back to f16
  const __half sh = __float2half_rn(__fmul_rn(__half2float(__float2half_rn((float)sum)), __half2float(dh)));
  *reinterpret_cast<uint16_t *>(b) = __half_as_ushort(dh);
  *reinterpret_cast<uint16_t *>(b + 2) = __half_as_ushort(sh);
}

// ---- matmul -----------------------------------------------------------------------------------------------------------
// A lane takes one 32-element piece of a weight row (a block of the 32-element formats, an eighth of a super-block), turns it
// into eight words of int8 codes in registers, and multiplies it with up to MT activation rows by dp4a: a weight is loaded and
// unpacked once for all of a tile's rows, an activation piece is loaded (L1) once for the warp's R weight rows.
//   codes   element 4 i + b of the piece in byte b of c[i], offsets (-16, -4) already applied
//   s0, s1  integer scales of the piece's first and second 16 elements (1 where the format has none); m0, m1 the integer mins
//   d, m    the block's f16 scale and min / min scale
struct Piece {
  uint32_t c[8];
  float d, m;
  int s0, s1, m0, m1;
};

__device__ __forceinline__ uint32_t ldw(const uint8_t *p) { return __ldg(reinterpret_cast<const unsigned int *>(p)); }
__device__ __forceinline__ uint4 ldw4(const uint8_t *p) { return __ldg(reinterpret_cast<const uint4 *>(p)); }
__device__ __forceinline__ float h_lo(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xffffu))); }
__device__ __forceinline__ float h_hi(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w >> 16))); }
// bits 0..3 of b to bit 0 of bytes 0..3
__device__ __forceinline__ uint32_t spread4(uint32_t b) { return ((b & 0xfu) * 0x00204081u) & 0x01010101u; }
// bytewise x - off for bytes below 128
__device__ __forceinline__ uint32_t sub_bytes(uint32_t x, uint32_t off) { return ((x | 0x80808080u) - off) ^ 0x80808080u; }

// The words a piece is made of, as loaded (all loads of a piece are issued before any of its arithmetic). Blocks of 22 and 110
// bytes are only 2-byte aligned: the words that cover them are loaded aligned (each holds at least one of the block's bytes, so
// none lies outside the allocation, whose size is a multiple of 256) and shifted into place.
template <int DT>
struct Raw;
template <>
struct Raw<XNQ_Q4_1> { // {f16 d; f16 m; u8 qs[16]}
  uint32_t w[5];
  __device__ __forceinline__ void load(const uint8_t *row, int j) {
#pragma unroll
    for (int i = 0; i < 5; i++) w[i] = ldw(row + (int64_t)j * 20 + 4 * i);
  }
  __device__ __forceinline__ void unpack(int, Piece &p) const {
    p.d = h_lo(w[0]), p.m = h_hi(w[0]);
#pragma unroll
    for (int i = 0; i < 4; i++) p.c[i] = w[1 + i] & 0x0f0f0f0fu, p.c[4 + i] = (w[1 + i] >> 4) & 0x0f0f0f0fu;
  }
};
template <>
struct Raw<XNQ_Q5_0> { // {f16 d; u8 qh[4]; u8 qs[16]}, 22 bytes
  uint32_t w[6];
  int sh;
  __device__ __forceinline__ void load(const uint8_t *row, int j) {
    const uint8_t *b = row + (int64_t)j * 22;
    const int off = (int)(reinterpret_cast<uintptr_t>(b) & 2);
    sh = 8 * off;
#pragma unroll
    for (int i = 0; i < 6; i++) w[i] = ldw(b - off + 4 * i);
  }
  __device__ __forceinline__ void unpack(int, Piece &p) const {
    uint32_t v[6];
#pragma unroll
    for (int i = 0; i < 6; i++) v[i] = __funnelshift_r(w[i], i < 5 ? w[i + 1] : 0u, sh);
    p.d = h_lo(v[0]), p.m = 0.f;
    const uint32_t qh = __funnelshift_r(v[0], v[1], 16);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t q = __funnelshift_r(v[1 + i], v[2 + i], 16);
      p.c[i] = sub_bytes((q & 0x0f0f0f0fu) | (spread4(qh >> (4 * i)) << 4), 0x10101010u);
      p.c[4 + i] = sub_bytes(((q >> 4) & 0x0f0f0f0fu) | (spread4(qh >> (16 + 4 * i)) << 4), 0x10101010u);
    }
  }
};
template <>
struct Raw<XNQ_Q5_1> { // {f16 d; f16 m; u8 qh[4]; u8 qs[16]}
  uint32_t w[6];
  __device__ __forceinline__ void load(const uint8_t *row, int j) {
#pragma unroll
    for (int i = 0; i < 6; i++) w[i] = ldw(row + (int64_t)j * 24 + 4 * i);
  }
  __device__ __forceinline__ void unpack(int, Piece &p) const {
    p.d = h_lo(w[0]), p.m = h_hi(w[0]);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      p.c[i] = (w[2 + i] & 0x0f0f0f0fu) | (spread4(w[1] >> (4 * i)) << 4);
      p.c[4 + i] = ((w[2 + i] >> 4) & 0x0f0f0f0fu) | (spread4(w[1] >> (16 + 4 * i)) << 4);
    }
  }
};
template <>
struct Raw<XNQ_Q2K> { // {u8 scales[16]; u8 qs[64]; f16 d; f16 dmin}, 84 bytes; piece s: bit pair s % 4 of half s / 4
  uint32_t q[8], sc, dm;
  __device__ __forceinline__ void load(const uint8_t *row, int j) {
    const uint8_t *b = row + (int64_t)(j >> 3) * 84;
    const int s = j & 7;
#pragma unroll
    for (int i = 0; i < 8; i++) q[i] = ldw(b + 16 + 32 * (s >> 2) + 4 * i);
    sc = ldw(b + 4 * (s >> 1));
    dm = ldw(b + 80);
  }
  __device__ __forceinline__ void unpack(int s, Piece &p) const {
    const uint32_t b2 = sc >> (16 * (s & 1));
    p.d = h_lo(dm), p.m = h_hi(dm);
    p.s0 = b2 & 15, p.m0 = (b2 >> 4) & 15, p.s1 = (b2 >> 8) & 15, p.m1 = (b2 >> 12) & 15;
#pragma unroll
    for (int i = 0; i < 8; i++) p.c[i] = (q[i] >> (2 * (s & 3))) & 0x03030303u;
  }
};
template <>
struct Raw<XNQ_Q3K> { // {u8 hmask[32]; u8 qs[64]; u8 scales[12]; f16 d}, 110 bytes
  uint32_t hm[9], q[9], sc[4];
  int sh;
  __device__ __forceinline__ void load(const uint8_t *row, int j) {
    const uint8_t *b = row + (int64_t)(j >> 3) * 110;
    const int s = j & 7, off = (int)(reinterpret_cast<uintptr_t>(b) & 2);
    sh = 8 * off;
    b -= off;
#pragma unroll
    for (int i = 0; i < 9; i++) hm[i] = ldw(b + 4 * i), q[i] = ldw(b + 32 + 32 * (s >> 2) + 4 * i);
#pragma unroll
    for (int i = 0; i < 4; i++) sc[i] = ldw(b + 96 + 4 * i);
  }
  __device__ __forceinline__ void unpack(int s, Piece &p) const {
    const uint32_t a0 = __funnelshift_r(sc[0], sc[1], sh), a1 = __funnelshift_r(sc[1], sc[2], sh), tmp = __funnelshift_r(sc[2], sc[3], sh);
    p.d = h_lo(sc[3] >> sh), p.m = 0.f;
    const int g = s >> 1; // the word of four scales (k_quants.rs:1122-1127), of which this piece takes two
    const uint32_t w4 = ((((g & 1) ? a1 : a0) >> (4 * (g >> 1))) & 0x0f0f0f0fu) | (((tmp >> (2 * g)) & 0x03030303u) << 4);
    const uint32_t b2 = w4 >> (16 * (s & 1));
    p.s0 = (int)(b2 & 0xffu) - 32, p.s1 = (int)((b2 >> 8) & 0xffu) - 32;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t lo = (__funnelshift_r(q[i], q[i + 1], sh) >> (2 * (s & 3))) & 0x03030303u;
      const uint32_t hi = (__funnelshift_r(hm[i], hm[i + 1], sh) >> s) & 0x01010101u;
      p.c[i] = sub_bytes(lo | (hi << 2), 0x04040404u);
    }
  }
};
template <>
struct Raw<XNQ_Q5K> { // {f16 d; f16 dmin; u8 scales[12]; u8 qh[32]; u8 qs[128]}, 176 = 11 x 16 bytes
  uint4 hdr, h[2], q[2];
  __device__ __forceinline__ void load(const uint8_t *row, int j) {
    const uint8_t *b = row + (int64_t)(j >> 3) * 176;
    const int s = j & 7;
    hdr = ldw4(b);
    h[0] = ldw4(b + 16), h[1] = ldw4(b + 32);
    q[0] = ldw4(b + 48 + 32 * (s >> 1)), q[1] = ldw4(b + 64 + 32 * (s >> 1));
  }
  __device__ __forceinline__ void unpack(int s, Piece &p) const {
    const K4Scales ks = unpack_k4(hdr.y, hdr.z, hdr.w);
    p.d = h_lo(hdr.x), p.m = h_hi(hdr.x);
    p.s0 = (int)k4_byte(ks.sc_lo, ks.sc_hi, s), p.m0 = (int)k4_byte(ks.mn_lo, ks.mn_hi, s);
    const uint32_t hw[8] = {h[0].x, h[0].y, h[0].z, h[0].w, h[1].x, h[1].y, h[1].z, h[1].w};
    const uint32_t qw[8] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w};
#pragma unroll
    for (int i = 0; i < 8; i++) p.c[i] = ((qw[i] >> (4 * (s & 1))) & 0x0f0f0f0fu) | (((hw[i] >> s) & 0x01010101u) << 4);
  }
};

// What one piece adds to the dot of a (weight row, activation row) pair: exact integer sums, scaled in f32 as the reference does
// (k_quants.rs:328-339 Q4_1, 423-436 Q5_0, 529-541 Q5_1, 904-945 Q2_K, 1087-1176 Q3_K, 1540-1604 Q5_K). lo, hi: the row's 32 codes;
// da: its block scale; b0, b1: the sums of its first and second 16 codes; as: its block's s (Q4_1, Q5_1).
template <int DT>
__device__ __forceinline__ float piece_dot(const Piece &p, const uint4 &lo, const uint4 &hi, float da, float as, int b0, int b1, float acc) {
  int t0 = __dp4a((int)p.c[0], (int)lo.x, 0);
  t0 = __dp4a((int)p.c[1], (int)lo.y, t0);
  t0 = __dp4a((int)p.c[2], (int)lo.z, t0);
  t0 = __dp4a((int)p.c[3], (int)lo.w, t0);
  int t1 = __dp4a((int)p.c[4], (int)hi.x, (DT == XNQ_Q2K || DT == XNQ_Q3K) ? 0 : t0);
  t1 = __dp4a((int)p.c[5], (int)hi.y, t1);
  t1 = __dp4a((int)p.c[6], (int)hi.z, t1);
  t1 = __dp4a((int)p.c[7], (int)hi.w, t1);
  if (DT == XNQ_Q4_1 || DT == XNQ_Q5_1) return acc + __fadd_rn(__fmul_rn(__fmul_rn((float)t1, p.d), da), __fmul_rn(p.m, as));
  if (DT == XNQ_Q5_0) return acc + __fmul_rn(__fmul_rn((float)t1, p.d), da);
  if (DT == XNQ_Q2K) return acc + __fsub_rn(__fmul_rn(__fmul_rn(da, p.d), (float)(p.s0 * t0 + p.s1 * t1)), __fmul_rn(__fmul_rn(da, p.m), (float)(p.m0 * b0 + p.m1 * b1)));
  if (DT == XNQ_Q3K) return acc + __fmul_rn(__fmul_rn(p.d, da), (float)(p.s0 * t0 + p.s1 * t1));
  return acc + __fsub_rn(__fmul_rn(__fmul_rn(p.d, da), (float)(p.s0 * t1)), __fmul_rn(__fmul_rn(p.m, da), (float)(p.m0 * (b0 + b1))));
}

// What bounds it: at a few rows the loads a warp keeps in flight against DRAM latency, at many the dp4a rate. A warp owns GR
// weight rows and every (32 KS)-th group of pieces; KS warps share the rows of a longer k (their sums meet in shared memory), so
// that a few thousand rows give every SM enough warps. The order of the sum over k depends on k alone: a row's result is the
// same bits in a batch, alone or in a shard. The weights of the first pieces are requested before the wait for the kernel that
// quantizes the activations. Measured, Q5_K 4096 x 4096, 7 rows: 381 us a call with one lane per super-block reading single bytes (each
// code extracted and multiplied by itself, one activation row after the other), 16 us like this, most of it the host's share of the call.
// Q2_K's lanes are added in f64: the CPU code adds one f32 term per super-block, here eight lanes have one each, and five levels of f32
// additions on top made the result up to 22 % less exact (1024 values: 7.7e-8 from the exact dot, the CPU code's order 6.3e-8).
constexpr int GR = 2;
template <int DT>
struct LaneSum { using T = float; };
template <>
struct LaneSum<XNQ_Q2K> { using T = double; };
__host__ __device__ constexpr int k_splits(int pieces) { return pieces < 64 ? 1 : (pieces < 128 ? 2 : 4); }

// Eight rows: the device's CTAs may walk all groups of weight rows, and the first pieces of a CTA's next group are requested while it multiplies
// the last ones of this (Q5_K 4096 x 4096, 7 rows 16.5 -> 13.9 us; Q4_1 3840 x 576, 62 rows 23.2 -> 17.7). With fewer rows more CTAs in flight do
// better (Q5_1 26309 x 2752, one row: 21.5 us, walking 31.8), and with Q3_K's 22 words a piece (20256 x 2304, 6 rows: 41.8, walking 43.5): a
// CTA has one group. So it has where one tile of activation rows meets weight rows of 32-value blocks whose pieces take a warp three turns or more (Q5_1 6582 x
// 10496, 8 rows: 40.8, walking 43.9; Q4_1 4096 x 14336, 6 rows: 30.2, walking 32.6; two turns, Q5_0 2048 x 8192, 6 rows: 13.2, walking 12.3; Q5_K
// 6582 x 10496, 8 rows: 58.3, walking 51.3), and where each has one anyway. Q5_1's one tile walks only over two rounds of groups or more (8192 x 1024, 8
// rows: walking 1.08 times as long; 4096 x 4096: 0.93), and not where the lanes of a warp part in its last turn (17980 x 2816, 6 rows: 30.6, walking 32.6).
__host__ __device__ constexpr bool walks(int dt, int mt) { return mt >= 8 && dt != XNQ_Q3K; }
__host__ __device__ constexpr bool blocks_of_32(int dt) { return dt == XNQ_Q4_1 || dt == XNQ_Q5_0 || dt == XNQ_Q5_1; }

// BIAS: a variant of its own, as in the dp4a kernels. With a test of the pointer beside the store, calls without a bias took, one row, Q5_K 14336 x 4096
// 26.8 us instead of 26.6, Q3_K 4096 x 4096 8.17 instead of 8.06, and four rows of Q4_1 14336 x 4096 27.3 instead of 26.9.
template <int DT, int MT, bool BIAS, bool WALK>
__global__ void __launch_bounds__(TPB, 2) generic_matmul_kernel(const uint8_t *__restrict__ w, ActView act, int64_t n, int64_t row_bytes, void *y, int y_dtype,
                                                             int64_t ldy, const void *__restrict__ bias, int64_t groups) {
  constexpr int NV = GR * MT;
  constexpr bool K256 = DT == XNQ_Q2K || DT == XNQ_Q3K || DT == XNQ_Q5K;
  using Sum = typename LaneSum<DT>::T;
  __shared__ Sum red[WALK ? 2 : 1][TPB / 32][NV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pieces = (int)(act.k / 32), ks_n = k_splits(pieces);
  const int ks = warp & (ks_n - 1), grp = warp / ks_n;
  const int64_t m0 = (int64_t)blockIdx.y * MT;
  const int rows = (int)min((int64_t)MT, act.m - m0);
  const int s = lane & 7;
  const uint8_t *wr[GR]; // the warp's rows of a group; past the last row: a duplicate, never stored
  auto bind = [&](int64_t group) {
    const int64_t row0 = (group * (TPB / 32 / ks_n) + grp) * GR;
#pragma unroll
    for (int r = 0; r < GR; r++) wr[r] = w + min(row0 + r, n - 1) * row_bytes;
  };
  bind(blockIdx.x);
  Raw<DT> raw[GR];
  const int j0 = ks * 32 + lane;
  if (j0 < pieces) {
#pragma unroll
    for (int r = 0; r < GR; r++) raw[r].load(wr[r], j0);
  }
  pdl_wait();
  const int nblk_a = K256 ? pieces >> 3 : pieces;
  const int8_t *aq = act.q + m0 * act.k;
  const float *ad = act.d + m0 * nblk_a;              // K256
  const int16_t *ab = act.bsum + m0 * (act.k / 16);   // K256
  const __half *hd = reinterpret_cast<const __half *>(act.d) + m0 * nblk_a, *hs = reinterpret_cast<const __half *>(act.bsum) + m0 * nblk_a; // the others
  int turn = 0;
  int64_t group = blockIdx.x;
  do {
  const int64_t row0 = (group * (TPB / 32 / ks_n) + grp) * GR;
  float acc[NV];
#pragma unroll
  for (int i = 0; i < NV; i++) acc[i] = 0.f;
  for (int j = j0; j < pieces;) {
    Piece p[GR];
#pragma unroll
    for (int r = 0; r < GR; r++) raw[r].unpack(s, p[r]);
    // the next pieces, of these rows or of the CTA's next ones, are on their way while these are multiplied
    const int jn = j + 32 * ks_n;
    if (jn < pieces) {
#pragma unroll
      for (int r = 0; r < GR; r++) raw[r].load(wr[r], jn);
    } else if (WALK && group + gridDim.x < groups) {
      bind(group + gridDim.x);
#pragma unroll
      for (int r = 0; r < GR; r++) raw[r].load(wr[r], j0);
    }
#pragma unroll
    for (int i = 0; i < MT; i++) {
      if (i < rows) {
        const uint4 *a = reinterpret_cast<const uint4 *>(aq + (int64_t)i * act.k + (int64_t)j * 32);
        const uint4 lo = a[0], hi = a[1];
        const int64_t blk = (int64_t)i * nblk_a + (K256 ? j >> 3 : j);
        const float da = K256 ? ad[blk] : __half2float(hd[blk]);
        const float as = DT == XNQ_Q4_1 || DT == XNQ_Q5_1 ? __half2float(hs[blk]) : 0.f;
        int b0 = 0, b1 = 0;
        if (DT == XNQ_Q2K || DT == XNQ_Q5K) {
          const uint32_t b = *reinterpret_cast<const uint32_t *>(ab + (int64_t)i * (act.k / 16) + 2 * (int64_t)j);
          b0 = (int)(int16_t)(b & 0xffffu), b1 = (int)(int16_t)(b >> 16);
        }
#pragma unroll
        for (int r = 0; r < GR; r++) acc[i * GR + r] = piece_dot<DT>(p[r], lo, hi, da, as, b0, b1, acc[i * GR + r]);
      }
    }
    j = jn;
  }
  // sums over the lanes: as long as a thread holds more than one value, each step hands half of them to the partner lane, so NV
  // values cost NV - 1 exchanges and end up in different lanes (value v in the lanes whose upper bits are v); the additions are
  // those of the plain xor tree
  Sum tot[NV];
#pragma unroll
  for (int i = 0; i < NV; i++) tot[i] = acc[i];
  int nv = NV, off = 16;
#pragma unroll
  for (int step = 0; step < 5; step++) {
    if (nv > 1) {
      nv >>= 1;
#pragma unroll
      for (int v = 0; v < NV / 2; v++) {
        if (v < nv) {
          const bool up = (lane & off) != 0;
          const Sum keep = up ? tot[v + nv] : tot[v], give = up ? tot[v] : tot[v + nv];
          tot[v] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
      }
    } else {
      tot[0] += __shfl_xor_sync(0xffffffffu, tot[0], off);
    }
    off >>= 1;
  }
  constexpr int PER = 32 / NV; // lanes that hold the same value
  const int v = lane / PER;
  if (ks_n > 1) { // (two buffers: a warp may be a group ahead of the one that adds)
    if (lane % PER == 0) red[turn][warp][v] = tot[0];
    __syncthreads();
    if (ks > 0) continue;
    for (int i = 1; i < ks_n; i++) tot[0] += red[turn][warp + i][v];
  }
  const int i = v / GR;
  const int64_t row = row0 + v % GR;
  if (lane % PER == 0 && i < rows && row < n) {
    const int64_t idx = (m0 + i) * ldy + row;
    float sum = (float)tot[0];
    if (BIAS) sum = with_bias(sum, bias_at(bias, y_dtype, row), y_dtype);
    if (y_dtype == XNQ_F32) static_cast<float *>(y)[idx] = sum;
    else if (y_dtype == XNQ_F16) static_cast<__half *>(y)[idx] = __float2half_rn(sum);
    else static_cast<__nv_bfloat16 *>(y)[idx] = __float2bfloat16_rn(sum);
  }
  } while (WALK && (turn ^= 1, (group += gridDim.x) < groups));
}

int g_sms = 148;

// CTAs that share a tile of activation rows and walk its groups of weight rows. Two fit an SM, and one that has an SM to itself runs 1.6 times as fast as one
// of two, so that a last round of up to a CTA per SM counts 0.62 of one; a CTA's start and end cost as much as 3/4 of a group. Of the numbers that
// just fill 1 to 16 rounds the best is taken. (As many as fill one round, rounded down, left up to half of the places empty, and one tile too many
// cost a second walk over the weight: Q4_1 4096 x 4096, 1200 rows 2350 us, now 1186; 2376 rows 3779, now 2339; Q5_K 512 x 512, 1200 rows 89.8, now 56.8.)
int64_t walk_parts(int64_t groups, int64_t tiles) {
  const int64_t places = 2 * g_sms, first = (tiles + places - 1) / places;
  int64_t best = 1;
  double least = 0;
  for (int64_t rounds = first; rounds < first + 16; rounds++) {
    const int64_t parts = std::min(groups, rounds * places / tiles), ctas = parts * tiles, left = ctas % places;
    const double time = ((double)(ctas / places) + (left == 0 ? 0. : left <= places / 2 ? 0.62 : 1.)) * ((double)((groups + parts - 1) / parts) + 0.75);
    if (rounds == first || time < least) least = time, best = parts;
    if (parts == groups) break;
  }
  return best;
}

template <int DT>
int launch_matmul_dt(const WeightView &w, const ActView &act, int64_t row_bytes, void *y, int y_dtype, int64_t ldy, cudaStream_t s, const void *bias) {
  const int rows_per_cta = TPB / 32 / k_splits((int)(w.k / 32)) * GR;
  const int64_t groups = (w.n + rows_per_cta - 1) / rows_per_cta;
  // Activation rows a warp takes at a time: eight, as far as that leaves the device enough CTAs (Q5_K 384 x 1536, 38 rows: 10.1 us with eight,
  // 6.4 with four; Q5_1 384 x 512, 10 rows: 5.9, 4.1, 3.3 and 2.9 with eight to one): one to an SM, and a third more for eight and where the last of
  // several tiles has fewer rows, whose CTAs are done sooner (779 x 8192, Q3_K, 3 rows: four at a time 5.8, two 7.6; 359 x 8192, Q4_1, 6 rows: two 1.3
  // times as fast as four). Q2_K's lanes' sums are f64: four where the CTAs would not fill
  // one and a half rounds with eight (476 x 8448, 20 rows: 15.5, with eight 16.9) and for several tiles against weight rows of three turns (4096 x
  // 14336, 20 rows: 103 and 135), else eight (4096 x 4096, 7 rows: 13.5, with four 18.0; 1200 rows: 1538 and 2308; 1280 x 6656, 39 rows: 35.2 and 48.9).
  // Sixteen, with spilled registers, were slower everywhere (Q5_K 384 x 1536: 25; Q4_1 3840 x 576, 62 rows: 32.3, eight 23.2).
  const int pieces = (int)(w.k / 32), turns = (pieces + 32 * k_splits(pieces) - 1) / (32 * k_splits(pieces)); // of a warp along k
  const bool eight = DT != XNQ_Q2K || (groups * ((act.m + 7) / 8) >= 3 * g_sms && (turns < 3 || act.m <= 8));
  int mt = act.m >= 5 && eight ? 8 : (act.m >= 3 ? 4 : (int)act.m);
  for (int64_t tiles = 0; mt > 1; mt /= 2) {
    tiles = (act.m + mt - 1) / mt;
    if (groups * tiles >= (mt == 8 || (tiles > 1 && act.m % mt) ? 4 * g_sms / 3 : g_sms)) break;
  }
  const bool k256 = act.act_dtype == XNQ_Q8K;
  const int64_t pass = (int64_t)mt * 65535; // grid.y is limited to 65535 tiles of activation rows
  for (int64_t r0 = 0; r0 < act.m; r0 += pass) {
    ActView a = act;
    a.m = std::min(act.m - r0, pass);
    a.q += r0 * w.k;
    a.d = reinterpret_cast<float *>(reinterpret_cast<char *>(act.d) + r0 * (k256 ? w.k / QK_K * 4 : w.k / QK * 2));
    if (act.bsum) a.bsum += r0 * (k256 ? w.k / 16 : w.k / QK);
    void *yp = static_cast<char *>(y) + (size_t)r0 * ldy * type_size(y_dtype);
    const int64_t tiles = (a.m + mt - 1) / mt;
    const bool plain = !walks(DT, mt) || (blocks_of_32(DT) && tiles == 1 &&
                                          (turns >= 3 || (DT == XNQ_Q5_1 && (groups < 4 * g_sms || (turns == 2 && pieces % 32 != 0)))));
    const int64_t parts = plain ? groups : walk_parts(groups, tiles);
    const dim3 grid((unsigned)parts, (unsigned)tiles);
    const auto launch = [&](auto rows_t, auto bias_t, auto walk_t) {
      return launch_pdl(generic_matmul_kernel<DT, decltype(rows_t)::value, decltype(bias_t)::value, decltype(walk_t)::value>, grid, dim3(TPB), 0, s, w.qs, a, w.n, row_bytes,
                        yp, y_dtype, ldy, bias, groups);
    };
    const auto launch_rows = [&](auto rows_t) {
      if constexpr (walks(DT, decltype(rows_t)::value))
        if (!blocks_of_32(DT) || parts < groups) return bias ? launch(rows_t, std::true_type{}, std::true_type{}) : launch(rows_t, std::false_type{}, std::true_type{});
      if constexpr (!walks(DT, decltype(rows_t)::value) || blocks_of_32(DT))
        return bias ? launch(rows_t, std::true_type{}, std::false_type{}) : launch(rows_t, std::false_type{}, std::false_type{});
    };
    cudaError_t e;
    switch (mt) {
      case 1: e = launch_rows(std::integral_constant<int, 1>{}); break;
      case 2: e = launch_rows(std::integral_constant<int, 2>{}); break;
      case 4: e = launch_rows(std::integral_constant<int, 4>{}); break;
      default: e = launch_rows(std::integral_constant<int, 8>{}); break;
    }
    XNQ_CUDA(e);
    count_launch();
  }
  return XNQ_OK;
}
template <int DT, int MT>
int init_matmul_rows() { // kernels are loaded before any stream capture
  cudaFuncAttributes fa;
  if constexpr (walks(DT, MT)) {
    XNQ_CUDA(cudaFuncGetAttributes(&fa, generic_matmul_kernel<DT, MT, false, true>));
    XNQ_CUDA(cudaFuncGetAttributes(&fa, generic_matmul_kernel<DT, MT, true, true>));
  }
  if constexpr (!walks(DT, MT) || blocks_of_32(DT)) {
    XNQ_CUDA(cudaFuncGetAttributes(&fa, generic_matmul_kernel<DT, MT, false, false>));
    XNQ_CUDA(cudaFuncGetAttributes(&fa, generic_matmul_kernel<DT, MT, true, false>));
  }
  return XNQ_OK;
}
template <int DT>
int init_matmul_dt() {
  int rc;
  if ((rc = init_matmul_rows<DT, 1>()) != XNQ_OK || (rc = init_matmul_rows<DT, 2>()) != XNQ_OK || (rc = init_matmul_rows<DT, 4>()) != XNQ_OK) return rc;
  return init_matmul_rows<DT, 8>();
}

inline unsigned grid_for(int64_t work, int per) { return (unsigned)((work + per - 1) / per); }

} // namespace

bool is_generic_dtype(int dt) { return dt == XNQ_Q4_1 || dt == XNQ_Q5_0 || dt == XNQ_Q5_1 || dt == XNQ_Q2K || dt == XNQ_Q3K || dt == XNQ_Q5K; }

int launch_generic_dequantize(const WeightView &w, int out_dtype, void *dst, cudaStream_t s) {
  if (w.n == 0) return XNQ_OK;
  const int64_t total = w.n * w.k;
  const int bs = block_size(w.dtype), ts = type_size(w.dtype);
  const unsigned g = grid_for(total, TPB);
  switch (out_dtype) {
    case XNQ_F32: generic_dequantize_kernel<float><<<g, TPB, 0, s>>>(w.dtype, w.qs, total, bs, ts, static_cast<float *>(dst)); break;
    case XNQ_F16: generic_dequantize_kernel<__half><<<g, TPB, 0, s>>>(w.dtype, w.qs, total, bs, ts, static_cast<__half *>(dst)); break;
    case XNQ_BF16: generic_dequantize_kernel<__nv_bfloat16><<<g, TPB, 0, s>>>(w.dtype, w.qs, total, bs, ts, static_cast<__nv_bfloat16 *>(dst)); break;
    default: return fail(XNQ_ERR_DTYPE, "dequantize: output dtype %d is not f32/f16/bf16", out_dtype);
  }
  XNQ_CUDA(cudaGetLastError());
  count_launch();
  return XNQ_OK;
}

int launch_quantize_q8_1(const void *x, int x_dtype, int64_t m, int64_t k, int64_t ldx, void *dst, cudaStream_t s) {
  if (m == 0) return XNQ_OK;
  const unsigned g = grid_for(m * (k / 32), TPB);
  uint8_t *d = static_cast<uint8_t *>(dst);
  switch (x_dtype) {
    case XNQ_F32: quantize_q8_1_kernel<float><<<g, TPB, 0, s>>>(static_cast<const float *>(x), m, k, ldx, d); break;
    case XNQ_F16: quantize_q8_1_kernel<__half><<<g, TPB, 0, s>>>(static_cast<const __half *>(x), m, k, ldx, d); break;
    case XNQ_BF16: quantize_q8_1_kernel<__nv_bfloat16><<<g, TPB, 0, s>>>(static_cast<const __nv_bfloat16 *>(x), m, k, ldx, d); break;
    default: return fail(XNQ_ERR_DTYPE, "quantize_act: activation dtype %d", x_dtype);
  }
  XNQ_CUDA(cudaGetLastError());
  count_launch();
  return XNQ_OK;
}

// The activations' planar image, no larger than the canonical blocks: Q8_K codes, f32 scales and 16-sums; Q8_0 / Q8_1 codes and f16 scales,
// and for Q8_1 the f16 s of every block.
static ActView generic_acts(const WeightView &w, void *ws, int64_t m) {
  const int adt = act_dtype_for(w.dtype);
  ActView a;
  a.act_dtype = adt, a.m = m, a.k = w.k;
  char *p = static_cast<char *>(ws);
  a.q = reinterpret_cast<int8_t *>(p);
  a.d = reinterpret_cast<float *>(p += m * w.k);
  p += m * (adt == XNQ_Q8K ? w.k / QK_K * 4 : w.k / QK * 2);
  a.bsum = adt == XNQ_Q8_0 ? nullptr : reinterpret_cast<int16_t *>(p);
  return a;
}
size_t generic_workspace_bytes(const WeightView &w, int64_t m) {
  const int adt = act_dtype_for(w.dtype);
  return ((size_t)m * (size_t)(w.k / block_size(adt)) * (size_t)type_size(adt) + 255) & ~(size_t)255;
}

// y[m, n] = x[m, k] . W^T for a weight held as canonical blocks; workspace: generic_workspace_bytes(w, m)
int launch_generic_matmul(const WeightView &w, const void *x, int x_dtype, int64_t m, int64_t ldx, void *y, int y_dtype, int64_t ldy, void *workspace,
                          cudaStream_t s, const void *bias) {
  // the reference's dots of the 32-element formats refuse an odd number of blocks (k_quants.rs:322-325, 413-415, 523-526)
  if (block_size(w.dtype) == 32 && (w.k / 32) % 2) return fail(XNQ_ERR_SHAPE, "matmul_t: k = %lld is not divisible by 64 (an even number of 32-value blocks)", (long long)w.k);
  const ActView act = generic_acts(w, workspace, m);
  int rc = act.act_dtype == XNQ_Q8K ? launch_quantize_act_planar(act, x, x_dtype, ldx, s) : launch_quantize_act_f16_scales(act, x, x_dtype, ldx, s);
  if (rc != XNQ_OK) return rc;
  const int64_t row_bytes = w.k / block_size(w.dtype) * type_size(w.dtype);
  profile_mark(s, true);
  switch (w.dtype) {
    case XNQ_Q4_1: rc = launch_matmul_dt<XNQ_Q4_1>(w, act, row_bytes, y, y_dtype, ldy, s, bias); break;
    case XNQ_Q5_0: rc = launch_matmul_dt<XNQ_Q5_0>(w, act, row_bytes, y, y_dtype, ldy, s, bias); break;
    case XNQ_Q5_1: rc = launch_matmul_dt<XNQ_Q5_1>(w, act, row_bytes, y, y_dtype, ldy, s, bias); break;
    case XNQ_Q2K: rc = launch_matmul_dt<XNQ_Q2K>(w, act, row_bytes, y, y_dtype, ldy, s, bias); break;
    case XNQ_Q3K: rc = launch_matmul_dt<XNQ_Q3K>(w, act, row_bytes, y, y_dtype, ldy, s, bias); break;
    case XNQ_Q5K: rc = launch_matmul_dt<XNQ_Q5K>(w, act, row_bytes, y, y_dtype, ldy, s, bias); break;
    default: rc = fail(XNQ_ERR_DTYPE, "matmul_t: dtype %d", w.dtype);
  }
  profile_mark(s, false);
  return rc;
}

int generic_init(int device) { // kernels are loaded before any stream capture
  XNQ_CUDA(cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, device));
  cudaFuncAttributes fa;
  XNQ_CUDA(cudaFuncGetAttributes(&fa, generic_dequantize_kernel<float>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, generic_dequantize_kernel<__half>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, generic_dequantize_kernel<__nv_bfloat16>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, quantize_q8_1_kernel<float>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, quantize_q8_1_kernel<__half>));
  XNQ_CUDA(cudaFuncGetAttributes(&fa, quantize_q8_1_kernel<__nv_bfloat16>));
  int rc;
  if ((rc = init_matmul_dt<XNQ_Q4_1>()) != XNQ_OK) return rc;
  if ((rc = init_matmul_dt<XNQ_Q5_0>()) != XNQ_OK) return rc;
  if ((rc = init_matmul_dt<XNQ_Q5_1>()) != XNQ_OK) return rc;
  if ((rc = init_matmul_dt<XNQ_Q2K>()) != XNQ_OK) return rc;
  if ((rc = init_matmul_dt<XNQ_Q3K>()) != XNQ_OK) return rc;
  return init_matmul_dt<XNQ_Q5K>();
}

} // namespace xnq
