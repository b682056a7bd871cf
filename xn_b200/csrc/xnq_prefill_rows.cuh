// Per-format weight producers of the prefill kernel.
//
// The weight rows of a tile are fetched and dequantized in row groups of 32 rows. A row group's bytes of one super-step (256 k,
// Q8_0: 128 k) are one slot of a shared-memory ring: ROWB bytes per row, an odd multiple of 16, so that a quarter warp's 128-bit
// reads of eight neighbouring rows fall into eight different bank groups.
//   item()   one of the ITEMS 16-byte copies that make up a row's super-step: where it comes from and how that moves with the
//            super-step. Consecutive threads take consecutive copies, so that a copy instruction of a warp touches four to six runs
//            of memory (one thread per row would touch 32).
//   head()   what the two halves of a row's 64-wide k-step share (scales, high bits)
//   half()   reads the row's bytes of half a k-step from the slot and dequantizes them to fp16: the 16 packed pairs that go to the
//            row's lane of tensor memory, where the MMA reads its weight operand.
//
// Stored k order inside a k-step (the activation image uses the same one, see kpair_shift in xnq_prefill.cu):
//   Q8_0, Q6_K  natural
//   Q4_0        chunk 4b + wi = elements [j, j+2, j+16, j+18, j+1, j+3, j+17, j+19] + 32b, j = 4wi
//   Q4_K        chunk wi      = elements [l, l+2, 32+l, 32+l+2, l+1, l+3, 32+l+1, 32+l+3], l = 4wi
#pragma once

#include "xnq_common.cuh"
#include "xnq_unpack.cuh"

namespace xnq {
namespace prefill_rows {

// bytes 0: zeros are written and nothing is read
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
// 0x6400 is 1024.0 in fp16 and its ulp is 1: OR-ing an integer 0..1023 into the low bits gives 1024 + i exactly.
__device__ __forceinline__ __half2 h2_from_bits(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }
__device__ __forceinline__ uint32_t bits_from_h2(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
// an f16 block scale times the tensor's power-of-two scale (which may itself lie outside the f16 range), as half2
__device__ __forceinline__ __half2 scaled_half2(uint32_t f16_bits, float wscale) {
  return __float2half2_rn(__half2float(__ushort_as_half((unsigned short)f16_bits)) * wscale);
}

// A copy's bytes of super-step ss are at p + ((ss * mul) & ~15); from lim on there is nothing (zeros are stored).
struct Item {
  const uint8_t *p;
  uint32_t mul, lim;
};
constexpr uint32_t NO_LIMIT = 0xffffffffu;

// KPS k-steps per super-step ss. KPS = 4: one thread converts both halves of a row's k-step kk; KPS = 2: two threads, a half each.

struct RowQ4_0 { // 128 nibble bytes | eight f16 scales
  static constexpr bool LIMITED = true; // rows may end inside a super-step
  static constexpr int KPS = 4, ROWB = 144, ITEMS = 9;
  __device__ static __forceinline__ Item item(const WeightView &w, int64_t row, int c) { // scales beyond the last block are zero
    if (c < 8) return Item{w.qs + row * (w.k / 2) + 16 * c, 128u, (uint32_t)max((int64_t)0, w.k / 2 - 16 * c)};
    return Item{reinterpret_cast<const uint8_t *>(w.d + row * w.dstride), 16u, NO_LIMIT};
  }
  struct Head {
    uint32_t dd;
    float wscale;
  };
  __device__ static __forceinline__ Head head(uint32_t slot, int, int kk, float wscale) { return Head{lds32(slot + 128 + 4 * kk), wscale}; }
  __device__ static __forceinline__ void half(const Head &hd, uint32_t slot, int kk, int hf, uint32_t (&o)[16]) { // half = one block
    const uint4 q = lds128(slot + 32 * kk + 16 * hf);
    const __half2 off = h2_from_bits(0x64086408u); // 1032 = 1024 + 8
    const __half2 d2 = scaled_half2(hf ? (hd.dd >> 16) : (hd.dd & 0xffffu), hd.wscale);
    const uint32_t wd[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int wi = 0; wi < 4; wi++)
#pragma unroll
      for (int p = 0; p < 4; p++) // nibble pairs (p, p+4) of the word
        o[4 * wi + p] = bits_from_h2(__hmul2(__hsub2(h2_from_bits(((wd[wi] >> (4 * p)) & 0x000f000fu) | 0x64006400u), off), d2));
  }
};

struct RowQ8_0 { // 128 codes | the f16 scales of this super-step and its neighbour
  static constexpr bool LIMITED = true;
  static constexpr int KPS = 2, ROWB = 144, ITEMS = 9;
  __device__ static __forceinline__ Item item(const WeightView &w, int64_t row, int c) {
    if (c < 8) return Item{w.qs + row * w.k + 16 * c, 128u, (uint32_t)max((int64_t)0, w.k - 16 * c)};
    return Item{reinterpret_cast<const uint8_t *>(w.d + row * w.dstride), 8u, NO_LIMIT};
  }
  using Head = RowQ4_0::Head;
  __device__ static __forceinline__ Head head(uint32_t slot, int ss, int kk, float wscale) { return Head{lds32(slot + 128 + 8 * (ss & 1) + 4 * kk), wscale}; }
  __device__ static __forceinline__ void half(const Head &hd, uint32_t slot, int kk, int hf, uint32_t (&o)[16]) { // half = one block
    const uint4 q[2] = {lds128(slot + 64 * kk + 32 * hf), lds128(slot + 64 * kk + 32 * hf + 16)};
    const __half2 d2 = scaled_half2(hf ? (hd.dd >> 16) : (hd.dd & 0xffffu), hd.wscale);
    const __half2 off = h2_from_bits(0x64806480u); // 1152 = 1024 + 128
#pragma unroll
    for (int c = 0; c < 4; c++) { // chunk = 8 codes
      const uint32_t ww[2] = {((c & 1) ? q[c >> 1].z : q[c >> 1].x) ^ 0x80808080u, ((c & 1) ? q[c >> 1].w : q[c >> 1].y) ^ 0x80808080u};
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const __half2 lo = h2_from_bits(__byte_perm(ww[j], 0x64646464u, 0x4140)); // bytes 0,1 -> 1024 + (b + 128)
        const __half2 hi = h2_from_bits(__byte_perm(ww[j], 0x64646464u, 0x4342)); // bytes 2,3
        o[4 * c + 2 * j] = bits_from_h2(__hmul2(__hsub2(lo, off), d2));
        o[4 * c + 2 * j + 1] = bits_from_h2(__hmul2(__hsub2(hi, off), d2));
      }
    }
  }
};

struct RowQ4K { // the 144-byte super-block: header | 128 nibble bytes
  static constexpr bool LIMITED = false;
  static constexpr int KPS = 4, ROWB = 144, ITEMS = 9;
  __device__ static __forceinline__ Item item(const WeightView &w, int64_t row, int c) { return Item{w.qs + row * (w.k / QK_K) * 144 + 16 * c, 144u, NO_LIMIT}; }
  struct Head {
    __half2 a_lo, a_hi, b_lo, b_hi;
  };
  // value = (d*sc) * code - (dmin*m): low nibbles are sub-block 2g, high nibbles sub-block 2g+1
  __device__ static __forceinline__ Head head(uint32_t slot, int, int g, float wscale) {
    const uint4 hdr = lds128(slot);
    const __half2 dm = *reinterpret_cast<const __half2 *>(&hdr.x);
    const uint32_t f = k4_field(hdr.y, hdr.z, hdr.w, g);
    const float d = __low2float(dm) * wscale, mn = __high2float(dm) * wscale;
    return Head{__float2half2_rn(d * (float)(f & 63)), __float2half2_rn(d * (float)((f >> 6) & 63)), __float2half2_rn(-mn * (float)((f >> 12) & 63)),
                __float2half2_rn(-mn * (float)(f >> 18))};
  }
  __device__ static __forceinline__ void half(const Head &hd, uint32_t slot, int g, int hf, uint32_t (&o)[16]) { // half = words 4 hf .. of the group
    const uint4 q = lds128(slot + 16 + 32 * g + 16 * hf);
    const __half2 k1024 = h2_from_bits(0x64006400u);
    const uint32_t wd[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int wi = 0; wi < 4; wi++)
#pragma unroll
      for (int p = 0; p < 4; p++) { // pairs: p=0 (l, l+2) low, p=1 (32+l, 32+l+2) high, p=2 (l+1, l+3) low, p=3 high
        const __half2 c = __hsub2(h2_from_bits(((wd[wi] >> (4 * p)) & 0x000f000fu) | 0x64006400u), k1024);
        o[4 * wi + p] = bits_from_h2((p & 1) ? __hfma2(c, hd.a_hi, hd.b_hi) : __hfma2(c, hd.a_lo, hd.b_lo));
      }
  }
};

struct RowQ6K { // 128 ql bytes | 64 qh bytes | 16 scales | the f16 d of eight super-blocks
  static constexpr bool LIMITED = false;
  static constexpr int KPS = 4, ROWB = 240, ITEMS = 14;
  __device__ static __forceinline__ Item item(const WeightView &w, int64_t row, int c) {
    const int64_t blk = row * (w.k / QK_K);
    if (c < 8) return Item{w.qs + blk * 128 + 16 * c, 128u, NO_LIMIT};
    if (c < 12) return Item{w.qh + blk * 64 + 16 * (c - 8), 64u, NO_LIMIT};
    if (c == 12) return Item{reinterpret_cast<const uint8_t *>(w.sc + blk * 16), 16u, NO_LIMIT};
    return Item{reinterpret_cast<const uint8_t *>(w.d + row * w.dstride), 2u, NO_LIMIT};
  }
  // k-step kk = 2 h + hi_pair of the super-block: group 0 takes ql[l] of half h, group 1 ql[l + 32], both the low (hi_pair 0) or high nibbles
  struct Head {
    uint4 qh[2];
    uint32_t sc4;
    float d;
  };
  __device__ static __forceinline__ Head head(uint32_t slot, int ss, int kk, float wscale) {
    const int h = kk >> 1;
    Head hd;
    hd.qh[0] = lds128(slot + 128 + 32 * h), hd.qh[1] = lds128(slot + 144 + 32 * h);
    hd.sc4 = lds32(slot + 192 + 8 * h + 4 * (kk & 1));
    const uint32_t dd = lds32(slot + 208 + 4 * ((ss >> 1) & 3));
    hd.d = __half2float(__ushort_as_half((unsigned short)((ss & 1) ? (dd >> 16) : (dd & 0xffffu)))) * wscale;
    return hd;
  }
  __device__ static __forceinline__ void half(const Head &hd, uint32_t slot, int kk, int hf, uint32_t (&o)[16]) {
    const int h = kk >> 1, sh = 4 * (kk & 1);
    const uint4 (&qh)[2] = hd.qh;
    const uint4 ql[2] = {lds128(slot + 64 * h + 32 * hf), lds128(slot + 64 * h + 32 * hf + 16)};
    const __half2 off = h2_from_bits(0x64206420u); // 1056 = 1024 + 32
    const int hsh = sh + 2 * hf; // bit position of this group's two high bits inside a qh byte
#pragma unroll
    for (int c = 0; c < 4; c++) { // chunk of 8 elements l = 8c .. 8c+7
      const uint32_t lw[2] = {(c & 1) ? ql[c >> 1].z : ql[c >> 1].x, (c & 1) ? ql[c >> 1].w : ql[c >> 1].y};
      const uint32_t hw[2] = {(c & 1) ? qh[c >> 1].z : qh[c >> 1].x, (c & 1) ? qh[c >> 1].w : qh[c >> 1].y};
      const int8_t sc = (int8_t)((hd.sc4 >> (8 * (2 * hf + (c >> 1)))) & 0xff);
      const __half2 s2 = __float2half2_rn(hd.d * (float)sc);
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const uint32_t code = ((lw[j] >> sh) & 0x0f0f0f0fu) | (((hw[j] >> hsh) << 4) & 0x30303030u);
        const __half2 lo = h2_from_bits(__byte_perm(code, 0x64646464u, 0x4140));
        const __half2 hi = h2_from_bits(__byte_perm(code, 0x64646464u, 0x4342));
        o[4 * c + 2 * j] = bits_from_h2(__hmul2(__hsub2(lo, off), s2));
        o[4 * c + 2 * j + 1] = bits_from_h2(__hmul2(__hsub2(hi, off), s2));
      }
    }
  }
};

} // namespace prefill_rows
} // namespace xnq
