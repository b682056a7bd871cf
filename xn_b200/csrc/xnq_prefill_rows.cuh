// Per-format weight producers of the prefill kernel.
//
// The weight rows of a tile are fetched one super-step (256 k, Q8_0: 128 k) at a time into a slot of a shared-memory ring: the boxes of the weight's
// tensor maps (xnq_common.cuh), as they lay the rows out, and behind them 16 bytes of scale data per row where the format keeps its scales
// apart.
//   boxes()  requests the boxes of super-step ss of the tile that starts at a row
//   scales() where the 16 bytes of scale data of a row and super-step lie (piece 0 .. SCALES - 1)
//   head()   what the two halves of a row's 64-wide k-step share (scales, high bits)
//   half()   reads the bytes of half a k-step of row r from the slot and dequantizes them to fp16: the 16 packed pairs that go to the
//            row's lane of tensor memory, where the MMA reads its weight operand. Lanes are rows: the swizzles and the 144-byte rows spread a
//            quarter warp's 128-bit reads over all bank groups.
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

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
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

// a box of a tensor map: x in bytes (a multiple of 16), y the first row
__device__ __forceinline__ void tma_box(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
constexpr uint32_t ROWS = 128; // of a tile
__device__ __forceinline__ uint4 chunk128(uint32_t at, int r, int c) { return lds128(at + (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4))); }
__device__ __forceinline__ uint4 chunk64(uint32_t at, int r, int c) { return lds128(at + (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4))); }

// KPS k-steps per super-step ss. KPS = 4: one thread converts both halves of a row's k-step kk; KPS = 2: two threads, a half each.

struct RowQ4_0 { // 128 nibble bytes per row, then eight f16 scales
  static constexpr int KPS = 4, SCALES = 1;
  static constexpr uint32_t BOX = ROWS * 128, SLOT = BOX + ROWS * 16;
  __device__ static __forceinline__ void boxes(uint32_t slot, const CUtensorMap *codes, const CUtensorMap *, int ss, int row, uint32_t bar) { tma_box(slot, codes, ss * 128, row, bar); }
  __device__ static __forceinline__ const void *scales(const WeightView &w, int64_t row, int ss, int) { // (beyond the last block they are zero)
    return reinterpret_cast<const uint8_t *>(w.d + row * w.dstride) + ss * 16;
  }
  struct Head {
    uint32_t dd;
    float wscale;
  };
  __device__ static __forceinline__ Head head(uint32_t slot, int r, int, int kk, float wscale) { return Head{lds32(slot + BOX + r * 16 + 4 * kk), wscale}; }
  __device__ static __forceinline__ void half(const Head &hd, uint32_t slot, int r, int kk, int hf, uint32_t (&o)[16]) { // half = one block
    const uint4 q = chunk128(slot, r, 2 * kk + hf);
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

struct RowQ8_0 { // 128 codes per row, then the f16 scales of this super-step and its neighbour
  static constexpr int KPS = 2, SCALES = 1;
  static constexpr uint32_t BOX = ROWS * 128, SLOT = BOX + ROWS * 16;
  __device__ static __forceinline__ void boxes(uint32_t slot, const CUtensorMap *codes, const CUtensorMap *, int ss, int row, uint32_t bar) { tma_box(slot, codes, ss * 128, row, bar); }
  __device__ static __forceinline__ const void *scales(const WeightView &w, int64_t row, int ss, int) {
    return reinterpret_cast<const uint8_t *>(w.d + row * w.dstride) + ((ss * 8) & ~15);
  }
  using Head = RowQ4_0::Head;
  __device__ static __forceinline__ Head head(uint32_t slot, int r, int ss, int kk, float wscale) {
    return Head{lds32(slot + BOX + r * 16 + 8 * (ss & 1) + 4 * kk), wscale};
  }
  __device__ static __forceinline__ void half(const Head &hd, uint32_t slot, int r, int kk, int hf, uint32_t (&o)[16]) { // half = one block
    const uint4 q[2] = {chunk128(slot, r, 4 * kk + 2 * hf), chunk128(slot, r, 4 * kk + 2 * hf + 1)};
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
  static constexpr int KPS = 4, SCALES = 0;
  static constexpr uint32_t BOX = ROWS * 144, SLOT = BOX;
  __device__ static __forceinline__ void boxes(uint32_t slot, const CUtensorMap *codes, const CUtensorMap *, int ss, int row, uint32_t bar) { tma_box(slot, codes, ss * 144, row, bar); }
  __device__ static __forceinline__ const void *scales(const WeightView &, int64_t, int, int) { return nullptr; }
  struct Head {
    __half2 a_lo, a_hi, b_lo, b_hi;
  };
  // value = (d*sc) * code - (dmin*m): low nibbles are sub-block 2g, high nibbles sub-block 2g+1
  __device__ static __forceinline__ Head head(uint32_t slot, int r, int, int g, float wscale) {
    const uint4 hdr = lds128(slot + r * 144);
    const __half2 dm = *reinterpret_cast<const __half2 *>(&hdr.x);
    const uint32_t f = k4_field(hdr.y, hdr.z, hdr.w, g);
    const float d = __low2float(dm) * wscale, mn = __high2float(dm) * wscale;
    return Head{__float2half2_rn(d * (float)(f & 63)), __float2half2_rn(d * (float)((f >> 6) & 63)), __float2half2_rn(-mn * (float)((f >> 12) & 63)),
                __float2half2_rn(-mn * (float)(f >> 18))};
  }
  __device__ static __forceinline__ void half(const Head &hd, uint32_t slot, int r, int g, int hf, uint32_t (&o)[16]) { // half = words 4 hf .. of the group
    const uint4 q = lds128(slot + r * 144 + 16 + 32 * g + 16 * hf);
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

struct RowQ6K { // 128 ql bytes per row, then 64 qh bytes, 16 scales, the f16 d of eight super-blocks
  static constexpr int KPS = 4, SCALES = 2;
  static constexpr uint32_t BOX = ROWS * 192, SLOT = BOX + ROWS * 32, HI = ROWS * 128;
  __device__ static __forceinline__ void boxes(uint32_t slot, const CUtensorMap *codes, const CUtensorMap *high, int ss, int row, uint32_t bar) {
    tma_box(slot, codes, ss * 128, row, bar);
    tma_box(slot + HI, high, ss * 64, row, bar);
  }
  __device__ static __forceinline__ const void *scales(const WeightView &w, int64_t row, int ss, int piece) {
    if (piece == 0) return w.sc + (row * (w.k / QK_K) + ss) * 16;
    return reinterpret_cast<const uint8_t *>(w.d + row * w.dstride) + ((ss * 2) & ~15);
  }
  // k-step kk = 2 h + hi_pair of the super-block: group 0 takes ql[l] of half h, group 1 ql[l + 32], both the low (hi_pair 0) or high nibbles
  struct Head {
    uint4 qh[2];
    uint32_t sc4;
    float d;
  };
  __device__ static __forceinline__ Head head(uint32_t slot, int r, int ss, int kk, float wscale) {
    const int h = kk >> 1;
    Head hd;
    hd.qh[0] = chunk64(slot + HI, r, 2 * h), hd.qh[1] = chunk64(slot + HI, r, 2 * h + 1);
    hd.sc4 = lds32(slot + BOX + r * 16 + 8 * h + 4 * (kk & 1));
    const uint32_t dd = lds32(slot + BOX + ROWS * 16 + r * 16 + 4 * ((ss >> 1) & 3));
    hd.d = __half2float(__ushort_as_half((unsigned short)((ss & 1) ? (dd >> 16) : (dd & 0xffffu)))) * wscale;
    return hd;
  }
  // A branch on which nibbles a warp's k-step takes, so that the shifts are constants: those by 0 and the pair of them that brings the high bits
  // up are gone. Logic, shifts and byte permutes run at half the rate of the rest, and they bound the kernel: seven for four values, now five.
  __device__ static __forceinline__ void half(const Head &hd, uint32_t slot, int r, int kk, int hf, uint32_t (&o)[16]) {
    if (kk & 1) nibbles<4>(hd, slot, r, kk >> 1, hf, o);
    else nibbles<0>(hd, slot, r, kk >> 1, hf, o);
  }
  template <int sh>
  __device__ static __forceinline__ void nibbles(const Head &hd, uint32_t slot, int r, int h, int hf, uint32_t (&o)[16]) {
    const uint4 (&qh)[2] = hd.qh;
    const uint4 ql[2] = {chunk128(slot, r, 4 * h + 2 * hf), chunk128(slot, r, 4 * h + 2 * hf + 1)};
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
        const uint32_t code = ((lw[j] >> sh) & 0x0f0f0f0fu) | ((hsh < 4 ? hw[j] << (4 - hsh) : hw[j] >> (hsh - 4)) & 0x30303030u);
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
