// Prefill (m > 64; Q6_K: m > 16): quantized weights x activations as a dense contraction on the 5th-generation
// tensor cores (tcgen05.mma, accumulators in TMEM).
//
//   D[128 weight rows, mt activation rows] += A[128, 64] . B[mt, 64]^T      per k-step of 64
//
//   A  weights of the tile, dequantized by sixteen producer warps from the quantized blocks into tensor
//      memory, from where the MMA reads them (a lane is a weight row, a column two values). In shared
//      memory, as they were before, they cost a write and a read of 16 KB per k-step, and with 256
//      activation rows the shared memory's 128 bytes a cycle were what bounded the kernel (105 KB and
//      850 cycles a k-step; now 73 KB). Every weight is dequantized once per m-tile (mt up to 256 rows).
//   B  activations, prepared once per call by prefill_prepare_acts: quantized to Q8_0 / Q8_K exactly
//      as the reference's quantize_lhs does (k_quants.rs:2015-2026), dequantized, scaled by a power of
//      two per row and stored as fp16 in the same swizzled image, so that one 1-D bulk-async copy
//      (cp.async.bulk, non-multicast) brings a whole stage.
//   D  f32 in tensor memory; eight drain warps read it back with tcgen05.ld, turn it over in shared memory
//      (in tensor memory a lane is a weight row, y is contiguous along weight rows), undo the power-of-two
//      scales and store y.
//
// Operand type. The contraction runs in fp16 (kind::f16 with f16 inputs), not bf16: both have the
// same tensor throughput, and fp16's 11-bit significand keeps the operand rounding 8x smaller: the
// result stays within about 3e-3 of the OUTPUT RMS of the reference's integer-exact CPU result. Under the
// reference's own element-wise metric |g - w| <= tol * max(|w|, 1) that is 1e-2 only while the output rms
// is below about 3; where outputs are larger the integer-exact kernels are the ones that meet it. Range is handled exactly: every activation row and the whole weight tensor are multiplied
// by powers of two that put their maxima near 2^11 / 2^10, and the epilogue divides them out.
//
// k order. A dot product does not care in which order k is visited as long as both operands agree,
// so within a k-step the 64 elements are stored in the order the nibble unpack produces them
// (xnq_prefill_rows.cuh) and the activation image uses the same order; no shuffles are needed.
//
// Synchronisation. Per stage: full (one arrival per producer warp of the stage and one of the loader, whose
// bulk copy adds its transaction bytes) and empty (tcgen05.commit by the MMA warp). Every wait is bounded; on
// expiry a status bit is set and every role falls through to the common exit, where tensor memory is released.
#include <algorithm>
#include <climits>
#include <cstring>

#include "xnq_common.cuh"
#include "xnq_quantize_act.cuh"
#include "xnq_prefill_rows.cuh"
#include "xnq_unpack.cuh"

namespace xnq {

__device__ unsigned int g_prefill_status; // sticky: 1 producer wait, 2 loader wait, 4 mma wait, 8 epilogue wait expired

namespace {

constexpr int BK = 64;             // k-step (elements) = one 128-byte swizzle row of fp16
constexpr int TILE_N = 128;        // weight rows per CTA = UMMA M
constexpr int MAX_MT = 256;        // activation rows per CTA = UMMA N
constexpr int PRODUCER_WARPS = 16; // four row groups of 32 rows x four warps
constexpr int EPI_WARPS = 8;       // two per accumulator lane quarter, which take turns in its chunks of 16 columns
constexpr int LOADER_WARP = PRODUCER_WARPS, MMA_WARP = LOADER_WARP + 1, EPI_WARP0 = MMA_WARP + 1, COPY_WARP = EPI_WARP0 + EPI_WARPS;
constexpr int NTHREADS = (COPY_WARP + 1) * 32;
constexpr uint32_t EPI_SLOT = 16 * 32 * 4; // a drain warp's chunk: 16 columns of 32 weight rows, f32
constexpr uint32_t WAIT_LIMIT = 1u << 26; // polls of a flag in global memory
constexpr int A_COLS = BK / 2;     // tensor-memory columns of a stage's weights
constexpr int A_COL0 = 256;        // they start behind the accumulators: one of 256 columns or two of 128
// Stages. At least as many as a super-step has k-steps: step i then waits for the MMAs of a step of an EARLIER super-step, whose
// producer (same row group) has already waited for the phase before; with fewer, a warp could test a barrier that is two phases
// behind, which reads as complete.
constexpr int MIN_STAGES = 4, MAX_STAGES = 8;
constexpr int MAX_RAW_SLOTS = 6;   // super-steps of raw weight bytes in shared memory

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// One wait attempt during which the hardware may keep the thread suspended for up to `ns` nanoseconds (it takes no issue slots).
__device__ __forceinline__ bool mbar_suspend(uint32_t bar, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(ns)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long wall_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull; // a wait that lasts two seconds is given up
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned int bit) {
  unsigned long long t0 = 0;
  for (unsigned int attempt = 1;; attempt++) { // the wall clock is read on every 16th failed attempt only
    if (mbar_suspend(bar, parity, 1000000u)) return true;
    if ((attempt & 15u) == 0) {
      const unsigned long long now = wall_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > WAIT_LIMIT_NS) break;
    }
  }
  atomicOr(&g_prefill_status, bit);
  return false;
}
// by a whole warp that stays converged; the result is the same in all lanes. (Each lane polls and reads the clock for itself, so one may give up while
// another sees the phase complete. A role that votes on what it looked at ahead has to go on with one answer: lanes that had given up would pass by a
// vote that the others wait in, without a limit.)
__device__ __forceinline__ bool mbar_wait_uniform(uint32_t bar, uint32_t parity, unsigned int bit) {
  const bool ok = mbar_wait(bar, parity, bit);
  return __all_sync(0xffffffffu, ok);
}
// Whether the phase has completed, without waiting for it. A wait takes 120 to 250 cycles even when there is nothing to wait for, and with 32 rows every
// role took a turn of 550 cycles that way. The loops below look at the next turn's barrier while this turn's work is under way and wait only for what was
// not there yet: Q4_K 28672 x 4096, 65 rows 38.0 -> 36.2 us; Q8_0 8192 x 4096, 128 rows 29.4 -> 28.4; with Q6_K's shorter conversion, Q6_K 128256 x 4096, 32
// rows 142 -> 131 in one run (137 in most; a long stream of calls, under the power limit). (Two k-steps a turn on top: no difference.)
__device__ __forceinline__ bool mbar_peek(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// ---- CTA pairs (a cluster of two) ----
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() { // by every thread of both CTAs
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// the same barrier in the leader's (rank 0's) shared memory
__device__ __forceinline__ uint32_t leader_addr(uint32_t bar) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(bar));
  return a;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// true in one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}

// ---- tcgen05 wrappers --------------------------------------------------------------------------------
// CG: CTAs that work together on a tile. All of a kernel's tcgen05 instructions name the same number.
template <int CG>
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  if (CG == 2) asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
  else asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
template <int CG>
__device__ __forceinline__ void tmem_relinquish() {
  if (CG == 2) asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  else asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <int CG>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
  else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// A from tensor memory, B from shared memory. CG 2: every CTA of the pair has its 128 weight rows in its own tensor memory and half of the
// activation rows in its own shared memory, both at the addresses that are named here, and gets its 128 rows of the result.
template <int CG>
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if (CG == 2)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the mbarrier (CG 2: on that of each CTA of the pair) once every MMA issued so far by this thread has finished reading and writing
template <int CG>
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  if (CG == 2)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
  else asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
      "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// K-major, 128-byte-swizzled operand tile: rows of 128 bytes, 8-row groups 1024 bytes apart.
// Fields: start address >> 4 [0,14), leading byte offset >> 4 [16,30) (unused for swizzled K-major),
// stride byte offset >> 4 [32,46), descriptor version 1 [46,48), swizzle mode 2 = 128 B [61,64).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3ffffu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// kind::f16 instruction descriptor: D f32 (bit 4), A/B format (0 = f16) at [7,10) / [10,13), both K-major,
// N >> 3 at [17,23), M >> 4 at [24,29).
__device__ __forceinline__ uint32_t idesc_f16(int umma_m, int umma_n) { return (1u << 4) | ((uint32_t)(umma_n >> 3) << 17) | ((uint32_t)(umma_m >> 4) << 24); }

struct PrefillArgs {
  WeightView w;
  const uint8_t *xh;      // activation image: [k-steps][m_pad][64] fp16, swizzled rows, k-step-permuted
  const float *row_unscale; // [m_pad]: 1 / (activation row scale * weight scale)
  void *y;
  const void *bias;       // n values of y's type, or null
  int y_dtype;
  int64_t ldy;
  int64_t m, m_pad;
  int mt;                 // activation rows of a tile (the last one may have fewer)
  int ksteps;
  int nstages;            // stages: weights in tensor memory, activations in shared memory
  int acc_bufs;           // accumulators: 1 of 256 columns, 2 of 128 (tiles of up to 128 activation rows)
  int raw_slots;          // raw super-steps in shared memory, the one being converted included
  int vec_out;            // rows of y start on 16 bytes and hold whole 16-byte pieces
  uint32_t b_stride;      // bytes between B stages (largest mt of the grid x 128, multiple of 1024)
  uint32_t raw_off, epi_off; // offsets of the raw ring and of the drain warps' chunks behind the B ring
  float wscale;           // power of two applied to every dequantized weight
  // persistent kernel: tile t = tile_n * tiles_m + tile_m; work unit u = t * ksteps + kt; CTA (or pair) c takes units
  // [units * c / G, units * (c + 1) / G), or whole tiles when the output cannot be accumulated atomically. share_q, share_r: what is divided
  // (units or tiles) by G and its remainder, set at launch: the 64-bit divisions held every thread of every CTA back before its first copy
  int tiles_n, tiles_m;   // tiles_n: of 128 weight rows, or of a pair's 256
  long long units, share_q;
  int share_r;
  int whole_tiles;
  int row_tiles;          // tiles of 128 weight rows: the last pair's second CTA may have none
  unsigned int *tile_cnt; // per (row tile, m-tile) arrival tickets, then "first partial stored" flags; zeroed by the prepare kernel
};

using namespace prefill_rows;

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }

// How a chunk (16 columns = activation rows, 32 weight rows) reaches y. In the accumulator a lane is a weight row, and y is contiguous along
// weight rows.
enum Store { STORE_F32, ADD_F32, STORE_F16, STORE_BF16 };
template <int ST>
__device__ __forceinline__ uint32_t pack16(float a, float b) {
  if (ST == STORE_F16) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
  }
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}
// Rows of y that start on 16 bytes: the chunk is turned over in shared memory (column j of weight row l at j * 128 + 4 l, 16-byte pieces
// swapped in odd columns so that the 16-bit types' reads of two neighbouring pieces touch all banks) and leaves in 16-byte stores, 8 or 4
// lanes to a row: a quarter of the store instructions. yp: this warp's first weight row in the chunk's first activation row; cols: how many
// columns exist; rows: how many of the 32 weight rows; ru: shared address of the chunk's row factors; bias: of the weight rows' bias in f32, or 0.
template <int ST>
__device__ __forceinline__ float plus(float v, float bias) { return with_bias(v, bias, ST == STORE_F16 ? XNQ_F16 : (ST == STORE_BF16 ? XNQ_BF16 : XNQ_F32)); }
template <int ST>
__device__ __forceinline__ float4 add4(float4 o, uint32_t bias) {
  const uint4 b = lds128(bias);
  return make_float4(plus<ST>(o.x, __uint_as_float(b.x)), plus<ST>(o.y, __uint_as_float(b.y)), plus<ST>(o.z, __uint_as_float(b.z)), plus<ST>(o.w, __uint_as_float(b.w)));
}
template <int ST>
__device__ __forceinline__ void store_turned(uint32_t slot, uint32_t ru, uint32_t bias, char *yp, int64_t row_bytes, int cols, int rows, int lane) {
  if (ST <= ADD_F32) {
    const int j0 = lane >> 3, piece = lane & 7;
    const uint32_t at = slot + (uint32_t)(j0 * 128 + ((piece ^ (j0 & 1)) << 4));
    char *p = yp + j0 * row_bytes + piece * 16;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint4 v = lds128(at + i * 512);
      const float f = __uint_as_float(lds32(ru + (uint32_t)((4 * i + j0) * 4)));
      float4 o = make_float4(__uint_as_float(v.x) * f, __uint_as_float(v.y) * f, __uint_as_float(v.z) * f, __uint_as_float(v.w) * f);
      if (ST != ADD_F32 && bias) o = add4<ST>(o, bias + piece * 16);
      if (4 * i + j0 < cols && piece * 4 < rows) {
        if (ST == STORE_F32) *reinterpret_cast<float4 *>(p) = o;
        else atomicAdd(reinterpret_cast<float4 *>(p), o);
      }
      p += 4 * row_bytes;
    }
  } else {
    const int j0 = lane >> 2, piece = (lane & 3) * 2;
    const uint32_t at = slot + (uint32_t)(j0 * 128);
    const uint32_t p0 = (uint32_t)((piece ^ (j0 & 1)) << 4), p1 = p0 ^ 16u;
    char *p = yp + j0 * row_bytes + piece * 8;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const uint4 a = lds128(at + i * 1024 + p0), b = lds128(at + i * 1024 + p1);
      const float f = __uint_as_float(lds32(ru + (uint32_t)((8 * i + j0) * 4)));
      float4 l = make_float4(__uint_as_float(a.x) * f, __uint_as_float(a.y) * f, __uint_as_float(a.z) * f, __uint_as_float(a.w) * f);
      float4 h = make_float4(__uint_as_float(b.x) * f, __uint_as_float(b.y) * f, __uint_as_float(b.z) * f, __uint_as_float(b.w) * f);
      if (bias) l = add4<ST>(l, bias + piece * 16), h = add4<ST>(h, bias + piece * 16 + 16);
      const uint4 o = make_uint4(pack16<ST>(l.x, l.y), pack16<ST>(l.z, l.w), pack16<ST>(h.x, h.y), pack16<ST>(h.z, h.w));
      if (8 * i + j0 < cols && piece * 4 < rows) *reinterpret_cast<uint4 *>(p) = o;
      p += 8 * row_bytes;
    }
  }
}
// Other rows: a lane stores its weight row's values one by one, neighbouring lanes to neighbouring addresses. ADDS: with the bias (with a
// test beside every value, and a load of each factor by itself, Q4_K 6890 x 512, 484 rows, bf16 results took 14.1 us instead of 13.4; Q8_0 9001 x 1024, 100 rows,
// f16 12.3 and 12.1).
template <int ST, bool ADDS>
__device__ __forceinline__ void store_each(const uint32_t (&v)[16], uint32_t ru, float add, char *p, int64_t row_bytes, int cols) {
#pragma unroll
  for (int j0 = 0; j0 < 16; j0 += 4) {
    const uint4 f4 = lds128(ru + (uint32_t)(j0 * 4));
    const uint32_t f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      float val = __uint_as_float(v[j0 + i]) * __uint_as_float(f[i]);
      if (ADDS) val = plus<ST>(val, add);
      if (j0 + i < cols) {
        if (ST == STORE_F32) *reinterpret_cast<float *>(p) = val;
        else if (ST == ADD_F32) atomicAdd(reinterpret_cast<float *>(p), val);
        else if (ST == STORE_F16) *reinterpret_cast<__half *>(p) = __float2half_rn(val);
        else *reinterpret_cast<__nv_bfloat16 *>(p) = __float2bfloat16_rn(val);
      }
      p += row_bytes;
    }
  }
}
template <int ST>
__device__ __forceinline__ void store_direct(const uint32_t (&v)[16], uint32_t ru, uint32_t bias, char *yp, int64_t row_bytes, int cols, bool row_ok, int lane) {
  char *const p = yp + lane * (ST <= ADD_F32 ? 4 : 2);
  if (!row_ok) cols = 0;
  if (ST != ADD_F32 && bias) store_each<ST, true>(v, ru, __uint_as_float(lds32(bias + lane * 4)), p, row_bytes, cols);
  else store_each<ST, false>(v, ru, 0.f, p, row_bytes, cols);
}

// ---- the kernel ------------------------------------------------------------------------------------------------
// CG 2: the CTAs of a cluster of two take 128 weight rows each of a tile and one MMA (cta_group::2) works for both, so that each CTA brings
// only half of the tile's activation rows: per k-step of 256 rows 16 KB instead of 32 through L2 and shared memory, which at 512 cycles of
// MMA were what bounded such tiles (28672 x 4096, 2000 rows: 415 -> 390 us at full clock). The leader issues the MMAs; the other CTA's warp
// of that role tells it when its half of a stage is there, and the commits arrive on both CTAs' barriers. (The relay's arrival and the
// leader's wait have the default semantics: with .release.cluster and .acquire.cluster each costs a fence of some 1000 cycles and the kernel
// took 654 us. PTX promises the order at that scope only; the default suffices because what it orders, tensor-memory stores and bulk copies, has been
// performed in the memory of the CTA whose half of the MMA reads it before that CTA's own barrier lets the relay pass.)
// One CTA per SM (or pair per two) walks a contiguous range of the flattened (tile, k-step) space, so all SMs finish
// together whatever the tile count, and a tile whose k-steps are split between CTAs is summed in
// global memory: the first CTA to finish its part stores it and raises the tile's flag, the others add
// theirs atomically after seeing the flag (two to three parts per split tile; f32 output only - other
// output types get whole tiles). Tiles of up to 128 activation rows have two accumulators, so the drain of one
// segment overlaps the MMAs of the next. Wider ones have one, whose halves of columns the drain gives back one by one: the first
// MMAs of the next segment go to the half that is free.
// Roles: 16 producer warps, one activation-loader warp (one bulk copy per stage), one MMA-issuing warp, eight drain
// warps, one warp that requests raw weights. Stage counters run on across segments.
// Producers: the four warps of a row group (32 weight rows) convert a k-step each of a super-step (or a half of one), so the k-steps of a
// super-step are converted side by side and a warp's chain of waits, loads, arithmetic and stores has a super-step's MMAs to run in.
// Measured, start of each -> with it (long stream of calls): the turned drain, the halves and copies by warps of their own, Q4_0 4096 x 4096, 200 rows
// 32.5 -> 25.6 us, Q4_K 4096 x 4096, 300 rows 31.9 -> 29.3; weights in boxes of tensor maps and a short turn of the activation loader, Q4_K 28672 x
// 4096, 2000 rows (bf16 results) 443 -> 417, Q8_0 11008 x 4096, 512 rows 64.0 -> 61.4, Q6_K 128256 x 4096, 32 rows 155 -> 138, Q4_K 14336 x 4096, 512
// rows 72.2 -> 70.3. What bounds it now: wide tiles the power limit and the tensor core's 512 cycles a k-step (pairs) or the 32 KB of activations that a
// k-step brings through L2 (single CTAs: 750 to 800 cycles), narrow ones the instructions of the conversion and the latencies between the roles (500
// cycles a k-step).
struct Cursor { // position in the flattened (tile, k-step) space; tile = tile_n * tiles_m + tile_m
  int tile_n, tile_m, kt;
  __device__ __forceinline__ void advance(int steps, int KT, int tiles_m) {
    kt += steps;
    while (kt >= KT) {
      kt -= KT;
      if (++tile_m == tiles_m) {
        tile_m = 0;
        tile_n++;
      }
    }
  }
};

// columns of an accumulator's first half, which is given back to the MMAs on its own; n: the widest tile's (narrower ones are divided there too,
// as a segment's first MMAs go by what the segment before has given back)
template <int CG>
__device__ __forceinline__ int first_half(int n) { return (n / 2 + 16 * CG - 1) / (16 * CG) * (16 * CG); }
// The activation row of a tile whose products are in accumulator column c. Pairs: each half of the n columns holds first rows of the leader's
// half of the tile, then rows of the other CTA's.
template <int CG>
__device__ __forceinline__ int row_of_column(int c, int n) {
  if (CG == 1) return c;
  const int h0 = first_half<2>(n), upper = c >= h0, q = (upper ? n - h0 : h0) / 2, cc = upper ? c - h0 : c;
  const int cta = cc >= q;
  return cta * (n / 2) + (upper ? h0 / 2 : 0) + cc - cta * q;
}

template <typename RowT, int CG>
__global__ void __launch_bounds__(NTHREADS, 1) prefill_persistent_kernel(const __grid_constant__ PrefillArgs p, const __grid_constant__ CUtensorMap codes, const __grid_constant__ CUtensorMap high) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  __shared__ __align__(8) uint64_t bars[2 * MAX_STAGES + 4 + 2 * MAX_RAW_SLOTS]; // full, empty (8 each), acc_full[2], acc_empty[2], raw_full, raw_empty
  __shared__ __align__(16) float s_ru[MAX_MT]; // the tile's row factors
  __shared__ __align__(16) float s_bias[TILE_N]; // and the bias of its weight rows
  __shared__ uint32_t tmem_slot;
  __shared__ unsigned int s_ticket;
  const int S = p.nstages;
  const uint32_t full = smem_u32(bars), empty = full + 8 * MAX_STAGES, acc_full = empty + 8 * MAX_STAGES, acc_empty = acc_full + 16, raw_full = acc_empty + 16,
                 raw_empty = raw_full + 8 * MAX_RAW_SLOTS;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31; // so that the compiler knows `warp` to be uniform
  const uint32_t b_ring = smem_base;
  const int NACC = p.acc_bufs;
  const int KT = p.ksteps;
  const uint32_t rank = CG == 2 ? cluster_rank() : 0u; // 0: the pair's leader, which issues its MMAs

  // this CTA's (or pair's) range of work units
  const int cta = (int)blockIdx.x / CG, ctas = (int)gridDim.x / CG;
  long long u0 = p.share_q * cta + cta * p.share_r / ctas, u1 = p.share_q * (cta + 1) + (cta + 1) * p.share_r / ctas;
  if (p.whole_tiles) u0 *= KT, u1 *= KT;
  const int nsteps = (int)(u1 - u0);
  const int TM = p.tiles_m;
  const int tile0 = p.units <= INT_MAX ? (int)u0 / KT : (int)(u0 / KT);
  const Cursor start{tile0 / TM, tile0 % TM, (int)(u0 - (long long)tile0 * KT)};

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(full + 8 * s, PRODUCER_WARPS / RowT::KPS + 1 + (CG == 2 && rank == 0 ? 1 : 0)); // the leader's: and one by the other CTA's relay
      mbar_init(empty + 8 * s, 1);
    }
    for (int r = 0; r < p.raw_slots; r++) {
      mbar_init(raw_full + 8 * r, 1 + (RowT::SCALES ? 32 : 0)); // the boxes, and the lanes that copy scale data
      mbar_init(raw_empty + 8 * r, PRODUCER_WARPS);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(acc_full + 8 * b, 1);
      mbar_init(acc_empty + 8 * b, EPI_WARPS * CG); // (used in the leader only)
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == LOADER_WARP) {
    tmem_alloc<CG>(smem_u32(&tmem_slot), 512);
    tmem_relinquish<CG>();
  }
  tc_fence_before();
  if (CG == 2) cluster_sync(); // the other CTA's barriers are set up
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();
  const uint32_t tmem_d = __shfl_sync(0xffffffffu, tmem_slot, 0);

  constexpr int KPS = RowT::KPS;
  constexpr uint32_t SLOT = RowT::SLOT;
  static_assert(ROWS == TILE_N && SLOT % 1024 == 0, "swizzled boxes start on 1024 bytes");
  const int SPT = (KT + KPS - 1) / KPS; // super-steps per tile
  const int R = p.raw_slots;
  const int last_kt = nsteps - 1 + start.kt; // counted from the start of the first tile
  const int nsuper = nsteps > 0 ? (last_kt / KT) * SPT + (last_kt % KT) / KPS - start.kt / KPS + 1 : 0; // super-steps of this CTA
  if (warp < PRODUCER_WARPS) {
    // ---- producers: the four warps of a row group convert a k-step of a super-step each (KPS 2: half of one) ----
    const int rg = warp & 3, kg = warp >> 2;
    const int kk = kg % KPS, hf = kg / KPS; // this warp's k-step of a super-step; which half of it (KPS = 2)
    const uint32_t raw = smem_base + p.raw_off;
    const int r = rg * 32 + lane; // row in the tile
    int c_s = start.kt / KPS, slot = 0;
    uint32_t raw_lap = 0;
    int base_i = -start.kt; // the CTA's step number of the current tile's first k-step
    int at = 0, s = 0;      // s = at % S, lap: parity of at / S, of the last step this warp looked at
    uint32_t lap = 0;
    const bool lockstep = KT % KPS != 0 && KPS + KT % KPS > S;
    bool alive = true, raw_ready = false, empty_ready = false;
    for (int left = nsuper; left > 0; left--) {
      if (alive && !__all_sync(0xffffffffu, raw_ready)) alive = mbar_wait_uniform(raw_full + 8 * slot, raw_lap, 1u);
      // A warp waits for a stage only on behalf of a step that it fills: that step's MMAs, and so the stage's next phase, wait for this warp in
      // turn, while a barrier that runs on without it may be two phases ahead by the time it looks, which a parity cannot tell from none. Where
      // a warp's k-step is missing from a tile's last super-step, two of its waits may then be more than S steps apart, and the second could
      // take an older phase for its own: there (Q4_0 with k not a multiple of 256) the four warps of a row group start a tile together.
      if (lockstep && c_s == 0) asm volatile("bar.sync %0, 128;" ::"r"(2 + rg) : "memory");
      const int kt = c_s * KPS + kk, i = base_i + kt;
      if (alive && kt < KT && i >= 0 && i < nsteps) {
        for (s += i - at, at = i; s >= S; lap ^= 1u) s -= S;
        if (i >= S && !__all_sync(0xffffffffu, empty_ready)) alive = mbar_wait_uniform(empty + 8 * s, lap ^ 1u, 1u);
        empty_ready = false;
        if (alive) {
          tc_fence_after();
          const uint32_t at_slot = raw + (uint32_t)slot * SLOT;
          const uint32_t dst = tmem_d + ((uint32_t)(32 * rg) << 16) + (uint32_t)(A_COL0 + s * A_COLS);
          const typename RowT::Head head = RowT::head(at_slot, r, c_s, kk, p.wscale);
#pragma unroll
          for (int h = 0; h < KPS / 2; h++) {
            const int half = KPS == 2 ? hf : h;
            uint32_t o[16];
            RowT::half(head, at_slot, r, kk, half, o); // (what a lane past the weight's last row makes is not stored)
            tmem_st16(dst + 16 * half, o);
          }
          const int next = s + KPS - (s + KPS >= S ? S : 0); // of this warp's next step, if this tile has one
          empty_ready = kt + KPS < KT && mbar_peek(empty + 8 * next, s + KPS >= S ? lap : lap ^ 1u);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(full + 8 * s);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(raw_empty + 8 * slot); // (also by a warp that gave up)
      if (++slot == R) slot = 0, raw_lap ^= 1u;
      raw_ready = mbar_peek(raw_full + 8 * slot, raw_lap);
      if (++c_s == SPT) {
        c_s = 0;
        base_i += KT;
      }
    }
  } else if (warp == COPY_WARP) {
    // ---- raw weights: one warp requests a super-step's boxes, and copies the rows' scale data where it lies apart, up to R super-steps ahead.
    // (While the rows were copied by cp.async, by the producers or by warps of their own, that took 1100 to 1700 cycles a super-step.) Nothing
    // here waits for the kernel that prepares the activations: weights are immutable. ----
    Cursor cur = start;
    int l_s = start.kt / KPS, slot = 0, issued = 0;
    uint32_t lap = 0;
    for (int j = 0; j < nsuper; j++) {
      if (j >= R && !mbar_wait_uniform(raw_empty + 8 * slot, lap ^ 1u, 1u)) break;
      const int64_t row0 = ((int64_t)cur.tile_n * CG + rank) * TILE_N;
      const uint32_t dst = smem_base + p.raw_off + (uint32_t)slot * SLOT, bar = raw_full + 8 * slot;
      if (elect_one()) {
        mbar_expect_tx(bar, RowT::BOX);
        RowT::boxes(dst, &codes, &high, l_s, (int)row0, bar);
      }
      __syncwarp();
      if constexpr (RowT::SCALES > 0) {
#pragma unroll
        for (int i = 0; i < 4 * RowT::SCALES; i++) {
          const int r = (i & 3) * 32 + lane;
          cp_async16(dst + RowT::BOX + (uint32_t)((i >> 2) * TILE_N * 16 + r * 16), RowT::scales(p.w, min(row0 + r, p.w.n - 1), l_s, i >> 2));
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory"); // when this lane's copies have landed
      }
      issued = j + 1;
      if (++slot == R) slot = 0, lap ^= 1u;
      if (++l_s == SPT) {
        l_s = 0;
        cur.kt = 0;
        cur.advance(KT, KT, TM);
      }
    }
    for (int j = max(0, issued - R); j < issued; j++) mbar_wait_uniform(raw_full + 8 * (j % R), (j / R) & 1, 1u);
    asm volatile("cp.async.wait_all;" ::: "memory"); // nothing in flight into this CTA's shared memory when it exits
  } else if (warp == LOADER_WARP) {
    // ---- activation loader: the whole warp runs the loop and one elected lane issues (see the MMA issuer). A turn is kept short (a wait, an
    // arrival, a copy, with what a tile needs worked out beforehand): it shares its scheduler with busy warps. (When every step was worked out in
    // 64 bits a turn took 650 cycles, more than the MMAs of 256 rows, and the activations were what every step waited for; as long with one
    // thread in a branch, whose copy's operands move to uniform registers one by one.) ----
    pdl_wait(); // the activation image is the previous kernel's output
    Cursor cur = start;
    int s = 0, i = 0;
    uint32_t lap = 0;
    bool alive = true, ready = false;
    while (i < nsteps) {
      // a pair's CTAs bring half of the tile's rows each (the last tile's second half may have fewer, or none: what is then left in the
      // stage reaches only columns that are not stored)
      const int64_t tm0 = (int64_t)cur.tile_m * p.mt, m0 = tm0 + (CG == 2 ? (int)rank * (p.mt / 2) : 0);
      const int rows = (int)min((int64_t)(p.mt / CG), min(tm0 + p.mt, p.m_pad) - m0);
      const uint32_t bytes = (uint32_t)max(rows, 0) * 128;
      const uint8_t *src = p.xh + ((size_t)cur.kt * p.m_pad + m0) * 128;
      const size_t step = (size_t)p.m_pad * 128;
      const int len = min(KT - cur.kt, nsteps - i), end = i + len;
      for (; i < end; i++, src += step) {
        if (i >= S && alive && !__all_sync(0xffffffffu, ready)) alive = mbar_wait_uniform(empty + 8 * s, lap ^ 1u, 2u);
        if (elect_one() && alive) {
          if (bytes) {
            mbar_expect_tx(full + 8 * s, bytes);
            bulk_g2s(b_ring + s * p.b_stride, src, bytes, full + 8 * s);
          } else {
            mbar_arrive(full + 8 * s);
          }
        }
        __syncwarp();
        if (++s == S) s = 0, lap ^= 1u;
        ready = mbar_peek(empty + 8 * s, lap ^ 1u);
      }
      cur.advance(len, KT, TM);
    }
    for (int j = max(0, nsteps - S); j < nsteps && alive; j++) alive = mbar_wait_uniform(full + 8 * (j % S), (j / S) & 1, 2u); // nothing in flight at exit
  } else if (CG == 2 && warp == MMA_WARP && rank != 0) {
    // ---- relay: tells the leader that this CTA's half of a stage is there ----
    const uint32_t to = leader_addr(full);
    bool alive = true;
    for (int i = 0, s = 0, round = 0; i < nsteps && alive; i++) {
      alive = mbar_wait_uniform(full + 8 * s, round & 1, 4u);
      tc_fence_after();
      tc_fence_before();
      if (alive && elect_one()) mbar_arrive_cluster(to + 8 * s);
      __syncwarp();
      if (++s == S) {
        s = 0;
        round++;
      }
    }
  } else if (warp == MMA_WARP) {
    // ---- MMA issuer: the whole warp runs the loop and one elected lane issues. Everything that decides a loop's course or a
    // descriptor is a function of launch parameters and counters (a wait that gave up only makes the rest of the loop idle), so
    // that the compiler can keep the descriptors in uniform registers: moving them there from vector registers, one after the
    // other, holds a thread for 96 cycles per MMA, while the tensor core takes one every 40 (N <= 32), 48 (64), 64 (128) or
    // 128 (256) cycles. ----
    Cursor cur = start;
    bool alive = true;
    int i = 0, s = 0;
    uint32_t round = 0;
    for (int seg = 0; i < nsteps; seg++) {
      const int len = min(KT - cur.kt, nsteps - i);
      const int N = CG == 2 ? p.mt : min(p.mt, (int)p.m_pad - cur.tile_m * p.mt);
      // A pair's MMAs always take the two halves of the columns one after the other: which CTA's activation rows are in which columns depends
      // on an instruction's width.
      const int h0 = min(first_half<CG>(p.mt), N);
      const uint32_t idesc = idesc_f16(TILE_N * CG, N), id0 = idesc_f16(TILE_N * CG, h0), id1 = idesc_f16(TILE_N * CG, N - h0);
      int j = 0;
      if (NACC == 1 && seg > 0) {
        // One accumulator: its first half of columns is free while the second is still drained. The first steps of the segment go there
        // alone and catch up in the second half when that is free too.
        const int early = min(len, S / 2), s0 = s;
        if (alive) alive = mbar_wait_uniform(acc_empty, (seg - 1) & 1, 4u);
        for (; j < early; j++) {
          if (alive) alive = mbar_wait_uniform(full + 8 * s, round & 1, 4u);
          tc_fence_after();
          __syncwarp();
          const uint32_t a = tmem_d + (uint32_t)(A_COL0 + s * A_COLS);
          const uint64_t bdesc = smem_desc_sw128(b_ring + s * p.b_stride);
          if (elect_one() && alive) {
#pragma unroll
            for (int ks = 0; ks < BK / 16; ks++) umma_f16<CG>(tmem_d, a + (uint32_t)(ks * 8), bdesc + (uint64_t)(ks * 2), id0, (j | ks) ? 1u : 0u);
          }
          __syncwarp();
          if (++s == S) {
            s = 0;
            round++;
          }
        }
        if (alive) alive = mbar_wait_uniform(acc_empty + 8, (seg - 1) & 1, 4u);
        tc_fence_after();
        __syncwarp();
        for (int t = 0, ts = s0; t < early; t++) {
          const uint32_t a = tmem_d + (uint32_t)(A_COL0 + ts * A_COLS);
          const uint64_t bdesc = smem_desc_sw128(b_ring + ts * p.b_stride + (uint32_t)(h0 / CG) * 128);
          if (elect_one() && alive) {
            if (N > h0) { // (an instruction of no columns is an illegal one)
#pragma unroll
              for (int ks = 0; ks < BK / 16; ks++) umma_f16<CG>(tmem_d + (uint32_t)h0, a + (uint32_t)(ks * 8), bdesc + (uint64_t)(ks * 2), id1, (t | ks) ? 1u : 0u);
            }
            umma_commit<CG>(empty + 8 * ts);
            if (t == len - 1) umma_commit<CG>(acc_full);
          }
          __syncwarp();
          if (++ts == S) ts = 0;
        }
      }
      const int buf = NACC == 2 ? seg & 1 : 0;
      if (NACC == 2 && seg >= 2 && alive) alive = mbar_wait_uniform(acc_empty + 8 * buf, ((seg >> 1) - 1) & 1, 4u); // the drain of this buffer's previous segment
      const uint32_t d = tmem_d + (uint32_t)(buf * 128);
      bool ready = false;
      for (; j < len; j++) {
        if (alive && !__all_sync(0xffffffffu, ready)) alive = mbar_wait_uniform(full + 8 * s, round & 1, 4u);
        tc_fence_after();
        __syncwarp();
        const uint32_t a = tmem_d + (uint32_t)(A_COL0 + s * A_COLS);
        const uint64_t bdesc = smem_desc_sw128(b_ring + s * p.b_stride);
        if (elect_one() && alive) {
#pragma unroll
          for (int ks = 0; ks < BK / 16; ks++) umma_f16<CG>(d, a + (uint32_t)(ks * 8), bdesc + (uint64_t)(ks * 2), CG == 2 ? id0 : idesc, (j | ks) ? 1u : 0u);
          if (CG == 2 && N > h0) {
#pragma unroll
            for (int ks = 0; ks < BK / 16; ks++)
              umma_f16<CG>(d + (uint32_t)h0, a + (uint32_t)(ks * 8), bdesc + (uint64_t)(h0 / CG * 8) + (uint64_t)(ks * 2), id1, (j | ks) ? 1u : 0u);
          }
          umma_commit<CG>(empty + 8 * s);
          if (j == len - 1) umma_commit<CG>(acc_full + 8 * buf);
        }
        __syncwarp();
        if (++s == S) {
          s = 0;
          round++;
        }
        ready = mbar_peek(full + 8 * s, round & 1);
      }
      i += len;
      cur.advance(len, KT, TM);
    }
  } else {
    // ---- drain: eight warps, two to a quarter q of the accumulator lanes (weight rows 32 q ..), which take turns in its chunks of 16 columns ----
    const int q = warp & 3; // tensor-memory lanes a warp may read are fixed by its index modulo 4
    const int half = (warp - EPI_WARP0) >> 2; // which of the quarter's two warps
    const int et = threadIdx.x - EPI_WARP0 * 32; // 0..255
    const uint32_t slot = smem_base + p.epi_off + (uint32_t)(warp - EPI_WARP0) * EPI_SLOT;
    auto give_back = [&](uint32_t bar) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2) mbar_arrive_cluster(leader_addr(bar));
        else mbar_arrive(bar);
      }
    };
    pdl_wait(); // the previous kernel writes the row factors and zeroes the tiles' tickets
    Cursor cur = start;
    bool alive = true;
    int i = 0;
    for (int seg = 0; i < nsteps && alive; seg++) {
      const int len = min(KT - cur.kt, nsteps - i);
      const int row_tile = cur.tile_n * CG + (int)rank, tile = row_tile * TM + cur.tile_m;
      const bool whole = CG == 2 || (cur.kt == 0 && len == KT); // (pairs take whole tiles of 16-bit results only)
      const int buf = NACC == 2 ? seg & 1 : 0, use = NACC == 2 ? seg >> 1 : seg;
      const int64_t m0 = (int64_t)cur.tile_m * p.mt;
      const int mt = CG == 2 ? p.mt : (int)min((int64_t)p.mt, p.m_pad - m0); // columns
      const int64_t m_end = min(p.m, m0 + mt);
      // one thread waits for the accumulator and, for a tile shared with other CTAs, settles who stores and
      // who adds; the eight warps then act on the same answers
      if (et == 0) {
        unsigned int t = mbar_wait(acc_full + 8 * buf, use & 1, 8u) ? 0u : 0x80000000u;
        if (!whole && t == 0) {
          t = atomicAdd(p.tile_cnt + tile, 1u);
          if (t > 0) { // wait (bounded) until the first finisher's stores are visible
            const unsigned int *flag = p.tile_cnt + (size_t)p.row_tiles * TM + tile;
            uint32_t spins = 0;
            unsigned int v = 0;
            do {
              asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
            } while (v == 0 && ++spins < WAIT_LIMIT);
            if (v == 0) {
              atomicOr(&g_prefill_status, 8u);
              t = 0x80000000u;
            }
          }
        }
        s_ticket = t;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
      if (et < mt) {
        const int64_t r = m0 + row_of_column<CG>(et, mt);
        s_ru[et] = r < p.m_pad ? p.row_unscale[r] : 0.f;
      }
      if (p.bias && et < TILE_N) {
        const int64_t r = (int64_t)row_tile * TILE_N + et;
        s_bias[et] = r < p.w.n ? bias_at(p.bias, p.y_dtype, r) : 0.f;
      }
      const unsigned int ticket = s_ticket & 0x7fffffffu;
      alive = (s_ticket & 0x80000000u) == 0;
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory"); // s_ticket may be rewritten from here on, s_ru is filled
      if (alive) {
        tc_fence_after();
        const uint32_t lane_addr = tmem_d + (uint32_t)(buf * 128) + ((uint32_t)(32 * q) << 16);
        const bool f32 = CG == 1 && p.y_dtype == XNQ_F32;
        const int es = f32 ? 4 : 2;
        const int64_t row_bytes = p.ldy * es, row0 = (int64_t)row_tile * TILE_N + 32 * q;
        const int rows = (int)max((int64_t)0, min((int64_t)32, p.w.n - row0)); // of this warp's 32
        char *const y0 = static_cast<char *>(p.y) + m0 * row_bytes + row0 * es;
        const uint32_t ru0 = smem_u32(s_ru), bias = p.bias ? smem_u32(s_bias) + 128 * q : 0u;
        const int h0 = NACC == 2 ? mt : min(first_half<CG>(p.mt), mt);
        int c = 16 * half;
        bool first_given = NACC == 2; // the barrier of the accumulator's first half of columns
        uint32_t v[16];
        if (c < mt) tmem_ld16(lane_addr + c, v);
        while (c < mt) {
          const int next = c + 16 * (EPI_WARPS / 4), r0 = row_of_column<CG>(c, mt), cols = (int)(m_end - m0) - r0; // (cols: none of a pair's may be left)
          const uint32_t ru = ru0 + (uint32_t)c * 4;
          char *const yp = y0 + r0 * row_bytes;
          tmem_ld_wait();
          if (!first_given && next >= h0) { // this warp has read all it needs of the first half: its columns may be overwritten
            first_given = true;
            give_back(acc_empty);
          }
          if (next >= mt) give_back(acc_empty + 8 * (NACC == 2 ? buf : 1));
          if (p.vec_out) {
#pragma unroll
            for (int j = 0; j < 16; j++) sts32(slot + (uint32_t)(j * 128) + ((uint32_t)(lane * 4) ^ ((j & 1) << 4)), v[j]);
            if (next < mt) tmem_ld16(lane_addr + next, v); // arrives while the chunk is stored
            __syncwarp();
            if (f32) {
              if (ticket == 0) store_turned<STORE_F32>(slot, ru, bias, yp, row_bytes, cols, rows, lane);
              else store_turned<ADD_F32>(slot, ru, bias, yp, row_bytes, cols, rows, lane);
            } else if (p.y_dtype == XNQ_F16) {
              store_turned<STORE_F16>(slot, ru, bias, yp, row_bytes, cols, rows, lane);
            } else {
              store_turned<STORE_BF16>(slot, ru, bias, yp, row_bytes, cols, rows, lane);
            }
            __syncwarp();
          } else {
            const bool row_ok = lane < rows;
            if (f32) {
              if (ticket == 0) store_direct<STORE_F32>(v, ru, bias, yp, row_bytes, cols, row_ok, lane);
              else store_direct<ADD_F32>(v, ru, bias, yp, row_bytes, cols, row_ok, lane);
            } else if (p.y_dtype == XNQ_F16) {
              store_direct<STORE_F16>(v, ru, bias, yp, row_bytes, cols, row_ok, lane);
            } else {
              store_direct<STORE_BF16>(v, ru, bias, yp, row_bytes, cols, row_ok, lane);
            }
            if (next < mt) tmem_ld16(lane_addr + next, v);
          }
          c = next;
        }
        // a warp that had no chunk (16 columns, the second warp of a quarter)
        if (16 * half >= mt) {
          if (NACC == 1) give_back(acc_empty);
          give_back(acc_empty + 8 * (NACC == 2 ? buf : 1));
        }
      }
      if (!whole && alive) {
        if (ticket == 0) __threadfence();
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
        if (ticket == 0 && et == 0) {
          unsigned int *flag = p.tile_cnt + (size_t)p.row_tiles * TM + tile;
          asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(1u) : "memory");
        }
      }
      i += len;
      cur.advance(len, KT, TM);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync(); // nothing of the pair reaches for this CTA's barriers or tensor memory any more
  if (warp == LOADER_WARP) tmem_dealloc<CG>(tmem_d, 512);
}

// ---- activation image -----------------------------------------------------------------------------------
// Stored order inside a k-step: Q8_0 and Q6_K natural. Q4_0 and Q4_K store pairs of 4-element runs that lie 16 (Q4_0) or 32
// (Q4_K) elements apart as one 8-element chunk [j, j+2, f+j, f+j+2, j+1, j+3, f+j+1, f+j+3], f = 16 or 32: the order the nibble
// unpack produces. A thread holds 8 consecutive elements (two such runs) and its partner, 2 or 4 lanes away, the other two.
__device__ __forceinline__ int kpair_shift(int wdtype) { return wdtype == XNQ_Q4_0 ? 2 : (wdtype == XNQ_Q4K ? 4 : 0); }
__device__ __forceinline__ uint32_t pack_h2(__half a, __half b) { return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16); }

// One CTA per activation row: Q8 quantize (the reference's activation blocks), dequantize, scale the row
// by a power of two so its largest magnitude lands in [2^11, 2^12), store fp16 into the swizzled image.
template <int ACT, typename XT>
__global__ void __launch_bounds__(256) prefill_prepare_acts(const XT *__restrict__ x, int64_t m, int64_t k, int64_t ldx, int64_t m_pad, int ksteps,
                                                            int wdtype, float wscale, uint8_t *__restrict__ xh, float *__restrict__ row_unscale,
                                                            unsigned int *__restrict__ tile_cnt, int tile_words) {
  __shared__ float red[8];
  pdl_launch_dependents(); // the matmul kernel may set itself up and request its first weights now
  pdl_wait();              // x may be the previous kernel's output; the scratch may still be read by the previous call
  const int64_t row = blockIdx.x;
  if (blockIdx.x == 0) // the persistent kernel's per-tile tickets and flags start every call at zero
    for (int i = threadIdx.x; i < tile_words; i += blockDim.x) tile_cnt[i] = 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t per_row = (int64_t)ksteps * 8; // 8-element groups in the padded row
  __half *img = reinterpret_cast<__half *>(xh);
  if (row >= m) { // padding rows: zeros
    for (int64_t t = threadIdx.x; t < per_row; t += blockDim.x) {
      const int64_t kt = t >> 3;
      *reinterpret_cast<uint4 *>(img + (kt * m_pad + row) * 64 + (t & 7) * 8) = make_uint4(0, 0, 0, 0);
    }
    if (threadIdx.x == 0) row_unscale[row] = 0.f;
    return;
  }
  const XT *xr = x + row * ldx;
  // pass 1: row maximum of the QUANTIZED-then-dequantized values is bounded by the raw maximum (codes <= 128/127 of it)
  float amax = 0.f;
  for (int64_t t = threadIdx.x; t < k / 8; t += blockDim.x) {
    float v[8];
    load8(xr + t * 8, v);
#pragma unroll
    for (int i = 0; i < 8; i++) amax = fmaxf(amax, fabsf(v[i]));
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  if (lane == 0) red[warp] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int i = 1; i < 8; i++) amax = fmaxf(amax, red[i]);
  // power of two s with amax * s in [2^10, 2^11): room for the 128/127 growth of the Q8_K codes
  int e = 0;
  if (amax > 0.f && amax < 3.0e38f) {
    (void)frexpf(amax, &e); // amax = f * 2^e, f in [0.5, 1)
  }
  const float rscale = amax > 0.f ? ldexpf(1.f, 11 - e) : 1.f;
  if (threadIdx.x == 0) row_unscale[row] = 1.f / (rscale * wscale); // exact: powers of two
  // pass 2: quantize per block, dequantize, scale, store. Whole warps stay together for the shuffles.
  const int64_t groups = k / 8;
  for (int64_t base = 0; base < per_row; base += blockDim.x) {
    const int64_t t = base + threadIdx.x;
    const bool valid = t < groups;
    float v[8];
    if (valid) load8(xr + t * 8, v);
    else {
#pragma unroll
      for (int i = 0; i < 8; i++) v[i] = 0.f;
    }
    const Quant8 q = ACT == XNQ_Q8_0 ? quantize8_q8_0(v, lane) : quantize8_q8k(v, lane);
    const float ds = q.d * rscale; // exact unless it leaves the normal range
    __half h[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int code = (int)(int8_t)(((i < 4 ? q.lo : q.hi) >> (8 * (i & 3))) & 0xff);
      h[i] = __float2half_rn(valid ? (float)code * ds : 0.f);
    }
    const int ps = kpair_shift(wdtype);
    uint4 out;
    int chunk = (int)(t & 7);
    if (ps == 0) {
      out = make_uint4(pack_h2(h[0], h[1]), pack_h2(h[2], h[3]), pack_h2(h[4], h[5]), pack_h2(h[6], h[7]));
    } else { // runs A (elements 0..3) and B (4..7): the lower thread of a pair stores both threads' runs A, the upper one their runs B
      const bool upper = (t & ps) != 0;
      const uint32_t a02 = pack_h2(h[0], h[2]), a13 = pack_h2(h[1], h[3]), b02 = pack_h2(h[4], h[6]), b13 = pack_h2(h[5], h[7]);
      const uint32_t g0 = __shfl_xor_sync(0xffffffffu, upper ? a02 : b02, ps), g1 = __shfl_xor_sync(0xffffffffu, upper ? a13 : b13, ps);
      out = upper ? make_uint4(g0, b02, g1, b13) : make_uint4(a02, g0, a13, g1);
      // Q4_0: block b = t >> 2, run pair (t & 1); Q4_K: run pair (t & 3)
      chunk = ps == 2 ? ((chunk >> 2) * 4 + (chunk & 1) * 2 + (upper ? 1 : 0)) : ((chunk & 3) * 2 + (upper ? 1 : 0));
    }
    if (t >= per_row) continue;
    *reinterpret_cast<uint4 *>(img + ((t >> 3) * m_pad + row) * 64 + ((chunk ^ (int)(row & 7)) << 3)) = out;
  }
}

int g_num_sms = 0, g_num_pairs = 0;

void pair_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute (&attr)[2], unsigned ctas, int threads, size_t smem, cudaStream_t s) {
  cfg->gridDim = dim3(ctas);
  cfg->blockDim = dim3(threads);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = s;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2, attr[1].val.clusterDim.y = 1, attr[1].val.clusterDim.z = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 2;
}
// ctas: CTAs, or pairs of them
template <typename RowT>
int launch_persistent_fmt(const PrefillArgs &a, bool pairs, unsigned ctas, size_t smem, cudaStream_t s) {
  if (pairs) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    pair_config(&cfg, attr, 2 * ctas, NTHREADS, smem, s);
    XNQ_CUDA(cudaLaunchKernelEx(&cfg, prefill_persistent_kernel<RowT, 2>, a, a.w.maps->codes, a.w.maps->high));
  } else {
    XNQ_CUDA(launch_pdl(prefill_persistent_kernel<RowT, 1>, dim3(ctas), dim3(NTHREADS), smem, s, a, a.w.maps->codes, a.w.maps->high));
  }
  count_launch();
  return XNQ_OK;
}

constexpr size_t SM_SMEM = 228 * 1024, MAX_SPREAD = SM_SMEM / 2;
static_assert(RowQ4_0::SLOT == RowQ4K::SLOT && RowQ8_0::SLOT == RowQ4K::SLOT, "the raw ring's plan assumes one slot size for these");
constexpr size_t PREFILL_SMEM = 225 * 1024; // everything an SM offers minus the static barriers and a reserve

// Shared-memory plan: B ring | raw ring | the drain warps' chunks. With up to eight stages a producer warp can be a whole super-step ahead of the MMAs;
// what is left goes to the raw ring (it covers the memory latency of the weights).
constexpr uint32_t b_stride_of(int rows) { return ((uint32_t)rows * 128 + 1023) & ~1023u; }
struct SmemPlan {
  int nstages, raw_slots;
};
constexpr SmemPlan smem_plan(int rows, uint32_t slot) { // rows: a CTA's activation rows of a tile; slot: bytes of a raw super-step
  const size_t budget = PREFILL_SMEM - 1024 - EPI_WARPS * EPI_SLOT, stride = b_stride_of(rows); // 1024: alignment slack
  SmemPlan p{0, 0};
  for (int raw = 3; raw >= 2 && p.nstages < MIN_STAGES; raw--) // at least so many raw slots
    p.nstages = (int)std::min<size_t>(MAX_STAGES, (budget - raw * slot) / stride);
  p.raw_slots = (int)std::min<size_t>(MAX_RAW_SLOTS, (budget - p.nstages * stride) / slot);
  return p;
}
constexpr bool plan_is(int rows, uint32_t slot, int stages, int slots) { return smem_plan(rows, slot).nstages == stages && smem_plan(rows, slot).raw_slots == slots; }
static_assert(plan_is(256, RowQ4K::SLOT, 4, 4) && plan_is(256, RowQ6K::SLOT, 4, 2), "a wide tile of one CTA: four stages");
static_assert(plan_is(128, RowQ4K::SLOT, 8, 4) && plan_is(128, RowQ6K::SLOT, 7, 3), "and half of it, of a pair's CTA");

template <typename RowT>
int init_fmt(int *pairs) { // pairs: lowered to what the device holds at a time of this kernel (0: not set yet)
  XNQ_CUDA(cudaFuncSetAttribute(prefill_persistent_kernel<RowT, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PREFILL_SMEM));
  XNQ_CUDA(cudaFuncSetAttribute(prefill_persistent_kernel<RowT, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PREFILL_SMEM));
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  pair_config(&cfg, attr, 2, NTHREADS, PREFILL_SMEM, nullptr);
  int clusters = 0;
  XNQ_CUDA(cudaOccupancyMaxActiveClusters(&clusters, prefill_persistent_kernel<RowT, 2>, &cfg));
  clusters = std::min(clusters, g_num_sms / 2);
  *pairs = *pairs ? std::min(*pairs, clusters) : clusters;
  return XNQ_OK;
}

} // namespace

static size_t tile_words(int64_t m_pad, int64_t n) { // tickets + flags of the persistent kernel
  const size_t tiles = (size_t)((n + TILE_N - 1) / TILE_N) * (size_t)((m_pad + MAX_MT - 1) / MAX_MT);
  return (2 * tiles * 4 + 255) & ~(size_t)255;
}

size_t prefill_workspace_bytes(int64_t m, int64_t k, int64_t n) {
  const int64_t m_pad = (m + 15) / 16 * 16;
  const int64_t ksteps = (k + BK - 1) / BK;
  return (size_t)ksteps * m_pad * 128 + (((size_t)m_pad * 4 + 255) & ~(size_t)255) + tile_words(m_pad, n) + 256;
}

int launch_prefill(const WeightView &w, float wscale, const void *x, int x_dtype, int64_t m, int64_t ldx, void *y, int y_dtype, int64_t ldy,
                   void *workspace, cudaStream_t s, const void *bias) {
  const int64_t k = w.k;
  const int64_t m_pad = (m + 15) / 16 * 16;
  const int ksteps = (int)((k + BK - 1) / BK);
  float *row_unscale = static_cast<float *>(workspace);
  unsigned int *tile_cnt = reinterpret_cast<unsigned int *>(static_cast<uint8_t *>(workspace) + ((((size_t)m_pad * 4 + 255) & ~(size_t)255)));
  const size_t cnt_bytes = tile_words(m_pad, w.n);
  uint8_t *xh = reinterpret_cast<uint8_t *>(tile_cnt) + cnt_bytes;
  const int act = act_dtype_for(w.dtype);
  // The rows' CTAs are started while the previous kernel drains, and the first SM that is free would take eight of them (10 us for
  // 32 rows instead of 3); unused shared memory, half of the share that ceil(rows / SMs) of them would have, keeps them apart: one to an
  // SM up to as many rows as SMs, above that less than twice the even share.
  const int64_t sms = g_num_sms > 0 ? g_num_sms : 148;
  const size_t spread = SM_SMEM / (size_t)((m_pad + sms - 1) / sms) / 2048 * 1024; // (each CTA also takes 1 KB of its own)
#define XNQ_PREP(ACT, XT)                                                                                                   \
  XNQ_CUDA(launch_pdl(prefill_prepare_acts<ACT, XT>, dim3((unsigned)m_pad), dim3(256), spread, s, static_cast<const XT *>(x), m, k, ldx, m_pad, ksteps, \
                      w.dtype, wscale, xh, row_unscale, tile_cnt, (int)(cnt_bytes / 4)))
  if (act == XNQ_Q8_0) {
    if (x_dtype == XNQ_F32) XNQ_PREP(XNQ_Q8_0, float);
    else if (x_dtype == XNQ_F16) XNQ_PREP(XNQ_Q8_0, __half);
    else XNQ_PREP(XNQ_Q8_0, __nv_bfloat16);
  } else {
    if (x_dtype == XNQ_F32) XNQ_PREP(XNQ_Q8K, float);
    else if (x_dtype == XNQ_F16) XNQ_PREP(XNQ_Q8K, __half);
    else XNQ_PREP(XNQ_Q8K, __nv_bfloat16);
  }
#undef XNQ_PREP
  count_launch();

  PrefillArgs a{};
  a.w = w;
  a.xh = xh;
  a.row_unscale = row_unscale;
  a.y = y;
  a.bias = bias;
  a.y_dtype = y_dtype;
  a.ldy = ldy;
  a.m = m;
  a.m_pad = m_pad;
  a.ksteps = ksteps;
  const int row_tiles = (int)((w.n + TILE_N - 1) / TILE_N);
  a.tiles_m = (int)((m_pad + MAX_MT - 1) / MAX_MT);
  a.whole_tiles = y_dtype == XNQ_F32 ? 0 : 1;
  // 16-bit results, whose tiles are whole: equal tiles of activation rows, in the MMA's steps of 16 columns (pairs: 32, 16 of each CTA), as many as
  // finish first: rounds of the CTAs times a tile's time. Measured for one round (18944 x 1024 and 4096; Q4_K, Q8_0 and Q6_K alike), a k-step takes
  // the same up to 128 rows (what bounds it is the conversion of the weights) and then a 256th more for every further row: 66 rows 0.277 us, 128
  // 0.290, 192 0.374, 256 0.423; a tile's start and end take two k-steps and another for 64 rows. Where more than half of the SMs are
  // at work all of it takes 1.4 us longer: 4096 x 1024, 165 rows 9.8 us as two tiles on 64 CTAs, 11.3 as three on 96; 8912 x 1280, 165 rows 12.6 as one on
  // 70 CTAs, 13.3 as two on 140 (Q8_0 12.9 and 14.6); but 9060 x 4480, 138 rows 28.5 as one on 71, 27.1 as two on 142.
  // Pairs halve the activation operand's traffic, which is what bounds wide tiles: from 224 rows a tile on they are the faster or the equal
  // ones (in a long stream of calls, Q4_K 14336 x 4096: 224 rows 41.8 against 42.6 us, 512 rows 74.5 / 77.5, 1024 rows 128 / 139; but 176 rows
  // 39.0 / 37.0). With few tiles a pair's coarser share of the work costs more than that (Q4_K 1536 x 2048, 2000 rows, 21 k-steps a pair: 35.2 / 33.5).
  // f32 results: tiles of 256 rows on single CTAs. Where the CTAs' shares cut a tile decides the last bits of its sums, and a last bit that
  // differs in a decoder's first linear moves its logits by 3 % of their norm (8-bit activation codes flip).
  bool pairs = false;
  a.mt = (int)std::min<int64_t>(MAX_MT, m_pad);
  if (a.whole_tiles) {
    double best = 0, best_crowded = 0;
    const auto consider = [&](int mt, bool pair) {
      const long long tiles_m = (m_pad + mt - 1) / mt, ctas = pair ? g_num_pairs : sms, count = (pair ? (row_tiles + 1) / 2 : row_tiles) * tiles_m;
      const double crowded = std::min(count, ctas) * (pair ? 2 : 1) > sms / 2 ? 1300. : 0.;
      const double time = (double)((count + ctas - 1) / ctas) * (ksteps * (256. + std::max(0, mt - 128)) * (pair ? 0.95 : 1.) + 512. + 4. * mt) + crowded;
      // fewer and wider ones where it makes no difference (the 1.4 us are allowed for as they are)
      if (best == 0 || time < (crowded > best_crowded ? 1. : 0.98) * best) best = time, best_crowded = crowded, a.mt = mt, a.tiles_m = (int)tiles_m, pairs = pair;
    };
    const int64_t fewest = a.tiles_m;
    for (int64_t t = fewest, last = 0; t <= std::min(4 * fewest, fewest + 12); t++) {
      const int even_mt = (int)((m_pad + t - 1) / t), pair_mt = (even_mt + 31) / 32 * 32, mt = (even_mt + 15) / 16 * 16;
      if (mt == last) continue;
      last = mt;
      if (g_num_pairs > 0 && pair_mt >= 224 && (long long)((row_tiles + 1) / 2) * t * ksteps >= 24ll * g_num_pairs) consider(pair_mt, true);
      consider(mt, false);
    }
  }
  const int cg = pairs ? 2 : 1;
  const uint32_t slot = w.dtype == XNQ_Q6K ? RowQ6K::SLOT : RowQ4K::SLOT;
  a.b_stride = b_stride_of(a.mt / cg);
  const SmemPlan plan = smem_plan(a.mt / cg, slot);
  if (plan.nstages < MIN_STAGES) return fail(XNQ_ERR_SIZE, "prefill: shared-memory plan does not fit");
  a.nstages = plan.nstages;
  a.raw_slots = plan.raw_slots;
  a.raw_off = a.nstages * a.b_stride;
  a.epi_off = a.raw_off + a.raw_slots * slot;
  const size_t yes = type_size(y_dtype), piece = 16 / yes;
  a.vec_out = (reinterpret_cast<uintptr_t>(y) & 15) == 0 && ldy % piece == 0 && w.n % piece == 0;
  a.acc_bufs = a.mt <= 128 ? 2 : 1;
  a.wscale = wscale;
  a.row_tiles = row_tiles;
  a.tiles_n = (row_tiles + cg - 1) / cg;
  const long long tiles = (long long)a.tiles_n * a.tiles_m;
  a.units = tiles * ksteps;
  a.tile_cnt = tile_cnt;
  profile_mark(s, true);
  int rc;
  const long long want = a.whole_tiles ? tiles : std::max<long long>(1, a.units / 8); // at least 8 k-steps per CTA
  const unsigned ctas = (unsigned)std::min<long long>(pairs ? g_num_pairs : g_num_sms, want);
  // The bias of split tiles is added when their parts have met, so that its addition is the last one.
  const bool bias_after = bias && !a.whole_tiles && tiles % ctas != 0;
  if (bias_after) a.bias = nullptr;
  a.share_q = (a.whole_tiles ? tiles : a.units) / ctas, a.share_r = (int)((a.whole_tiles ? tiles : a.units) % ctas);
  switch (w.dtype) {
    case XNQ_Q4_0: rc = launch_persistent_fmt<RowQ4_0>(a, pairs, ctas, PREFILL_SMEM, s); break;
    case XNQ_Q8_0: rc = launch_persistent_fmt<RowQ8_0>(a, pairs, ctas, PREFILL_SMEM, s); break;
    case XNQ_Q4K: rc = launch_persistent_fmt<RowQ4K>(a, pairs, ctas, PREFILL_SMEM, s); break;
    case XNQ_Q6K: rc = launch_persistent_fmt<RowQ6K>(a, pairs, ctas, PREFILL_SMEM, s); break;
    default: rc = fail(XNQ_ERR_DTYPE, "prefill: dtype %d", w.dtype);
  }
  profile_mark(s, false);
  return rc == XNQ_OK && bias_after ? launch_add_bias(y, y_dtype, bias, m, w.n, ldy, s) : rc;
}

int prefill_init(int device) {
  cudaDeviceProp prop;
  XNQ_CUDA(cudaGetDeviceProperties(&prop, device));
  g_num_sms = prop.multiProcessorCount;
  // pairs that are resident together: the rule on the number of tiles counts rounds of them
  int pairs = 0, rc = XNQ_OK;
  if ((rc = init_fmt<RowQ4_0>(&pairs)) != XNQ_OK || (rc = init_fmt<RowQ8_0>(&pairs)) != XNQ_OK || (rc = init_fmt<RowQ4K>(&pairs)) != XNQ_OK ||
      (rc = init_fmt<RowQ6K>(&pairs)) != XNQ_OK)
    return rc;
  g_num_pairs = pairs;
#define XNQ_PREP_INIT(ACT, XT) XNQ_CUDA(cudaFuncSetAttribute(prefill_prepare_acts<ACT, XT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SPREAD))
  XNQ_PREP_INIT(XNQ_Q8_0, float);
  XNQ_PREP_INIT(XNQ_Q8_0, __half);
  XNQ_PREP_INIT(XNQ_Q8_0, __nv_bfloat16);
  XNQ_PREP_INIT(XNQ_Q8K, float);
  XNQ_PREP_INIT(XNQ_Q8K, __half);
  XNQ_PREP_INIT(XNQ_Q8K, __nv_bfloat16);
#undef XNQ_PREP_INIT
  unsigned int zero = 0;
  XNQ_CUDA(cudaMemcpyToSymbol(g_prefill_status, &zero, sizeof(zero)));
  return XNQ_OK;
}

int prefill_status(unsigned int *bits) {
  XNQ_CUDA(cudaMemcpyFromSymbol(bits, g_prefill_status, sizeof(*bits)));
  return XNQ_OK;
}

} // namespace xnq
