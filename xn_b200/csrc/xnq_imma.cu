// Small batches (2 <= m <= 64 activation rows per pass) on the 5th-generation tensor cores with exact
// integer arithmetic: tcgen05.mma.kind::i8, one tensor-memory accumulator slice per 32-element block.
//
// The reference's dots are exact integer sums over one 32-element (sub-)block, scaled in f32
// (k_quants.rs:287-304 Q4_0, 677-691 Q8_0, 1337-1416 Q4_K). One MMA
//
//     D[128 weight rows, NP activation rows] = A[128, 32] . B[NP, 32]^T          (s8 x s8 -> s32, no accumulation)
//
// is exactly those sums for 128 x NP (weight row, activation row) pairs and one block, so every MMA writes
// its own slice of tensor memory and the drain warps apply the block's scales to it in f32 exactly as the
// CPU code does: integer sub-block scales and mins for Q4_K (min term from the activations' 32-sums with
// dp4a), f16 block scale times f16-rounded activation scale for Q4_0 / Q8_0. Nothing is rounded before the
// f32 scaling, so results stay within the f32-accumulate bound (2e-3) at every batch size served.
//
// Q6_K (6 to 16 rows) has a scale per 16 elements, half an MMA's K. Its activation operand holds every row twice, once with the
// upper and once with the lower 16 of each 32 codes zeroed, so that one MMA yields both 16-sums; the drain multiplies the sixteen sums
// of a super-block with the int8 scales, adds them as integers and scales once, as the CPU code does (k_quants.rs:1743-1799).
//
// Roles of the 20 or 28 warps of a CTA (one CTA per SM, persistent):
//   activations (1) one elected thread requests, per 256-k step, the 1-D bulk copies of the quantized activations (already in
//                   the MMA's shared-memory layout) and of their per-block metadata into rings of stages guarded by
//                   mbarriers.
//   weights (1)     one elected thread requests a step's boxes of the weight's tensor maps (xnq_common.cuh), up to six steps ahead. Q8_0's
//                   codes arrive as the operand image the MMA reads.
//   converters (8)  two groups of four warps, one thread per weight row; the groups take alternate 256-k steps, so a step's
//                   chain of waits, loads, stores and fences has two steps' time to run in. They unpack the 4- and 6-bit codes of a raw stage
//                   to int8 into the 128-byte-swizzled K-major operand image, and hand the rows' scale bytes on to the drain.
//                   (Until the boxes, every warp copied its 32 rows with 16-byte cp.async and the CTA asked its share of the weight into
//                   L2 first: a third of all instructions, and 17 to 24 cycles a copy instruction whatever was done, 16 to 30 bytes a cycle.
//                   With the boxes, in a stream of calls: Q8_0 11008 x 4096, 45 rows 30.9 -> 26.4 us, 16 rows 21.4 -> 18.8; Q4_K 28672 x 4096, 16 rows
//                   34.0 -> 30.5; 14336 x 4096, 64 rows 36.6 -> 34.7; Q6_K 32000 x 4096, 16 rows 46.5 -> 39.3. An earlier trial of boxes had the
//                   L2 requests queue in front of them in the same unit: 5000 cycles a box.)
//   MMA issuers (2) one warp per half step issues its four K = 32 MMAs into accumulator buffer h and commits them;
//   drain (16, or 8 with 16 activation rows) read the slices of a step back with tcgen05.ld, scale, and keep f32 sums in registers
//                   across the k steps of a tile; the warps of an accumulator lane quarter split the columns.
//
// Work is the flattened (tile of 128 weight rows, 256-k step) space, cut into equal contiguous ranges, one
// per CTA, so all SMs finish together however few tiles there are. A tile whose steps are split between
// CTAs is summed deterministically: every part is written to a scratch slot, an arrival ticket elects the
// last part, and that CTA adds the parts in k order and stores y.
//
// Every wait is bounded; on expiry a status bit is set and the roles fall through to the common exit, where
// tensor memory is released.
#include <algorithm>

#include "xnq_common.cuh"
#include "xnq_quantize_act.cuh"

namespace xnq {

__device__ unsigned int g_imma_status; // sticky: 1 producer, 2 converter, 4 mma, 8 drain wait expired
namespace {

constexpr int TILE_N = 128;         // weight rows per tile = UMMA M
constexpr int MAX_NP = 64;          // activation rows per pass = UMMA N (multiple of 16)
constexpr int CONV_WARPS = 8, DRAIN_WARPS = 16;
constexpr int ACT_PRODUCER_WARP = 0, MMA_WARP = 1, WEIGHT_PRODUCER_WARP = 3, CONV_WARP0 = 4, DRAIN_WARP0 = CONV_WARP0 + CONV_WARPS; // MMA issuers: warps 1 and 2
constexpr int A_STAGE_BYTES = TILE_N * 128; // one 128-k half step of int8 codes
constexpr int SIDE_STAGES = 8, MAX_B_STAGES = 8; // side stages are small (scale bytes and records of one step): enough of them that
                                                                   // the converters, which fill them, never wait for the drain, which frees them
constexpr int HDR_BYTES = TILE_N * 16;      // per 256-k step: 16 bytes of scale data per weight row
constexpr int TMEM_COLS = 512;              // all of the SM's tensor memory: 512 / (4 slices x NP) accumulator buffers, at most 8
constexpr size_t IMMA_SMEM = 226 * 1024, MAX_SPREAD = 120 * 1024;
constexpr int SCALE_SLOTS = 2;              // a converter warp's slots of scale bytes (Q4_0, Q8_0, Q6_K): copied that many of its steps ahead

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
// One wait attempt: the thread is suspended by the hardware until the phase completes or a system-chosen time limit
// passes (it takes no issue slots meanwhile, unlike a test_wait spin, which with two dozen polling warps per SM slowed
// the threads that issue copies and MMAs several times over).
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// the same with a suspend-time hint in nanoseconds: the hardware may keep the thread suspended that long before it
// returns false (a plain try_wait returned after a system-chosen, short time, and two dozen waiting warps per SM then
// spent a large share of the SM's issue slots re-issuing their waits: 60 % issue utilisation, a fifth of it in the
// unit that executes barrier instructions)
__device__ __forceinline__ bool mbar_test_hint(uint32_t bar, uint32_t parity, uint32_t ns) {
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
// bounded wait of one thread
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned int bit) {
  if (mbar_test(bar, parity)) return true;
  unsigned long long t0 = 0;
  for (unsigned int attempt = 1;; attempt++) { // the wall clock is read on every 16th failed attempt only
    if (mbar_test_hint(bar, parity, 1000000u)) return true;
    if ((attempt & 15u) == 0) {
      const unsigned long long now = wall_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > WAIT_LIMIT_NS) break;
    }
  }
  atomicOr(&g_imma_status, bit);
  return false;
}
// bounded wait of a whole warp (one instruction per attempt for all lanes); the result is the same in all lanes
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, unsigned int bit) {
  const bool ok = mbar_wait(bar, parity, bit);
  return __all_sync(0xffffffffu, ok);
}
// whether the phase has completed, without waiting for it
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
// a ticket of a tile: releases what the CTA stored before the barrier that precedes it, acquires what the others released
__device__ __forceinline__ unsigned int take_ticket(unsigned int *word) {
  unsigned int t;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(t) : "l"(word) : "memory");
  return t;
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
// a box of a tensor map: x in bytes (a multiple of 16), y the first row
__device__ __forceinline__ void tma_box(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
// 16-byte asynchronous copy global -> shared, bypassing L1; src_bytes 0 writes zeros instead (the address is not read)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_oldest() { asm volatile("cp.async.wait_group %0;" ::"n"(SCALE_SLOTS - 1) : "memory"); }
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
__device__ __forceinline__ void sts128(uint32_t addr, const uint4 &v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}


// ---- tcgen05 wrappers --------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// D = A . B^T (no accumulation: every MMA owns its accumulator slice)
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(0u)
      : "memory");
}
// arrives on the mbarrier once every MMA issued so far by this thread has finished reading smem / writing tmem
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[N]);
template <>
__device__ __forceinline__ void tmem_ld<4>(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld<8>(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// K-major, 128-byte-swizzled operand tile: rows of 128 bytes, 8-row groups 1024 bytes apart.
// Fields: start address >> 4 [0,14), leading byte offset >> 4 [16,30) (unused for swizzled K-major),
// stride byte offset >> 4 [32,46), descriptor version 1 [46,48), swizzle mode 2 = 128 B [61,64).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3ffffu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// kind::i8 instruction descriptor: D s32 (2 at [4,6)), A and B signed 8-bit (1 at [7,10) / [10,13)), both K-major,
// N >> 3 at [17,23), M >> 4 at [24,29).
__device__ __forceinline__ uint32_t idesc_i8(int umma_n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(umma_n >> 3) << 17) | ((uint32_t)(TILE_N >> 4) << 24);
}
__device__ __forceinline__ int dp4a_uu(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

struct ImmaArgs {
  WeightView w;
  const uint8_t *bimg; // quantized activations in operand layout: [half steps][NP rows x 128 bytes, 128-byte swizzle]
  const uint8_t *meta; // per 256-k step and activation row: 32 bytes of scales / sums (layout per format below)
  void *y;
  const void *bias;    // n values of y's type, or null
  int y_dtype;
  int64_t ldy;
  int64_t m;           // activation rows of this pass (<= NP)
  int nsteps;          // 256-k steps per tile
  int tiles;
  int units;           // tiles * nsteps
  int units_q, units_r; // CTA c works on units [c * units_q + min(c, units_r), + units_q + (c < units_r)): set at launch, so that
                        // no thread divides 64-bit numbers before its first copy
  unsigned int *tile_cnt; // [tiles] arrival tickets of split tiles, zeroed by the prepare kernel
  float *partials;        // [2 * grid][activation rows of the operand][128] partial sums of split tiles
  uint32_t step_x;        // bytes of one 256-k step of a row in the code stream
  // a row's 16 scale bytes of a step (Q4_0, Q8_0: eight f16 block scales, Q6_K: sixteen int8 ones; Q4_K has them in the code stream)
  const uint8_t *scales;
  uint32_t scale_row_bytes;
  int raw_stages, b_stages, a_stages;
  uint32_t b_stage_bytes, side_stage_bytes;
  uint32_t a_off, b_off, raw_off, side_off, scale_off; // offsets from the 1024-aligned base of dynamic shared memory
};

// the flattened (tile, step) space is cut into contiguous ranges: the first units_r CTAs take units_q + 1 units, the others units_q
__device__ __forceinline__ int cta_first_unit(int c, int q, int r) { return c * q + min(c, r); }
__device__ __forceinline__ int cta_of(int u, int q, int r) {
  const int big = r * (q + 1); // units held by the CTAs that take q + 1
  return u < big ? u / (q + 1) : r + (u - big) / q;
}

// ---- converters: raw bytes of (row, 64 of the step's 256 k) -> 64 bytes of int8 codes ------------------------
// A raw stage holds a step's boxes of the tile as the tensor maps lay them out (WeightMaps). raw: shared address of the stage; r: row in the
// tile; h: half step; p: which 64 k of the half step. Lanes read chunk c of their own rows: the swizzles and Q4_K's 144-byte rows spread
// a quarter warp's reads over all banks.
__device__ __forceinline__ uint4 chunk128(uint32_t raw, int r, int c) { return lds128(raw + (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4))); }
__device__ __forceinline__ uint4 chunk64(uint32_t raw, int r, int c) { return lds128(raw + (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4))); }
template <int CH>
struct DrainBlockScaled;
template <int CH>
struct DrainQ4K;
struct ConvQ8_0 { // the boxes are the MMA's operand as they are: they go straight to the operand stages
  static constexpr uint32_t RAW = 0;       // bytes of a raw stage
  static constexpr int SCALES = 512;       // bytes of scale data that a converter warp copies for a step
  static constexpr bool PAIRED = false;    // two operand columns per activation row
  template <int CH>
  using Drain = DrainBlockScaled<CH>;
};
__device__ __forceinline__ uint32_t nib_lo_s8(uint32_t w) { return (((w & 0x0f0f0f0fu) | 0x80808080u) - 0x08080808u) ^ 0x80808080u; } // code - 8 per byte
__device__ __forceinline__ uint32_t nib_hi_s8(uint32_t w) { return ((((w >> 4) & 0x0f0f0f0fu) | 0x80808080u) - 0x08080808u) ^ 0x80808080u; }
struct ConvQ4_0 { // eight blocks of 16 nibble bytes per row and step; element j < 16 low nibble of byte j, j >= 16 high nibble of byte j - 16
  static constexpr uint32_t RAW = TILE_N * 128;
  static constexpr int SCALES = 512;
  static constexpr bool PAIRED = false;
  template <int CH>
  using Drain = DrainBlockScaled<CH>;
  __device__ static __forceinline__ void run(uint32_t raw, int r, int h, int p, uint4 (&out)[4]) {
#pragma unroll
    for (int bb = 0; bb < 2; bb++) {
      const uint4 q = chunk128(raw, r, 4 * h + 2 * p + bb);
      out[2 * bb] = make_uint4(nib_lo_s8(q.x), nib_lo_s8(q.y), nib_lo_s8(q.z), nib_lo_s8(q.w));
      out[2 * bb + 1] = make_uint4(nib_hi_s8(q.x), nib_hi_s8(q.y), nib_hi_s8(q.z), nib_hi_s8(q.w));
    }
  }
};
struct ConvQ4K { // super-blocks: 16 header bytes, then four 32-byte chunks; chunk c = sub-block 2c in the low nibbles, 2c+1 in the high ones
  static constexpr uint32_t RAW = TILE_N * 144;
  static constexpr int SCALES = 0;
  static constexpr bool PAIRED = false;
  template <int CH>
  using Drain = DrainQ4K<CH>;
  __device__ static __forceinline__ void run(uint32_t raw, int r, int h, int p, uint4 (&out)[4]) {
    const uint32_t at = raw + (uint32_t)(r * 144 + 16 + 32 * (2 * h + p));
    const uint4 a = lds128(at), b = lds128(at + 16);
    out[0] = make_uint4(a.x & 0x0f0f0f0fu, a.y & 0x0f0f0f0fu, a.z & 0x0f0f0f0fu, a.w & 0x0f0f0f0fu);
    out[1] = make_uint4(b.x & 0x0f0f0f0fu, b.y & 0x0f0f0f0fu, b.z & 0x0f0f0f0fu, b.w & 0x0f0f0f0fu);
    out[2] = make_uint4((a.x >> 4) & 0x0f0f0f0fu, (a.y >> 4) & 0x0f0f0f0fu, (a.z >> 4) & 0x0f0f0f0fu, (a.w >> 4) & 0x0f0f0f0fu);
    out[3] = make_uint4((b.x >> 4) & 0x0f0f0f0fu, (b.y >> 4) & 0x0f0f0f0fu, (b.z >> 4) & 0x0f0f0f0fu, (b.w >> 4) & 0x0f0f0f0fu);
  }
};

__device__ __forceinline__ uint32_t q6_code(uint32_t ql, int sh, uint32_t qh, int hsh) { // four 6-bit codes - 32 as int8
  const uint32_t c = ((ql >> sh) & 0x0f0f0f0fu) | (((qh >> hsh) & 0x03030303u) << 4);
  return ((c | 0x80808080u) - 0x20202020u) ^ 0x80808080u;
}
struct ConvQ6K { // 128 ql bytes, behind the rows' 64 qh bytes. 64 k number 2 h + p: the two 32-element groups 2 p, 2 p + 1 of half h
  static constexpr uint32_t RAW = TILE_N * 192;
  static constexpr int SCALES = 1024;      // and the 16 bytes that hold the super-block's f16 d
  static constexpr bool PAIRED = true;
  __device__ static __forceinline__ void run(uint32_t raw, int r, int h, int p, uint4 (&out)[4]) {
    const uint32_t hi = raw + TILE_N * 128;
#pragma unroll
    for (int half = 0; half < 2; half++) { // elements 0..15 and 16..31 of the groups
      const uint4 a = chunk128(raw, r, 4 * h + half), b = chunk128(raw, r, 4 * h + 2 + half), q = chunk64(hi, r, 2 * h + half);
      const int sh = 4 * p, h0 = 4 * p, h1 = 4 * p + 2; // groups 0, 1: low nibbles of ql[l], ql[l + 32]; groups 2, 3: the high nibbles
      out[half] = make_uint4(q6_code(a.x, sh, q.x, h0), q6_code(a.y, sh, q.y, h0), q6_code(a.z, sh, q.z, h0), q6_code(a.w, sh, q.w, h0));
      out[2 + half] = make_uint4(q6_code(b.x, sh, q.x, h1), q6_code(b.y, sh, q.y, h1), q6_code(b.z, sh, q.z, h1), q6_code(b.w, sh, q.w, h1));
    }
  }
};

// ---- drain: scale the eight slices of a step and add them to the running sums --------------------------------
// hdr: the row's 16 scale bytes of the 256-k step; meta: shared address of the step's per-activation-row records
// (32 bytes each); v[j][c]: slice j (block j of the step), column c of this thread; c0: first column.
//   Q4_0 / Q8_0  hdr = eight f16 block scales; record = eight f32 activation block scales
//   Q4_K         hdr = f16 d, f16 dmin, four 24-bit fields sc[2g] | sc[2g+1] << 6 | mn[2g] << 12 | mn[2g+1] << 18;
//                record = {lo(h=0), hi(h=0), lo(h=1), hi(h=1), f32 d, 0, 0, 0}: the 32-sums of the activation codes of
//                each half's four sub-blocks, s = 128 * hi + lo with lo in 0..127 (one byte each)
// The eight block terms of a step are added first, the step's sum then to the running sum: one rounding at the running sum's magnitude
// per step. One by one they made the results 7 to 20 % less exact than the two chains of half steps that were added before (relative
// error against the exact dot of the quantized operands, 1000 x 1024: 7.9e-8, with two chains 6.6e-8).
// Two columns to an instruction (f32x2): with 33 and more rows the drain's issue slots bound the kernel. Same operations in the same order.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
template <int CH>
struct DrainBlockScaled {
  // np: rows of the records, which are stored block by block
  __device__ static __forceinline__ void run(const uint4 &hdr, uint32_t meta, int np, int c0, const uint32_t (&v)[8][CH], float *acc) {
    const uint32_t w[4] = {hdr.x, hdr.y, hdr.z, hdr.w};
    uint64_t step[CH / 2];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const __half2 h = *reinterpret_cast<const __half2 *>(&w[j >> 1]);
      const float d = (j & 1) ? __high2float(h) : __low2float(h);
      const uint64_t d2 = pack2(d, d);
#pragma unroll
      for (int c = 0; c < CH; c += 4) {
        const uint4 a = lds128(meta + (uint32_t)(j * np + c0 + c) * 4);
        const uint64_t t0 = mul2(d2, pack2(__uint_as_float(a.x), __uint_as_float(a.y))), t1 = mul2(d2, pack2(__uint_as_float(a.z), __uint_as_float(a.w)));
        const uint64_t v0 = pack2((float)(int)v[j][c], (float)(int)v[j][c + 1]), v1 = pack2((float)(int)v[j][c + 2], (float)(int)v[j][c + 3]);
        step[c / 2] = j == 0 ? mul2(v0, t0) : fma2(v0, t0, step[c / 2]);
        step[c / 2 + 1] = j == 0 ? mul2(v1, t1) : fma2(v1, t1, step[c / 2 + 1]);
      }
    }
#pragma unroll
    for (int c = 0; c < CH; c += 2) {
      const uint64_t sum = add2(pack2(acc[c], acc[c + 1]), step[c / 2]);
      asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[c]), "=f"(acc[c + 1]) : "l"(sum));
    }
  }
};
template <int CH>
struct DrainQ4K { // integer sums over the whole super-block, scaled once, as the CPU code does
  __device__ static __forceinline__ void run(const uint4 &hdr, uint32_t meta, int, int c0, const uint32_t (&v)[8][CH], float *acc) {
    const __half2 dm = *reinterpret_cast<const __half2 *>(&hdr.x);
    const float d = __low2float(dm), dmin = __high2float(dm);
    const uint32_t F[4] = {hdr.y & 0xffffffu, __funnelshift_r(hdr.y, hdr.z, 24) & 0xffffffu, __funnelshift_r(hdr.z, hdr.w, 16) & 0xffffffu, hdr.w >> 8};
    const uint32_t mins0 = ((F[0] >> 12) & 63u) | (((F[0] >> 18) & 63u) << 8) | (((F[1] >> 12) & 63u) << 16) | (((F[1] >> 18) & 63u) << 24);
    const uint32_t mins1 = ((F[2] >> 12) & 63u) | (((F[2] >> 18) & 63u) << 8) | (((F[3] >> 12) & 63u) << 16) | (((F[3] >> 18) & 63u) << 24);
#pragma unroll
    for (int c = 0; c < CH; c++) {
      const uint32_t rec = meta + (uint32_t)(c0 + c) * 32;
      const uint4 bs = lds128(rec);
      const float da = __uint_as_float(lds32(rec + 16));
      int isum = 0;
#pragma unroll
      for (int j = 0; j < 8; j++) isum += (int)((F[j >> 1] >> (6 * (j & 1))) & 63u) * (int)v[j][c];
      const int msum = dp4a_uu(mins0, bs.x, dp4a_uu(mins1, bs.z, 0)) + 128 * dp4a_us(mins0, bs.y, dp4a_us(mins1, bs.w, 0));
      acc[c] += da * (d * (float)isum - dmin * (float)msum);
    }
  }
};

// Q6_K, the four slices of half step h: v[2 j + u][c] is the sum of the u-th 16 elements of block j. hdr: the row's sixteen int8 scales.
template <int CH>
__device__ __forceinline__ void q6k_sums(const uint4 &hdr, int h, const uint32_t (&v)[8][CH], int (&isum)[CH]) {
  const uint32_t w[2] = {h ? hdr.z : hdr.x, h ? hdr.w : hdr.y};
#pragma unroll
  for (int c = 0; c < CH; c++)
#pragma unroll
    for (int j = 0; j < 8; j++) isum[c] += (int)(int8_t)((w[j >> 2] >> (8 * (j & 3))) & 0xffu) * (int)v[j][c];
}

// Long f32 chains are cut: after SUM_RUN terms the chain's sum goes to a second one. Q6_K's steps (a CTA may add all of a long row's:
// 14336 / 256 = 56) and, with 16 rows, the parts of a tile. (Q6_K, 600 x 14336: 1.06e-7 from the exact dot in one chain; the dp4a kernel, whose
// 32 lanes take a part each, 8.3e-8. Wider operands add their parts in one chain, as they did before their drain took whole steps: with
// runs, in 72 registers, the loop over the parts of 600 x 14336 took 44 us instead of 29 at 64 rows.)
constexpr int SUM_RUN = 8;

// Drain warps: a warp's waits and its decoding of the row's scales cost as much as four columns' arithmetic; with 16 rows eight warps of
// eight columns each do better than sixteen of four (Q6_K 32000 x 4096, 16 rows: 48.5 -> 46.4 us; Q8_0 11008 x 4096, 8 rows: 21.7 -> 20.9).
__host__ __device__ constexpr int drain_warps(int rows) { return rows == 16 ? 8 : DRAIN_WARPS; }
__host__ __device__ constexpr int imma_threads(int rows) { return (DRAIN_WARP0 + drain_warps(rows)) * 32; }

// BIAS: a variant of its own (one kernel with a test of p.bias took 22.1 instead of 21.4 us for Q4_K 4096 x 14336, 16 rows without a bias).
template <typename Conv, int NP, bool BIAS>
__global__ void __launch_bounds__(imma_threads(Conv::PAIRED ? NP / 2 : NP), 1) imma_kernel(const __grid_constant__ ImmaArgs p, const __grid_constant__ CUtensorMap codes, const __grid_constant__ CUtensorMap high) {
  constexpr int ROWS = Conv::PAIRED ? NP / 2 : NP; // activation rows of the operand; NP: its columns
  constexpr int DW = drain_warps(ROWS);
  constexpr int NPT = ROWS / (DW / 4); // rows per drain thread: the warps of an accumulator lane quarter split them
  constexpr int CH = DW == 8 ? 8 : 4;  // columns read back at a time, all eight slices of a step: what the register budget holds
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u; // operand stages need 1024-byte alignment
  constexpr int NBUF = TMEM_COLS / (8 * NP) > 4 ? 8 : TMEM_COLS / (8 * NP) * 2; // accumulator buffers (even: buffer parity = half step parity)
  constexpr int BUF_COLS = 4 * NP;
  // barriers: b_full/b_empty [8], side_full/side_empty [8], a_full/mma_done [8], acc_empty [8], raw_full/raw_empty [8]
  __shared__ __align__(8) uint64_t bars[72];
  __shared__ uint32_t tmem_slot;
  __shared__ unsigned int s_ticket[2];
  const uint32_t b_full = smem_u32(bars), b_empty = b_full + 64, side_full = b_full + 128, side_empty = b_full + 192, a_full = b_full + 256,
                 mma_done = b_full + 320, acc_empty = b_full + 384, raw_full = b_full + 448, raw_empty = b_full + 512;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31; // so that the compiler knows `warp` to be uniform
  const int RS = p.raw_stages, BS = p.b_stages, AS = p.a_stages, AP = AS / 2; // AP: operand stages in whole steps
  const int NB = min(NBUF, AS); // accumulator buffers in use: a drain group waiting on mma_done must not be lapped by the MMA thread,
                                // which can run ahead by NB half steps, so the ring of mma_done barriers (AS) is at least that long
  const int KT = p.nsteps;
  const int u0 = cta_first_unit((int)blockIdx.x, p.units_q, p.units_r);
  const int nunits = p.units_q + ((int)blockIdx.x < p.units_r ? 1 : 0);
  const int tile0 = u0 / KT, kt0 = u0 - tile0 * KT;
  const bool first_part = kt0 != 0 && nunits > KT - kt0; // the CTA's range starts inside a tile and goes on after it

  if (threadIdx.x == 0) {
    for (int s = 0; s < 8; s++) {
      mbar_init(a_full + 8 * s, Conv::RAW ? CONV_WARPS / 2 : 1); // the four converter warps of the step's group (one barrier per step: entries 0 .. AP - 1); Q8_0: the boxes
      mbar_init(mma_done + 8 * s, 1);            // the half step's MMAs have read their operands and written their slices
      mbar_init(acc_empty + 8 * s, DW);
      mbar_init(side_full + 8 * s, 1 + CONV_WARPS / 2); // the producer's transaction + the four converter warps that copy the scale bytes
      mbar_init(side_empty + 8 * s, DW);
      mbar_init(b_full + 8 * s, 1);
      mbar_init(b_empty + 8 * s, 2); // both half steps' MMAs
      mbar_init(raw_full + 8 * s, 1);
      mbar_init(raw_empty + 8 * s, CONV_WARPS / 2);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) { // one warp owns the tensor-memory allocation
    tmem_alloc(smem_u32(&tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents(); // the next kernel in the stream may be set up while this one runs
  const uint32_t tmem_d = __shfl_sync(0xffffffffu, tmem_slot, 0);

  if (warp == ACT_PRODUCER_WARP) {
    // ---- activation producer: per 256-k step the activations' operand image and their records. The whole warp runs the loop and
    // one elected lane issues (see the MMA issuers). ----
    pdl_wait();
    bool alive = true;
    int kt = kt0, bs = 0;
    uint32_t b_ph = 0; // (i / BS) & 1
    for (int i = 0; i < nunits; i++) {
      const int ss = i % SIDE_STAGES;
      if (alive && i >= BS) alive = mbar_wait(b_empty + 8 * bs, b_ph ^ 1u, 1u);
      if (alive && i >= SIDE_STAGES) alive = mbar_wait(side_empty + 8 * ss, ((i / SIDE_STAGES) - 1) & 1, 1u);
      __syncwarp();
      if (elect_one() && alive) {
        mbar_expect_tx(b_full + 8 * bs, p.b_stage_bytes);
        mbar_expect_tx(side_full + 8 * ss, (uint32_t)NP * 32u);
        bulk_g2s(base + p.b_off + bs * p.b_stage_bytes, p.bimg + ((size_t)kt * 2) * (NP * 128), p.b_stage_bytes, b_full + 8 * bs);
        bulk_g2s(base + p.side_off + ss * p.side_stage_bytes + HDR_BYTES, p.meta + (size_t)kt * (NP * 32), (uint32_t)NP * 32u, side_full + 8 * ss);
      }
      __syncwarp();
      if (++kt == KT) kt = 0;
      if (++bs == BS) bs = 0, b_ph ^= 1u;
    }
  } else if (warp == MMA_WARP || warp == MMA_WARP + 1) {
    // ---- MMA issuers: one warp per half step. The whole warp runs the loop and one elected lane issues; everything that decides the
    // loop's course or a descriptor is a function of launch parameters and counters (a wait that gave up only makes the rest of the
    // loop idle), so the compiler keeps the descriptors in uniform registers. In a branch on the lane number they were moved there
    // from vector registers, one after the other, which held the thread for 96 cycles per MMA; the tensor core takes one every 40
    // (NP <= 32) or 48 (NP = 64) cycles. ----
    const int h = warp - MMA_WARP;
    const uint32_t idesc = idesc_i8(NP);
    bool alive = true;
    int ap = 0, bs = 0, nb = 0; // i % AP, i % BS, i % (NB / 2): half step j = 2 i + h uses A stage 2 ap + h and buffer 2 nb + h
    uint32_t a_ph = 0, b_ph = 0, acc_ph = 0; // the parities of the laps
    for (int i = 0; i < nunits; i++) {
      const int sa = 2 * ap + h, buf = 2 * nb + h;
      if (alive) alive = mbar_wait(b_full + 8 * bs, b_ph, 4u);
      if (alive) alive = mbar_wait(a_full + 8 * ap, a_ph, 4u); // both halves of the step's operand image
      if (alive && 2 * i >= NB) alive = mbar_wait(acc_empty + 8 * buf, acc_ph ^ 1u, 4u); // the drain of the buffer's previous half step
      tc_fence_after();
      __syncwarp();
      const uint64_t adesc = smem_desc_sw128(base + p.a_off + sa * A_STAGE_BYTES);
      const uint64_t bdesc = smem_desc_sw128(base + p.b_off + bs * p.b_stage_bytes + h * (NP * 128));
      if (elect_one() && alive) {
#pragma unroll
        for (int q = 0; q < 4; q++) // K = 32 per instruction: advance 32 bytes inside the swizzle row; slice q of the buffer
          umma_i8(tmem_d + (uint32_t)(buf * BUF_COLS + q * NP), adesc + (uint64_t)(q * 2), bdesc + (uint64_t)(q * 2), idesc);
        umma_commit(mma_done + 8 * sa); // serves the drain (the slices are written) and, with the other half's, the converters (the stages are free)
        umma_commit(b_empty + 8 * bs);
      }
      __syncwarp();
      if (++ap == AP) ap = 0, a_ph ^= 1u;
      if (++bs == BS) bs = 0, b_ph ^= 1u;
      if (2 * ++nb == NB) nb = 0, acc_ph ^= 1u;
    }
  } else if (warp == WEIGHT_PRODUCER_WARP) {
    // ---- weight producer: the boxes of a step, as many steps ahead as there are stages (weights are immutable after upload: nothing here waits
    // for the kernel that prepares the activations). Q8_0's are the operand stages themselves, free again when both halves' MMAs are done. ----
    const int S = Conv::RAW ? RS : AP;
    int kt = kt0, tile = tile0, s = 0, issued = 0;
    uint32_t lap = 0; // (i / S) & 1
    bool alive = true;
    for (int i = 0; i < nunits && alive; i++) {
      if (i >= S) {
        if (Conv::RAW) alive = mbar_wait_warp(raw_empty + 8 * s, lap ^ 1u, 1u);
        else alive = mbar_wait_warp(mma_done + 8 * (2 * s), lap ^ 1u, 1u) && mbar_wait_warp(mma_done + 8 * (2 * s + 1), lap ^ 1u, 1u);
      }
      if (alive && elect_one()) {
        const int x = kt * (int)p.step_x, y = tile * TILE_N;
        if (Conv::RAW) {
          const uint32_t dst = base + p.raw_off + (uint32_t)s * Conv::RAW, bar = raw_full + 8 * s;
          mbar_expect_tx(bar, Conv::RAW);
          tma_box(dst, &codes, x, y, bar);
          if (Conv::PAIRED) tma_box(dst + TILE_N * 128, &high, x / 2, y, bar);
        } else {
          const uint32_t dst = base + p.a_off + (uint32_t)(2 * s) * A_STAGE_BYTES, bar = a_full + 8 * s;
          mbar_expect_tx(bar, 2 * A_STAGE_BYTES);
          tma_box(dst, &codes, x, y, bar);
          tma_box(dst + A_STAGE_BYTES, &codes, x + 128, y, bar);
        }
      }
      __syncwarp();
      if (alive) issued = i + 1;
      if (++kt == KT) kt = 0, tile++;
      if (++s == S) s = 0, lap ^= 1u;
    }
    if (first_part) { // a release takes about a microsecond, which stops a drain warp in the middle of the range; this warp is done with its own work
      asm volatile("bar.sync 2, %0;" ::"n"(DW * 32 + 32) : "memory");
      if (elect_one()) s_ticket[0] = take_ticket(p.tile_cnt + tile0);
      __syncwarp();
      asm volatile("bar.arrive 3, %0;" ::"n"(DW * 32 + 32) : "memory");
    }
    for (int i = max(0, issued - S); i < issued; i++) mbar_wait_warp((Conv::RAW ? raw_full : a_full) + 8 * (i % S), (i / S) & 1, 1u); // nothing in flight at exit
  } else if (warp < DRAIN_WARP0) {
    // ---- converters: group g (four warps, one thread per weight row) produces the steps i = g, g + 2, ... of this CTA: a
    // step's chain of waits, loads, stores and fences has the time of two steps' MMAs to run in ----
    const int cw = warp - CONV_WARP0;
    const int r = (cw & 3) * 32 + lane, g = cw >> 2;
    const int sw = r & 7;
    // the rows' scale bytes, SCALE_SLOTS of the warp's steps ahead, into slots of its own: lane l copies those of its row
    const uint32_t slot0 = base + p.scale_off + (uint32_t)(cw * SCALE_SLOTS * Conv::SCALES);
    int l_i = g, l_tile = tile0, l_kt = kt0 + g, l_s = 0;
    while (l_kt >= KT) l_kt -= KT, l_tile++;
    auto issue = [&]() {
      const int64_t grow = (int64_t)l_tile * TILE_N + r, at = min(grow, p.w.n - 1);
      const uint32_t dst = slot0 + (uint32_t)(l_s * Conv::SCALES) + lane * 16;
      const bool ok = grow < p.w.n && (uint32_t)l_kt * 16 + 16 <= p.scale_row_bytes;
      cp_async16(dst, p.scales + (size_t)at * p.scale_row_bytes + (ok ? (size_t)l_kt * 16 : 0), ok ? 16u : 0u);
      if constexpr (Conv::PAIRED) cp_async16(dst + 512, p.w.d + at * p.w.dstride + (l_kt & ~7), 16u);
      l_i += 2, l_kt += 2;
      while (l_kt >= KT) l_kt -= KT, l_tile++;
      if (++l_s == SCALE_SLOTS) l_s = 0;
    };
    if constexpr (Conv::SCALES > 0) {
      for (int u = 0; u < SCALE_SLOTS; u++) { // weights are immutable after upload: nothing here waits for the kernel that prepares the activations
        if (l_i < nunits) issue();
        cp_async_commit();
      }
    }
    bool alive = true;
    int ls = 0, rs = g % RS, bs = g % AP;
    uint32_t a_ph = (uint32_t)(g / AP) & 1u, raw_ph = (uint32_t)(g / RS) & 1u; // (i / AP) & 1, (i / RS) & 1
    for (int i = g; i < nunits && alive; i += 2) {
      const int ss = i % SIDE_STAGES;
      const uint32_t raw = base + p.raw_off + (uint32_t)rs * Conv::RAW;
      if constexpr (Conv::RAW > 0) alive = mbar_wait_warp(raw_full + 8 * rs, raw_ph, 2u);
      if (alive && i >= SIDE_STAGES) alive = mbar_wait_warp(side_empty + 8 * ss, ((i / SIDE_STAGES) - 1) & 1, 2u);
      if (!alive) break;
      { // hand the row's 16 scale bytes to the drain
        uint4 hv;
        if constexpr (Conv::SCALES > 0) {
          cp_async_wait_oldest(); // one group per step and lane, committed in step order: step i's has landed (a lane reads what it copied itself)
          const uint32_t slot = slot0 + (uint32_t)(ls * Conv::SCALES) + lane * 16;
          hv = lds128(slot);
          if constexpr (Conv::PAIRED) { // the super-block's d, widened, behind the records
            const int sb = (kt0 + i) % KT;
            const uint32_t dd = lds32(slot + 512 + 4 * ((sb >> 1) & 3));
            const float d = __half2float(__ushort_as_half((unsigned short)((sb & 1) ? (dd >> 16) : (dd & 0xffffu))));
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(base + p.side_off + ss * p.side_stage_bytes + HDR_BYTES + (uint32_t)(NP * 32) + (uint32_t)r * 4), "f"(d) : "memory");
          }
        } else {
          hv = lds128(raw + (uint32_t)(r * 144)); // the head of the Q4_K super-block
        }
        sts128(base + p.side_off + ss * p.side_stage_bytes + (uint32_t)r * 16, hv);
        __syncwarp();
        if (lane == 0) mbar_arrive(side_full + 8 * ss);
      }
      if constexpr (Conv::RAW > 0) {
        if (i >= AP) alive = mbar_wait_warp(mma_done + 8 * (2 * bs), a_ph ^ 1u, 2u) && mbar_wait_warp(mma_done + 8 * (2 * bs + 1), a_ph ^ 1u, 2u); // both halves of the stage have been multiplied
        if (!alive) break;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          uint4 lo[4], hi[4];
          Conv::run(raw, r, h, 0, lo);
          Conv::run(raw, r, h, 1, hi);
          const uint32_t dst_row = base + p.a_off + (2 * bs + h) * A_STAGE_BYTES + (uint32_t)r * 128;
#pragma unroll
          for (int c = 0; c < 4; c++) {
            sts128(dst_row + (uint32_t)((c ^ sw) << 4), lo[c]);
            sts128(dst_row + (uint32_t)(((4 + c) ^ sw) << 4), hi[c]);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic-proxy stores -> visible to the tensor core
        __syncwarp(); // every lane has stored its row and has read all it needs of the stage
        if (lane == 0) mbar_arrive(a_full + 8 * bs), mbar_arrive(raw_empty + 8 * rs);
        for (int t = 0; t < 2; t++) {
          if (++bs == AP) bs = 0, a_ph ^= 1u;
          if (++rs == RS) rs = 0, raw_ph ^= 1u;
        }
      }
      if constexpr (Conv::SCALES > 0) {
        if (l_i < nunits) issue(); // into the slot just read
        cp_async_commit();
        if (++ls == SCALE_SLOTS) ls = 0;
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory"); // nothing may be in flight into this CTA's shared memory when it exits
  } else {
    // ---- drain: warp quarter q reads accumulator lanes 32q.. (weight rows), the warps of a quarter split the columns; every warp
    // takes both half steps of every step and keeps f32 sums in registers. (Two groups of eight warps that took one half step each had
    // twice the columns per thread: at 64 rows they read them back four at a time, eight trips to tensor memory of 550 cycles per
    // half step; twice the integer-to-float conversions; and the groups' sums had to meet in memory at the end of a tile.) ----
    const int dwi = warp - DRAIN_WARP0;
    const int q = warp & 3, c0 = (dwi >> 2) * NPT;
    const int et = threadIdx.x - DRAIN_WARP0 * 32; // 0..511
    pdl_wait(); // the kernel that prepares the activations also zeroes the tiles' tickets
    bool alive = true;
    int tile = tile0, kt = kt0;
    float acc[NPT];
#pragma unroll
    for (int c = 0; c < NPT; c++) acc[c] = 0.f;
    float run[Conv::PAIRED ? NPT : 1]; // Q6_K: the finished runs of steps
#pragma unroll
    for (int c = 0; c < (Conv::PAIRED ? NPT : 1); c++) run[c] = 0.f;
    auto store_one = [&](int64_t row, int64_t col, float val) {
      if (row >= p.w.n || col >= p.m) return;
      const int64_t idx = col * p.ldy + row;
      const float v = BIAS ? with_bias(val, bias_at(p.bias, p.y_dtype, row), p.y_dtype) : val;
      if (p.y_dtype == XNQ_F32) static_cast<float *>(p.y)[idx] = v;
      else if (p.y_dtype == XNQ_F16) static_cast<__half *>(p.y)[idx] = __float2half_rn(v);
      else static_cast<__nv_bfloat16 *>(p.y)[idx] = __float2bfloat16_rn(v);
    };
    int ap = 0, nb = 0;  // i % AP, i % (NB / 2)
    uint32_t a_ph = 0;   // (i / AP) & 1
    // The next step's records and products were seen to be there while this step's were read back. The three waits one after the other took 500
    // cycles even when nothing was left to wait for, of 1400 that a step of 16 rows takes a drain warp.
    bool ready = false;
    for (int i = 0; i < nunits; i++) {
      const int ss = i % SIDE_STAGES;
      if (!__all_sync(0xffffffffu, ready)) { // else the step was there when the one before was read back
        if (alive) alive = mbar_wait_warp(side_full + 8 * ss, (i / SIDE_STAGES) & 1, 8u);
        if (alive) alive = mbar_wait_warp(mma_done + 8 * (2 * ap), a_ph, 8u);
        if (alive) alive = mbar_wait_warp(mma_done + 8 * (2 * ap + 1), a_ph, 8u);
      }
      ready = false;
      const uint32_t side = base + p.side_off + ss * p.side_stage_bytes;
      uint4 hdr = make_uint4(0, 0, 0, 0);
      float dw = 0.f;
      if (alive) hdr = lds128(side + (uint32_t)(32 * q + lane) * 16);
      if (Conv::PAIRED && alive) dw = __uint_as_float(lds32(side + HDR_BYTES + (uint32_t)(NP * 32 + (32 * q + lane) * 4)));
      if (alive) {
        tc_fence_after();
        const uint32_t taddr = tmem_d + ((uint32_t)(32 * q) << 16) + (uint32_t)(2 * nb * BUF_COLS + c0); // the halves' buffers are neighbours
#pragma unroll
        for (int ch = 0; ch < NPT / CH; ch++) {
          uint32_t v[8][CH];
          if constexpr (Conv::PAIRED) {
            int isum[CH] = {};
#pragma unroll
            for (int h = 0; h < 2; h++) {
#pragma unroll
              for (int j = 0; j < 8; j++) tmem_ld<CH>(taddr + (uint32_t)(h * BUF_COLS + (j >> 1) * NP + (j & 1) * ROWS + ch * CH), v[j]);
              tmem_ld_wait();
              q6k_sums<CH>(hdr, h, v, isum);
            }
#pragma unroll
            for (int c = 0; c < CH; c++) acc[ch * CH + c] += (dw * __uint_as_float(lds32(side + HDR_BYTES + (uint32_t)(c0 + ch * CH + c) * 32 + 16))) * (float)isum[c];
          } else {
#pragma unroll
            for (int j = 0; j < 8; j++) tmem_ld<CH>(taddr + (uint32_t)(j * NP + ch * CH), v[j]);
            tmem_ld_wait();
          }
          if (ch == NPT / CH - 1) { // every value of the buffers this warp needs is in registers: they may be overwritten
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty + 8 * (2 * nb)), mbar_arrive(acc_empty + 8 * (2 * nb + 1));
            const uint32_t next = mma_done + (ap + 1 == AP ? 0u : 16u * (uint32_t)(ap + 1)), ph = ap + 1 == AP ? a_ph ^ 1u : a_ph;
            ready = (i + 1 < nunits) & mbar_peek(side_full + 8 * ((i + 1) % SIDE_STAGES), ((i + 1) / SIDE_STAGES) & 1) & mbar_peek(next, ph) & mbar_peek(next + 8, ph);
          }
          if constexpr (!Conv::PAIRED) Conv::template Drain<CH>::run(hdr, side + HDR_BYTES, NP, c0 + ch * CH, v, acc + ch * CH);
        }
      }
      __syncwarp();
      if (alive && lane == 0) mbar_arrive(side_empty + 8 * ss);
      // ---- end of a segment (the tile's last step, or this CTA's last unit): store or hand over the sums ----
      const bool tile_end = kt == KT - 1, range_end = i == nunits - 1;
      if constexpr (Conv::PAIRED) {
        if ((kt & (SUM_RUN - 1)) == SUM_RUN - 1 || tile_end || range_end) {
          const bool last = tile_end || range_end;
#pragma unroll
          for (int c = 0; c < NPT; c++) {
            const float all = run[c] + acc[c];
            run[c] = last ? 0.f : all, acc[c] = last ? all : 0.f;
          }
        }
      }
      if (tile_end || range_end) {
        const int64_t row = (int64_t)tile * TILE_N + 32 * q + lane;
        if (tile_end && (tile != tile0 || kt0 == 0)) {
          if (alive) {
#pragma unroll
            for (int c = 0; c < NPT; c++) store_one(row, c0 + c, acc[c]);
          }
        } else {
          // this CTA's first segment (it starts where the CTA's range starts) uses scratch slot 2c, its last one, if another, 2c + 1
          const int slot = tile == tile0 ? 0 : 1;
          float *mine = p.partials + ((size_t)2 * blockIdx.x + slot) * ROWS * TILE_N;
#pragma unroll
          for (int c = 0; c < NPT; c++)
            if (c0 + c < p.m) mine[(size_t)(c0 + c) * TILE_N + 32 * q + lane] = acc[c];
          if (!range_end) asm volatile("bar.arrive 2, %0;" ::"n"(DW * 32 + 32) : "memory"); // a first segment (first_part): the weight producer takes its ticket
        }
#pragma unroll
        for (int c = 0; c < NPT; c++) acc[c] = 0.f;
      }
      if (++kt == KT) {
        kt = 0;
        tile++;
      }
      if (++ap == AP) ap = 0, a_ph ^= 1u;
      if (2 * ++nb == NB) nb = 0;
    }
    // ---- tiles that other CTAs have parts of: the last part to arrive adds all parts in k order (16 rows: in runs) ----
    // A release of the CTA's stores and the ticket take a microsecond, a trip to the parts 0.8. So: a first segment's ticket is taken by the weight
    // producer while this warp goes on with the next tile (in the loop, by a drain warp, it held up everything: Q8_0 11008 x 4096, 45 rows 28.5 us
    // instead of 25.0; both tickets at the end made one CTA the last of two tiles: Q8_0 4096 x 4096, 8 rows 14.1 instead of 10.8), one thread releases
    // for all. With the look ahead at the barriers, before -> now in a stream of calls: Q4_K 4096 x 14336, 16 rows 21.0 -> 18.2 us;
    // 512 x 13568 14.8 -> 12.4; 28672 x 4096 30.0 -> 25.4; 4096 x 4096 11.9 -> 10.9; Q8_0 11008 x 4096, 16 rows 18.5 -> 15.7; Q6_K 32000 x 4096, 16 rows
    // 38.8 -> 34.8; Q4_K 4096 x 4096, 64 rows 19.6 -> 17.7.
    const int last = tile0 + (kt0 + nunits - 1) / KT; // the tiles whose parts are in this CTA's scratch slots, or -1
    const int part0 = kt0 != 0 || nunits < KT ? tile0 : -1, part1 = last != tile0 && (kt0 + nunits) % KT != 0 ? last : -1;
    if (part0 >= 0 || part1 >= 0) {
      asm volatile("bar.sync 1, %0;" ::"n"(DW * 32) : "memory");
      const int ticket_of = et == 0 ? (first_part ? -1 : part0) : et == 1 ? part1 : -1;
      if (ticket_of >= 0) s_ticket[et] = take_ticket(p.tile_cnt + ticket_of);
      asm volatile("bar.sync 1, %0;" ::"n"(DW * 32) : "memory");
      if (first_part) asm volatile("bar.sync 3, %0;" ::"n"(DW * 32 + 32) : "memory");
#pragma unroll 1
      for (int slot = 0; slot < 2; slot++) {
        const int t = slot ? part1 : part0;
        if (t < 0) continue;
        const int t_u0 = t * KT;
        const int c_first = cta_of(t_u0, p.units_q, p.units_r), c_last = cta_of(t_u0 + KT - 1, p.units_q, p.units_r);
        if ((int)s_ticket[slot] != c_last - c_first) continue;
        if (et == 0) p.tile_cnt[t] = 0u; // every part has its ticket: the word is zero again for the next call
        // A thread adds four rows (4 lane ..) of the columns et / 32 + e DW. This code runs once and its instructions come from memory: 16 rows' parts are
        // requested four at a time, wider operands' one by one (three or four at a time took 20.4 us instead of 17.6 for Q4_K 4096 x 4096, 64 rows).
        constexpr int EV = ROWS * TILE_N / 4 / (DW * 32), AHEAD = DW == 8 ? 4 : 1;
        float sum[EV][4] = {}, some[DW == 8 ? EV : 1][4] = {};
        const float4 *parts = reinterpret_cast<const float4 *>(p.partials) + et;
#pragma unroll 1
        for (int cc = c_first; cc <= c_last; cc += AHEAD) {
          float4 v[AHEAD][EV];
#pragma unroll
          for (int a = 0; a < AHEAD; a++) {
            const int from = min(cc + a, c_last);
            const float4 *part = parts + (size_t)(2 * from + (cta_first_unit(from, p.units_q, p.units_r) >= t_u0 ? 0 : 1)) * (ROWS * TILE_N / 4);
#pragma unroll
            for (int e = 0; e < EV; e++) v[a][e] = et / 32 + e * DW < p.m ? __ldcg(part + e * DW * 32) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
          for (int a = 0; a < AHEAD; a++) {
            if (cc + a > c_last) break;
#pragma unroll
            for (int e = 0; e < EV; e++) {
              float (&to)[4] = DW == 8 ? some[DW == 8 ? e : 0] : sum[e];
              to[0] += v[a][e].x, to[1] += v[a][e].y, to[2] += v[a][e].z, to[3] += v[a][e].w;
            }
          }
          if constexpr (DW == 8) {
            if ((cc - c_first) % SUM_RUN == SUM_RUN - AHEAD || cc + AHEAD > c_last) { // a run is complete
#pragma unroll
              for (int e = 0; e < EV; e++)
#pragma unroll
                for (int j = 0; j < 4; j++) sum[e][j] += some[e][j], some[e][j] = 0.f;
            }
          }
        }
#pragma unroll
        for (int e = 0; e < EV; e++)
#pragma unroll
          for (int j = 0; j < 4; j++) store_one((int64_t)t * TILE_N + lane * 4 + j, et / 32 + e * DW, sum[e][j]);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) tmem_dealloc(tmem_d, TMEM_COLS);
}

// ---- activations: quantize (or take an activation image), lay out as the MMA's B operand, write the records ----
// CTAs of 256 threads over (activation row of the padded pass, 2048-element stretch of k); rows >= m are zero.
// Thread t handles elements 8t..8t+7 of a stretch; a warp covers one 256-element block.
template <int ACT, typename XT>
__global__ void __launch_bounds__(256) imma_prepare(const XT *__restrict__ x, const int8_t *__restrict__ img_q, const float *__restrict__ img_d,
                                                    const int16_t *__restrict__ img_b, int64_t m, int64_t k, int64_t ldx, int NP, int nsteps,
                                                    uint8_t *__restrict__ bimg, uint8_t *__restrict__ meta, unsigned int *__restrict__ tile_cnt, int tiles, int paired) {
  pdl_launch_dependents(); // the matmul kernel may start its set-up and its weight loads now
  pdl_wait();              // x may be the previous kernel's output; the scratch may still be read by the previous call
  const int row = blockIdx.x;
  if (blockIdx.x == 0 && blockIdx.y == 0)
    for (int i = threadIdx.x; i < tiles; i += blockDim.x) tile_cnt[i] = 0;
  const int lane = threadIdx.x & 31;
  const int64_t kpad = (int64_t)nsteps * 256;
  const int nblk_act = (int)(k / (ACT == XNQ_Q8_0 ? QK : QK_K));
  for (int64_t base = (int64_t)blockIdx.y * 2048; base < kpad; base += (int64_t)gridDim.y * 2048) {
    const int64_t k8 = base + (int64_t)threadIdx.x * 8;
    if (base + (int64_t)(threadIdx.x & ~31) * 8 >= kpad) break; // whole warps leave together
    uint32_t lo = 0, hi = 0;
    float d = 0.f;
    int sum16 = 0;
    const bool valid = row < m && k8 < k;
    if (img_q) {
      if (valid) {
        const uint2 c = *reinterpret_cast<const uint2 *>(img_q + (int64_t)row * k + k8);
        lo = c.x, hi = c.y;
        d = img_d[(int64_t)row * nblk_act + (ACT == XNQ_Q8_0 ? k8 / QK : k8 / QK_K)];
        sum16 = img_b[(int64_t)row * (k / 16) + k8 / 16];
      }
    } else {
      float v[8];
      if (valid) load8(x + (int64_t)row * ldx + k8, v);
      else {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = 0.f;
      }
      const Quant8 qv = ACT == XNQ_Q8_0 ? quantize8_q8_0(v, lane) : quantize8_q8k(v, lane);
      lo = qv.lo, hi = qv.hi, d = qv.d, sum16 = qv.sum16;
    }
    if (k8 < kpad) {
      // operand image: half step hs = k8 / 128, row `row`, 16-byte chunk (k8 % 128) / 16 swizzled with the row
      const int64_t hs = k8 >> 7;
      const int chunk = (int)((k8 & 127) >> 4);
      uint8_t *dst = bimg + (size_t)hs * (NP * 128) + (size_t)(row >> 3) * 1024 + (size_t)(row & 7) * 128 + (size_t)((chunk ^ (row & 7)) << 4) + (k8 & 8);
      if (paired) { // column `row` holds the first 16 of every 32 elements, column NP / 2 + row (a multiple of 8 further on) the others
        uint8_t *dst2 = dst + (size_t)(NP / 2 >> 3) * 1024;
        *reinterpret_cast<uint2 *>((chunk & 1) ? dst2 : dst) = make_uint2(lo, hi);
        *reinterpret_cast<uint2 *>((chunk & 1) ? dst : dst2) = make_uint2(0u, 0u);
      } else {
        *reinterpret_cast<uint2 *>(dst) = make_uint2(lo, hi);
      }
      uint32_t *rec = reinterpret_cast<uint32_t *>(meta + ((size_t)(k8 >> 8) * NP + row) * 32);
      if (ACT == XNQ_Q8_0) {
        // eight f32 block scales (0 beyond k), those of a block's rows side by side
        if ((lane & 3) == 0) reinterpret_cast<float *>(meta)[((size_t)(k8 >> 8) * 8 + ((k8 & 255) >> 5)) * NP + row] = d;
      } else {
        // 32-sums of the block's eight sub-blocks: lanes 4s .. 4s+3 hold sub-block s; sum16 is the pair sum on both lanes of a pair
        const int s32 = sum16 + __shfl_xor_sync(0xffffffffu, sum16, 2);
        const int sub = lane >> 2;
        uint32_t lo_b = (lane & 3) == 0 ? ((uint32_t)(s32 & 127) << (8 * (sub & 3))) : 0u;
        uint32_t hi_b = (lane & 3) == 0 ? ((uint32_t)((s32 >> 7) & 0xff) << (8 * (sub & 3))) : 0u;
        // combine the four sub-blocks of each half of the block: lanes 0..15 -> words 0 / 1, lanes 16..31 -> words 2 / 3
#pragma unroll
        for (int off = 4; off <= 8; off <<= 1) {
          lo_b |= __shfl_xor_sync(0xffffffffu, lo_b, off);
          hi_b |= __shfl_xor_sync(0xffffffffu, hi_b, off);
        }
        if (lane == 0 || lane == 16) {
          rec[(lane >> 4) * 2] = lo_b;
          rec[(lane >> 4) * 2 + 1] = hi_b;
        }
        if (lane == 0) {
          rec[4] = __float_as_uint(d);
          rec[5] = rec[6] = rec[7] = 0u;
        }
      }
    }
  }
}

int g_sms = 0;

struct Plan {
  int NP, nsteps, tiles, grid;
  size_t bimg_bytes, meta_bytes, cnt_bytes, part_bytes;
};
// operand images have their own row counts (operand_np); paired: two operand columns per row
Plan plan_for(int64_t m, int64_t k, int64_t n, bool operand, bool paired) {
  Plan pl{};
  pl.NP = operand ? operand_np(m) : (int)((m + 15) / 16 * 16) * (paired ? 2 : 1);
  pl.nsteps = (int)((k + 255) / 256);
  pl.tiles = (int)((n + TILE_N - 1) / TILE_N);
  const long long units = (long long)pl.tiles * pl.nsteps;
  pl.grid = (int)std::max<long long>(1, std::min<long long>(g_sms > 0 ? g_sms : 148, units / 2)); // at least two steps per CTA
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  pl.bimg_bytes = up((size_t)pl.nsteps * 2 * pl.NP * 128);
  pl.meta_bytes = up((size_t)pl.nsteps * pl.NP * 32);
  pl.cnt_bytes = up((size_t)pl.tiles * 4);
  pl.part_bytes = up((size_t)2 * (g_sms > 0 ? g_sms : 148) * (paired ? pl.NP / 2 : pl.NP) * TILE_N * 4);
  return pl;
}

template <typename Conv, bool BIAS>
int launch_np(const ImmaArgs &a, int NP, unsigned grid, cudaStream_t s) {
  // programmatic stream serialization: the kernel starts while the one that prepares the activations still runs; only
  // its weight loads are issued before griddepcontrol.wait
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3((unsigned)imma_threads(Conv::PAIRED ? NP / 2 : NP));
  cfg.dynamicSmemBytes = IMMA_SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if constexpr (Conv::PAIRED) { // 16 rows, 32 columns
    XNQ_CUDA(cudaLaunchKernelEx(&cfg, imma_kernel<Conv, 32, BIAS>, a, a.w.maps->codes, a.w.maps->high));
  } else if (NP == 16) XNQ_CUDA(cudaLaunchKernelEx(&cfg, imma_kernel<Conv, 16, BIAS>, a, a.w.maps->codes, a.w.maps->high));
  else if (NP == 32) XNQ_CUDA(cudaLaunchKernelEx(&cfg, imma_kernel<Conv, 32, BIAS>, a, a.w.maps->codes, a.w.maps->high));
  else if (NP == 48) XNQ_CUDA(cudaLaunchKernelEx(&cfg, imma_kernel<Conv, 48, BIAS>, a, a.w.maps->codes, a.w.maps->high));
  else XNQ_CUDA(cudaLaunchKernelEx(&cfg, imma_kernel<Conv, 64, BIAS>, a, a.w.maps->codes, a.w.maps->high));
  count_launch();
  return XNQ_OK;
}

template <typename Conv, bool BIAS>
int init_np() {
  if constexpr (!Conv::PAIRED) {
    XNQ_CUDA(cudaFuncSetAttribute(imma_kernel<Conv, 64, BIAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)IMMA_SMEM));
    XNQ_CUDA(cudaFuncSetAttribute(imma_kernel<Conv, 16, BIAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)IMMA_SMEM));
    XNQ_CUDA(cudaFuncSetAttribute(imma_kernel<Conv, 48, BIAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)IMMA_SMEM));
  }
  XNQ_CUDA(cudaFuncSetAttribute(imma_kernel<Conv, 32, BIAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)IMMA_SMEM));
  return XNQ_OK;
}
template <typename Conv>
int init_fmt() {
  const int rc = init_np<Conv, false>();
  return rc != XNQ_OK ? rc : init_np<Conv, true>();
}
template <typename Conv>
int launch_fmt(const ImmaArgs &a, int NP, unsigned grid, cudaStream_t s) {
  return a.bias ? launch_np<Conv, true>(a, NP, grid, s) : launch_np<Conv, false>(a, NP, grid, s);
}

} // namespace

bool imma_supported(const WeightView &w, int64_t m) {
  if (g_sms <= 0 || m < 1 || w.n < 1) return false;
  if (w.dtype == XNQ_Q6K) {
    if (m < IMMA_Q6K_MIN_M || m > IMMA_Q6K_MAX_M) return false;
  } else if (w.dtype != XNQ_Q4_0 && w.dtype != XNQ_Q8_0 && w.dtype != XNQ_Q4K) {
    return false;
  }
  if (((w.n + TILE_N - 1) / TILE_N) * ((w.k + 255) / 256) >= (1ll << 30)) return false; // the (tile, step) space is indexed with 32-bit integers
  return true;
}

// scratch of one call of m rows: the activations' operand image and records, the split tiles' tickets and partial sums. Grows with m.
size_t imma_workspace_bytes(const WeightView &w, int64_t m) {
  const Plan pl = plan_for(std::min<int64_t>(m, MAX_NP), w.k, w.n, w.dtype == XNQ_Q4K, w.dtype == XNQ_Q6K); // Q4_K: an operand image's columns are the most
  return pl.bimg_bytes + pl.meta_bytes + pl.cnt_bytes + pl.part_bytes + 256;
}

// x: float activations [m, k] (x_dtype F32 / F16 / BF16, row stride ldx) or an activation image (XNQ_ACT_IMAGE) of m rows.
int launch_imma(const WeightView &w, const void *x, int x_dtype, int64_t m, int64_t ldx, void *y, int y_dtype, int64_t ldy, void *workspace,
                cudaStream_t s, const void *bias) {
  const int64_t k = w.k;
  const int act = act_dtype_for(w.dtype);
  const size_t yes = type_size(y_dtype);
  const bool paired = w.dtype == XNQ_Q6K;
  const bool operand = x_dtype == XNQ_ACT_OPERAND; // the activations arrive in the kernel's own layout, with their ticket words: no activation kernel
  if (operand && (w.dtype != XNQ_Q4K || k % 256 || m > MAX_NP)) return fail(XNQ_ERR_UNSUPPORTED, "imma: an operand image serves Q8_K activations of one pass (m = %lld)", (long long)m);
  for (int64_t r0 = 0; r0 < m; r0 += MAX_NP) { // passes of at most 64 activation rows
    const int64_t rows = std::min<int64_t>(MAX_NP, m - r0);
    const Plan pl = plan_for(rows, k, w.n, operand, paired);
    uint8_t *ws = static_cast<uint8_t *>(workspace);
    uint8_t *bimg = ws;
    uint8_t *meta = bimg + pl.bimg_bytes;
    unsigned int *cnt = reinterpret_cast<unsigned int *>(meta + pl.meta_bytes);
    float *partials = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(cnt) + pl.cnt_bytes); // always in the caller's workspace
    if (operand) {
      if (pl.tiles > OPERAND_MAX_TILES) return fail(XNQ_ERR_SIZE, "imma: an operand image has ticket words for %d tiles of 128 rows, the weight has %d", OPERAND_MAX_TILES, pl.tiles);
      uint8_t *img = static_cast<uint8_t *>(const_cast<void *>(x));
      cnt = reinterpret_cast<unsigned int *>(img);
      bimg = img + OPERAND_TICKET_BYTES;
      meta = bimg + operand_bimg_bytes(pl.NP, k);
    }
    // ---- activations ----
    const int8_t *iq = nullptr;
    const float *id = nullptr;
    const int16_t *ib = nullptr;
    if (x_dtype == XNQ_ACT_IMAGE) {
      const ActView av = act_view(const_cast<void *>(x), m, k, act);
      const int blk = act == XNQ_Q8_0 ? QK : QK_K;
      iq = av.q + r0 * k, id = av.d + r0 * (k / blk), ib = av.bsum + r0 * (k / 16);
    }
    // The CTAs are started while the previous kernel drains, and the first SM that is free would take eight of them (3.9 us instead of
    // 1.3): unused shared memory keeps them apart.
    const dim3 prep_grid((unsigned)(paired ? pl.NP / 2 : pl.NP), (unsigned)std::min<int64_t>(16, (k + 2047) / 2048));
    const size_t spread = MAX_SPREAD / ((prep_grid.x * prep_grid.y + g_sms - 1) / g_sms) / 1024 * 1024;
#define XNQ_IMMA_PREP(ACT, XT)                                                                                                          \
  XNQ_CUDA(launch_pdl(imma_prepare<ACT, XT>, prep_grid, dim3(256), spread, s,     \
                      iq ? nullptr : static_cast<const XT *>(x) + r0 * ldx, iq, id, ib, rows, k, ldx, pl.NP, pl.nsteps, bimg, meta, cnt, pl.tiles, paired ? 1 : 0))
    if (operand) {
      // nothing to prepare
    } else if (act == XNQ_Q8_0) {
      if (x_dtype == XNQ_F16) XNQ_IMMA_PREP(XNQ_Q8_0, __half);
      else if (x_dtype == XNQ_BF16) XNQ_IMMA_PREP(XNQ_Q8_0, __nv_bfloat16);
      else XNQ_IMMA_PREP(XNQ_Q8_0, float);
    } else {
      if (x_dtype == XNQ_F16) XNQ_IMMA_PREP(XNQ_Q8K, __half);
      else if (x_dtype == XNQ_BF16) XNQ_IMMA_PREP(XNQ_Q8K, __nv_bfloat16);
      else XNQ_IMMA_PREP(XNQ_Q8K, float);
    }
#undef XNQ_IMMA_PREP
    if (!operand) count_launch();

    ImmaArgs a{};
    a.w = w;
    a.bimg = bimg;
    a.meta = meta;
    a.y = static_cast<char *>(y) + (size_t)r0 * ldy * yes;
    a.bias = bias;
    a.y_dtype = y_dtype;
    a.ldy = ldy;
    a.m = rows;
    a.nsteps = pl.nsteps;
    a.tiles = pl.tiles;
    a.units = pl.tiles * pl.nsteps;
    a.units_q = a.units / pl.grid, a.units_r = a.units % pl.grid;
    a.tile_cnt = cnt;
    a.partials = partials;
    int rc;
    uint32_t raw = 0, scales = 0; // bytes of a raw stage and of a converter warp's scale slot
    switch (w.dtype) {
      case XNQ_Q4K: a.step_x = 144, raw = ConvQ4K::RAW; break;
      case XNQ_Q8_0:
        a.step_x = 256, scales = ConvQ8_0::SCALES, a.scales = reinterpret_cast<const uint8_t *>(w.d), a.scale_row_bytes = (uint32_t)(w.dstride * 2);
        break;
      case XNQ_Q4_0:
        a.step_x = 128, raw = ConvQ4_0::RAW, scales = ConvQ4_0::SCALES, a.scales = reinterpret_cast<const uint8_t *>(w.d), a.scale_row_bytes = (uint32_t)(w.dstride * 2);
        break;
      case XNQ_Q6K:
        a.step_x = 128, raw = ConvQ6K::RAW, scales = ConvQ6K::SCALES, a.scales = reinterpret_cast<const uint8_t *>(w.sc), a.scale_row_bytes = (uint32_t)(k / 16);
        break;
      default: return fail(XNQ_ERR_DTYPE, "imma: dtype %d", w.dtype);
    }
    a.b_stage_bytes = (uint32_t)pl.NP * 256;
    a.side_stage_bytes = HDR_BYTES + (uint32_t)pl.NP * 32 + (paired ? TILE_N * 4 : 0);
    // Shared-memory plan: A stages (half steps of operand image) | raw stages (weights, whole steps) | B stages (activations, whole steps) | side
    // stages | scale slots. The first plan that leaves as many B stages as it names. Four raw stages in flight (Q8_0: operand stages) are what
    // DRAM's latency takes at its rate; an even number of them, so that a stage is always read by the same group of converter warps (a group
    // that took turns with the other could test a barrier two phases behind, which reads as complete).
    struct { int as, rs, bs; } static constexpr direct[] = {{8, 2, 3}, {6, 2, 2}, {4, 2, 2}}, converted[] = {{6, 4, 5}, {4, 6, 4}, {4, 4, 2}, {4, 2, 2}};
    const size_t budget = IMMA_SMEM - 1024; // 1024: alignment slack of the base
    a.a_stages = 0;
    auto try_plan = [&](int as, int rs, int least) {
      const size_t fixed = (size_t)as * A_STAGE_BYTES + (size_t)rs * raw + (size_t)SIDE_STAGES * a.side_stage_bytes + (size_t)CONV_WARPS * SCALE_SLOTS * scales;
      const int bs = fixed >= budget ? 0 : (int)std::min<size_t>(MAX_B_STAGES, (budget - fixed) / a.b_stage_bytes);
      if (!a.a_stages && bs >= least) a.a_stages = as, a.raw_stages = rs, a.b_stages = bs;
    };
    if (raw) for (const auto &c : converted) try_plan(c.as, c.rs, c.bs);
    else for (const auto &c : direct) try_plan(c.as, c.rs, c.bs);
    if (!a.a_stages) return fail(XNQ_ERR_SIZE, "imma: shared-memory plan does not fit");
    a.a_off = 0;
    a.raw_off = (uint32_t)a.a_stages * A_STAGE_BYTES;
    a.b_off = a.raw_off + (uint32_t)a.raw_stages * raw;
    a.side_off = a.b_off + a.b_stages * a.b_stage_bytes;
    a.scale_off = a.side_off + SIDE_STAGES * a.side_stage_bytes;
    profile_mark(s, true);
    if (w.dtype == XNQ_Q4K) rc = launch_fmt<ConvQ4K>(a, pl.NP, (unsigned)pl.grid, s);
    else if (w.dtype == XNQ_Q8_0) rc = launch_fmt<ConvQ8_0>(a, pl.NP, (unsigned)pl.grid, s);
    else if (w.dtype == XNQ_Q6K) rc = launch_fmt<ConvQ6K>(a, pl.NP, (unsigned)pl.grid, s);
    else rc = launch_fmt<ConvQ4_0>(a, pl.NP, (unsigned)pl.grid, s);
    profile_mark(s, false);
    if (rc != XNQ_OK) return rc;
  }
  return XNQ_OK;
}

int imma_init(int device) {
  cudaDeviceProp prop;
  XNQ_CUDA(cudaGetDeviceProperties(&prop, device));
  g_sms = prop.multiProcessorCount;
  int rc;
  if ((rc = init_fmt<ConvQ4K>()) != XNQ_OK) return rc;
  if ((rc = init_fmt<ConvQ8_0>()) != XNQ_OK) return rc;
  if ((rc = init_fmt<ConvQ6K>()) != XNQ_OK) return rc;
  if ((rc = init_fmt<ConvQ4_0>()) != XNQ_OK) return rc;
#define XNQ_IMMA_PREP_INIT(ACT, XT) XNQ_CUDA(cudaFuncSetAttribute(imma_prepare<ACT, XT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SPREAD))
  XNQ_IMMA_PREP_INIT(XNQ_Q8_0, float);
  XNQ_IMMA_PREP_INIT(XNQ_Q8_0, __half);
  XNQ_IMMA_PREP_INIT(XNQ_Q8_0, __nv_bfloat16);
  XNQ_IMMA_PREP_INIT(XNQ_Q8K, float);
  XNQ_IMMA_PREP_INIT(XNQ_Q8K, __half);
  XNQ_IMMA_PREP_INIT(XNQ_Q8K, __nv_bfloat16);
#undef XNQ_IMMA_PREP_INIT
  unsigned int zero = 0;
  XNQ_CUDA(cudaMemcpyToSymbol(g_imma_status, &zero, sizeof(zero)));
  return XNQ_OK;
}

int imma_status(unsigned int *bits) {
  XNQ_CUDA(cudaMemcpyFromSymbol(bits, g_imma_status, sizeof(*bits)));
  return XNQ_OK;
}

} // namespace xnq
