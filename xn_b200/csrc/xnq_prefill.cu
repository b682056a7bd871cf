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
//   D  f32 in tensor memory; eight epilogue warps read it back with tcgen05.ld, undo the power-of-two
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
constexpr int LOADER_WARP = PRODUCER_WARPS, MMA_WARP = LOADER_WARP + 1;
constexpr int NTHREADS = PRODUCER_WARPS * 32 + 64; // warps 0-15 producers, then the loader warp and the MMA warp
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
// by a whole warp that stays converged; the result is the same in all lanes
__device__ __forceinline__ bool mbar_wait_uniform(uint32_t bar, uint32_t parity, unsigned int bit) {
  const bool ok = mbar_wait(bar, parity, bit);
  return __all_sync(0xffffffffu, ok);
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
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// A from tensor memory, B from shared memory
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the mbarrier once every MMA issued so far by this thread has finished reading smem / writing tmem
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
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
__device__ __forceinline__ uint32_t idesc_f16(int umma_n) { return (1u << 4) | ((uint32_t)(umma_n >> 3) << 17) | ((uint32_t)(TILE_N >> 4) << 24); }

struct PrefillArgs {
  WeightView w;
  const uint8_t *xh;      // activation image: [k-steps][m_pad][64] fp16, swizzled rows, k-step-permuted
  const float *row_unscale; // [m_pad]: 1 / (activation row scale * weight scale)
  void *y;
  int y_dtype;
  int64_t ldy;
  int64_t m, m_pad;
  int ksteps;
  int nstages;            // stages: weights in tensor memory, activations in shared memory
  int acc_bufs;           // accumulators: 1 of 256 columns, 2 of 128 (tiles of up to 128 activation rows)
  int raw_slots;          // raw super-steps in shared memory, the one being converted included
  uint32_t b_stride;      // bytes between B stages (largest mt of the grid x 128, multiple of 1024)
  uint32_t raw_off;       // offset of the raw ring behind the B ring
  float wscale;           // power of two applied to every dequantized weight
  // persistent kernel: tile t = tile_n * tiles_m + tile_m; work unit u = t * ksteps + kt; CTA c takes units
  // [units * c / G, units * (c + 1) / G), or whole tiles when the output cannot be accumulated atomically
  int tiles_n, tiles_m;
  long long units;
  int whole_tiles;
  unsigned int *tile_cnt; // [tiles] arrival tickets then [tiles] "first partial stored" flags; zeroed by the prepare kernel
};

using namespace prefill_rows;

// waits until at most `pending` of this thread's committed copy groups are still in flight
__device__ __forceinline__ void cp_async_wait(int pending) {
  switch (pending) {
    case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
    case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
    case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
    case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
    default: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
  }
}

// Writes one 32-column chunk of an accumulator row block: column j of the chunk is activation row
// m_first + j, this lane's accumulator lane is weight row `row`. MODE: 0 f32 store, 1 f32 atomic add,
// 2 f16 store, 3 bf16 store.
template <int MODE>
__device__ __forceinline__ void drain_chunk(const uint32_t (&v)[32], float ru_lane, void *y, int64_t ldy, int64_t row, int64_t m_first, int64_t m_end,
                                            bool row_ok) {
  // a running pointer and one small count: the few warps that drain have nobody to hide instruction latency
  // behind, so every instruction per column counts
  const int es = MODE <= 1 ? 4 : 2;
  char *yp = static_cast<char *>(y) + (m_first * ldy + row) * es;
  const int64_t step = ldy * es;
  const int nvalid = row_ok ? (int)min((int64_t)32, m_end - m_first) : 0;
#pragma unroll
  for (int j = 0; j < 32; j++) {
    const float val = __uint_as_float(v[j]) * __shfl_sync(0xffffffffu, ru_lane, j);
    if (j < nvalid) {
      if (MODE == 0) *reinterpret_cast<float *>(yp) = val;
      else if (MODE == 1) atomicAdd(reinterpret_cast<float *>(yp), val);
      else if (MODE == 2) *reinterpret_cast<__half *>(yp) = __float2half_rn(val);
      else *reinterpret_cast<__nv_bfloat16 *>(yp) = __float2bfloat16_rn(val);
    }
    yp += step;
  }
}

// ---- the kernel ------------------------------------------------------------------------------------------------
// One CTA per SM walks a contiguous range of the flattened (tile, k-step) space, so all SMs finish
// together whatever the tile count, and a tile whose k-steps are split between CTAs is summed in
// global memory: the first CTA to finish its part stores it and raises the tile's flag, the others add
// theirs atomically after seeing the flag (two to three parts per split tile; f32 output only - other
// output types get whole tiles). Tiles of up to 128 activation rows have two accumulators, so the drain of one
// segment overlaps the MMAs of the next; wider ones have one, and the producers fill the stages meanwhile.
// Roles: 16 producer warps, one activation-loader warp (one bulk copy per stage), one MMA-issuing warp, eight drain
// warps. Stage counters run on across segments.
// Producers: the four warps of a row group (32 weight rows) fetch the group's bytes of a super-step together, several
// super-steps ahead, and each then converts its own k-step of it (or its half of one), so the k-steps of a super-step are
// converted side by side and a warp's chain of waits, loads, arithmetic and stores has a super-step's MMAs to run in. One
// barrier of the row group's four warps per super-step makes the copies visible to all of them and tells that the slot of
// the previous super-step has been read.
constexpr int EPI_WARPS = 8; // two per accumulator lane quarter, splitting the columns
constexpr int EPI_WARP0 = MMA_WARP + 1;
constexpr int NTHREADS_SK = NTHREADS + EPI_WARPS * 32;

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
  __device__ __forceinline__ int tile(int tiles_m) const { return tile_n * tiles_m + tile_m; }
};

template <typename RowT>
__global__ void __launch_bounds__(NTHREADS_SK, 1) prefill_persistent_kernel(PrefillArgs p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  __shared__ __align__(8) uint64_t bars[2 * MAX_STAGES + 4]; // full, empty (8 each), acc_full[2], acc_empty[2]
  __shared__ uint32_t tmem_slot;
  __shared__ unsigned int s_ticket;
  const int S = p.nstages;
  const uint32_t full = smem_u32(bars), empty = full + 8 * MAX_STAGES, acc_full = empty + 8 * MAX_STAGES, acc_empty = acc_full + 16;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31; // so that the compiler knows `warp` to be uniform
  const uint32_t b_ring = smem_base;
  const int NACC = p.acc_bufs;
  const int KT = p.ksteps;

  // this CTA's range of work units
  long long u0, u1;
  if (p.whole_tiles) {
    const long long T = (long long)p.tiles_n * p.tiles_m;
    u0 = (T * blockIdx.x / gridDim.x) * KT;
    u1 = (T * (blockIdx.x + 1) / gridDim.x) * KT;
  } else {
    u0 = p.units * blockIdx.x / gridDim.x;
    u1 = p.units * (blockIdx.x + 1) / gridDim.x;
  }
  const int nsteps = (int)(u1 - u0);
  const int TM = p.tiles_m;
  const Cursor start{(int)((u0 / KT) / TM), (int)((u0 / KT) % TM), (int)(u0 % KT)};

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(full + 8 * s, PRODUCER_WARPS / RowT::KPS + 1);
      mbar_init(empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(acc_full + 8 * b, 1);
      mbar_init(acc_empty + 8 * b, EPI_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == LOADER_WARP) {
    tmem_alloc(smem_u32(&tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();
  const uint32_t tmem_d = __shfl_sync(0xffffffffu, tmem_slot, 0);

  if (warp < PRODUCER_WARPS) {
    // ---- producers (nothing here waits for the kernel that prepares the activations: weights are immutable) ----
    constexpr int KPS = RowT::KPS, NCOPY = (32 * RowT::ITEMS + 127) / 128;
    const int rg = warp & 3, kg = warp >> 2;
    const int kk = kg % KPS, hf = kg / KPS; // this warp's k-step of a super-step; which half of it (KPS = 2)
    const int t = kg * 32 + lane; // 0..127 in the row group
    const uint32_t raw = smem_base + p.raw_off + (uint32_t)(rg * 32 * RowT::ROWB);
    constexpr uint32_t SLOT = TILE_N * RowT::ROWB;
    const int SPT = (KT + KPS - 1) / KPS; // super-steps per tile
    const int R = p.raw_slots;
    // position of the copies in the super-step space
    int l_n = start.tile_n, l_m = start.tile_m, l_s = start.kt / KPS, l_slot = 0;
    const int last_kt = nsteps - 1 + start.kt; // counted from the start of the first tile
    int l_left = nsteps > 0 ? (last_kt / KT) * SPT + (last_kt % KT) / KPS - l_s + 1 : 0; // super-steps still to be copied
    int left = l_left;
    Item it[NCOPY]; // this thread's copies; their addresses change with the tile only
    auto bind = [&]() {
#pragma unroll
      for (int i = 0; i < NCOPY; i++) {
        const int item = min(i * 128 + t, 32 * RowT::ITEMS - 1);
        it[i] = RowT::item(p.w, min((int64_t)l_n * TILE_N + 32 * rg + item / RowT::ITEMS, p.w.n - 1), item % RowT::ITEMS);
      }
    };
    bind();
    uint32_t to[NCOPY]; // where they go in a slot
#pragma unroll
    for (int i = 0; i < NCOPY; i++) to[i] = raw + (uint32_t)(((i * 128 + t) / RowT::ITEMS) * RowT::ROWB + ((i * 128 + t) % RowT::ITEMS) * 16);
    auto issue = [&]() {
      if (l_left > 0) {
        l_left--;
        const uint32_t slot = (uint32_t)l_slot * SLOT;
#pragma unroll
        for (int i = 0; i < NCOPY; i++) {
          if ((32 * RowT::ITEMS) % 128 == 0 || i * 128 + t < 32 * RowT::ITEMS) {
            const uint32_t off = ((uint32_t)l_s * it[i].mul) & ~15u;
            if (RowT::LIMITED) cp_async16(to[i] + slot, it[i].p + (off < it[i].lim ? off : 0u), off < it[i].lim ? 16u : 0u);
            else cp_async16(to[i] + slot, it[i].p + off, 16u);
          }
        }
        if (++l_slot == R) l_slot = 0;
        if (++l_s == SPT) {
          l_s = 0;
          if (++l_m == TM) {
            l_m = 0, l_n++;
            bind();
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int j = 0; j < R - 1; j++) issue();
    int c_s = start.kt / KPS, c_slot = 0;
    int base_i = -start.kt; // the CTA's step number of the current tile's first k-step
    int at = 0, s = 0;      // s = at % S, lap: parity of at / S, of the last step this warp looked at
    uint32_t lap = 0;
    bool alive = true;
    for (; left > 0; left--) {
      cp_async_wait(R - 2); // the super-step's copies of this thread have landed
      asm volatile("bar.sync %0, 128;" ::"r"(2 + rg) : "memory"); // ... and those of the row group's other threads; all have read the previous slot
      issue();              // into the previous slot
      const int kt = c_s * KPS + kk, i = base_i + kt;
      if (alive && kt < KT && i >= 0 && i < nsteps) {
        for (s += i - at, at = i; s >= S; lap ^= 1u) s -= S;
        if (i >= S) alive = mbar_wait_uniform(empty + 8 * s, lap ^ 1u, 1u); // a warp that gave up still takes part in the barriers
        if (alive) {
          tc_fence_after();
          const uint32_t slot = raw + (uint32_t)c_slot * SLOT + (uint32_t)(lane * RowT::ROWB);
          const uint32_t dst = tmem_d + ((uint32_t)(32 * rg) << 16) + (uint32_t)(A_COL0 + s * A_COLS);
          const typename RowT::Head head = RowT::head(slot, c_s, kk, p.wscale);
#pragma unroll
          for (int h = 0; h < KPS / 2; h++) {
            const int half = KPS == 2 ? hf : h;
            uint32_t o[16];
            RowT::half(head, slot, kk, half, o); // a lane past the weight's last row repeats that row and is not stored
            tmem_st16(dst + 16 * half, o);
          }
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(full + 8 * s);
        }
      }
      if (++c_slot == R) c_slot = 0;
      if (++c_s == SPT) {
        c_s = 0;
        base_i += KT;
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  } else if (warp == LOADER_WARP) {
    // ---- activation loader: the whole warp runs the loop, one elected lane issues (see the MMA issuer) ----
    pdl_wait(); // the activation image is the previous kernel's output
    Cursor cur = start;
    int s = 0, issued = 0;
    uint32_t lap = 0;
    for (int i = 0; i < nsteps; i++) {
      if (i >= S && !mbar_wait_uniform(empty + 8 * s, lap ^ 1u, 2u)) break;
      const int64_t m0 = (int64_t)cur.tile_m * MAX_MT;
      const uint32_t bytes = (uint32_t)min((int64_t)MAX_MT, p.m_pad - m0) * 128;
      if (elect_one()) {
        mbar_expect_tx(full + 8 * s, bytes);
        bulk_g2s(b_ring + s * p.b_stride, p.xh + ((size_t)cur.kt * p.m_pad + m0) * 128, bytes, full + 8 * s);
      }
      __syncwarp();
      issued = i + 1;
      cur.advance(1, KT, TM);
      if (++s == S) s = 0, lap ^= 1u;
    }
    for (int i = max(0, issued - S); i < issued; i++) mbar_wait_uniform(full + 8 * (i % S), (i / S) & 1, 2u); // nothing in flight at exit
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
      const int buf = NACC == 2 ? seg & 1 : 0, use = NACC == 2 ? seg >> 1 : seg;
      if (use > 0 && alive) alive = mbar_wait(acc_empty + 8 * buf, (use - 1) & 1, 4u); // the drain of this buffer's previous segment
      const uint32_t idesc = idesc_f16(min(MAX_MT, (int)p.m_pad - cur.tile_m * MAX_MT));
      const uint32_t d = tmem_d + (uint32_t)(buf * 128);
      for (int j = 0; j < len; j++) {
        if (alive) alive = mbar_wait(full + 8 * s, round & 1, 4u);
        tc_fence_after();
        __syncwarp();
        const uint32_t a = tmem_d + (uint32_t)(A_COL0 + s * A_COLS);
        const uint64_t bdesc = smem_desc_sw128(b_ring + s * p.b_stride);
        if (elect_one() && alive) {
#pragma unroll
          for (int ks = 0; ks < BK / 16; ks++) umma_f16(d, a + (uint32_t)(ks * 8), bdesc + (uint64_t)(ks * 2), idesc, (j | ks) ? 1u : 0u);
          umma_commit(empty + 8 * s);
          if (j == len - 1) umma_commit(acc_full + 8 * buf);
        }
        __syncwarp();
        if (++s == S) {
          s = 0;
          round++;
        }
      }
      i += len;
      cur.advance(len, KT, TM);
    }
  } else {
    // ---- drain: eight warps, two to a quarter q of the accumulator lanes (weight rows 32 q ..), which take turns in its chunks of 32 columns ----
    const int q = warp & 3; // tensor-memory lanes a warp may read are fixed by its index modulo 4
    const int half = (warp - EPI_WARP0) >> 2; // which half of the 32-column chunks this warp takes
    const int et = threadIdx.x - EPI_WARP0 * 32; // 0..255
    pdl_wait(); // the previous kernel writes the row factors and zeroes the tiles' tickets
    Cursor cur = start;
    bool alive = true;
    int i = 0;
    for (int seg = 0; i < nsteps && alive; seg++) {
      const int len = min(KT - cur.kt, nsteps - i);
      const bool whole = cur.kt == 0 && len == KT;
      const int buf = NACC == 2 ? seg & 1 : 0, use = NACC == 2 ? seg >> 1 : seg;
      const int tile_n = cur.tile_n, tile_m = cur.tile_m, tile = cur.tile(TM);
      const int64_t row = (int64_t)tile_n * TILE_N + 32 * q + lane;
      const int64_t m0 = (int64_t)tile_m * MAX_MT;
      const int mt = (int)min((int64_t)MAX_MT, p.m_pad - m0);
      // one thread waits for the accumulator and, for a tile shared with other CTAs, settles who stores and
      // who adds; the eight warps then act on the same answers
      if (et == 0) {
        unsigned int t = mbar_wait(acc_full + 8 * buf, use & 1, 8u) ? 0u : 0x80000000u;
        if (!whole && t == 0) {
          t = atomicAdd(p.tile_cnt + tile, 1u);
          if (t > 0) { // wait (bounded) until the first finisher's stores are visible
            const unsigned int *flag = p.tile_cnt + (size_t)p.tiles_n * p.tiles_m + tile;
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
      const unsigned int ticket = s_ticket & 0x7fffffffu;
      alive = (s_ticket & 0x80000000u) == 0;
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory"); // s_ticket may be rewritten from here on
      if (alive) {
        tc_fence_after();
        const uint32_t lane_addr = tmem_d + (uint32_t)(buf * 128) + ((uint32_t)(32 * q) << 16);
        for (int c0 = 32 * half; c0 < mt; c0 += 32 * (EPI_WARPS / 4)) {
          uint32_t v[32];
          tmem_ld32(lane_addr + c0, v);
          const float ru_lane = (m0 + c0 + lane < p.m_pad) ? p.row_unscale[m0 + c0 + lane] : 0.f; // the chunk's 32 row factors
          tmem_ld_wait();
          const bool row_ok = row < p.w.n;
          if (p.y_dtype == XNQ_F32) {
            if (ticket == 0) drain_chunk<0>(v, ru_lane, p.y, p.ldy, row, m0 + c0, p.m, row_ok);
            else drain_chunk<1>(v, ru_lane, p.y, p.ldy, row, m0 + c0, p.m, row_ok);
          } else if (p.y_dtype == XNQ_F16) {
            drain_chunk<2>(v, ru_lane, p.y, p.ldy, row, m0 + c0, p.m, row_ok);
          } else {
            drain_chunk<3>(v, ru_lane, p.y, p.ldy, row, m0 + c0, p.m, row_ok);
          }
        }
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty + 8 * buf); // this warp has read its lanes: the buffer may be overwritten
      if (!whole && alive) {
        if (ticket == 0) __threadfence();
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
        if (ticket == 0 && et == 0) {
          unsigned int *flag = p.tile_cnt + (size_t)p.tiles_n * p.tiles_m + tile;
          asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag), "r"(1u) : "memory");
        }
      }
      i += len;
      cur.advance(len, KT, TM);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == LOADER_WARP) tmem_dealloc(tmem_d, 512);
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

int g_num_sms = 0;

template <typename RowT>
int launch_persistent_fmt(const PrefillArgs &a, unsigned ctas, size_t smem, cudaStream_t s) {
  XNQ_CUDA(launch_pdl(prefill_persistent_kernel<RowT>, dim3(ctas), dim3(NTHREADS_SK), smem, s, a));
  count_launch();
  return XNQ_OK;
}

constexpr size_t SM_SMEM = 228 * 1024, MAX_SPREAD = SM_SMEM / 2;
static_assert(RowQ4_0::ROWB == RowQ4K::ROWB && RowQ8_0::ROWB == RowQ4K::ROWB, "the raw ring's plan assumes one slot size for these");
constexpr size_t PREFILL_SMEM = 226 * 1024; // everything an SM offers minus the static barriers and a reserve

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
                   void *workspace, cudaStream_t s) {
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
  a.y_dtype = y_dtype;
  a.ldy = ldy;
  a.m = m;
  a.m_pad = m_pad;
  a.ksteps = ksteps;
  // Shared-memory plan: B ring | raw ring. With up to eight stages a producer warp can be a whole super-step ahead of the MMAs; what is
  // left goes to the raw ring (it covers the memory latency of the weights). At 256 activation rows that is five stages and three
  // raw slots (two for Q6_K).
  const uint32_t slot = TILE_N * (w.dtype == XNQ_Q6K ? RowQ6K::ROWB : RowQ4K::ROWB);
  const uint32_t mt_max = (uint32_t)std::min<int64_t>(MAX_MT, m_pad);
  a.b_stride = (mt_max * 128 + 1023) & ~1023u;
  const size_t budget = PREFILL_SMEM - 1024; // alignment slack
  a.nstages = (int)std::min<size_t>(MAX_STAGES, (budget - 2 * slot) / a.b_stride);
  if (a.nstages < MIN_STAGES) return fail(XNQ_ERR_SIZE, "prefill: shared-memory plan does not fit");
  a.raw_slots = (int)std::min<size_t>(MAX_RAW_SLOTS, (budget - (size_t)a.nstages * a.b_stride) / slot);
  a.raw_off = a.nstages * a.b_stride;
  a.acc_bufs = m_pad <= 128 ? 2 : 1;
  a.wscale = wscale;
  const dim3 grid((unsigned)((w.n + TILE_N - 1) / TILE_N), (unsigned)((m_pad + MAX_MT - 1) / MAX_MT));
  a.tiles_n = (int)grid.x;
  a.tiles_m = (int)grid.y;
  a.units = (long long)grid.x * grid.y * ksteps;
  a.whole_tiles = y_dtype == XNQ_F32 ? 0 : 1;
  a.tile_cnt = tile_cnt;
  profile_mark(s, true);
  int rc;
  const long long tiles = (long long)grid.x * grid.y;
  const long long want = a.whole_tiles ? tiles : std::max<long long>(1, a.units / 8); // at least 8 k-steps per CTA
  const unsigned ctas = (unsigned)std::min<long long>(g_num_sms, want);
  switch (w.dtype) {
    case XNQ_Q4_0: rc = launch_persistent_fmt<RowQ4_0>(a, ctas, PREFILL_SMEM, s); break;
    case XNQ_Q8_0: rc = launch_persistent_fmt<RowQ8_0>(a, ctas, PREFILL_SMEM, s); break;
    case XNQ_Q4K: rc = launch_persistent_fmt<RowQ4K>(a, ctas, PREFILL_SMEM, s); break;
    case XNQ_Q6K: rc = launch_persistent_fmt<RowQ6K>(a, ctas, PREFILL_SMEM, s); break;
    default: rc = fail(XNQ_ERR_DTYPE, "prefill: dtype %d", w.dtype);
  }
  profile_mark(s, false);
  return rc;
}

int prefill_init(int device) {
  cudaDeviceProp prop;
  XNQ_CUDA(cudaGetDeviceProperties(&prop, device));
  g_num_sms = prop.multiProcessorCount;
  XNQ_CUDA(cudaFuncSetAttribute(prefill_persistent_kernel<RowQ4_0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PREFILL_SMEM));
  XNQ_CUDA(cudaFuncSetAttribute(prefill_persistent_kernel<RowQ8_0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PREFILL_SMEM));
  XNQ_CUDA(cudaFuncSetAttribute(prefill_persistent_kernel<RowQ4K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PREFILL_SMEM));
  XNQ_CUDA(cudaFuncSetAttribute(prefill_persistent_kernel<RowQ6K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PREFILL_SMEM));
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
