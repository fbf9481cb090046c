// Blackwell tensor-core GEMM for the complex products of the mixed solver:
// tcgen05.mma issued by one thread, BF16 operands staged by TMA
// (cp.async.bulk.tensor) into 128-byte-swizzled shared memory through rings
// of plane slots guarded by mbarriers, FP32 accumulators in tensor memory (TMEM)
// drained by the epilogue warps with tcgen05.ld.
//
// Complex products as one real GEMM.  For C = op(A) B (A: m x k, B: k x n
// complex) the kernel computes the real product D = A' B'^T with
//   A'(r, :)     = [ Re op(A)(r, 0..k) | Im op(A)(r, 0..k) ]            (K' = 2 kp)
//   B'^T(2c, :)   = [ Re B(0..k, c)     | -Im B(0..k, c) ]
//   B'^T(2c+1, :) = [ Im B(0..k, c)     |  Re B(0..k, c) ]
// so that D(r, 2c) = Re C(r, c) and D(r, 2c+1) = Im C(r, c): every epilogue
// thread owns one row and writes interleaved complex results.  Both operands
// are K-major (K contiguous), the layout tcgen05 reads without transposition.
//
// Operands are "planes" of BF16 values: digit planes of a fixed-point split
// or the three BF16 pieces of an FP32 number.  Within one K-step (one or two
// K-blocks, 64 of K' each) a launch runs a list of plane pairs; every plane's
// tile is staged once per K-block, in a slot of its own, and stays until the
// last pair that uses it.  The pairs form groups that share an accumulator;
// the epilogue drains a group's sums from one TMEM accumulator while the
// tensor cores fill the next.
//
//  * fixed mode (FP64-accurate products): every row of op(A) and column of B
//    is scaled by a power of two and cut into signed 8-bit digits, balanced
//    (|d| <= 128, the leading digit up to 256; BF16 holds every integer up to
//    256 exactly).  A group is the digit pairs (s, t) of one weight s + t; its
//    FP32 sum over the K-step, at most 64 (2 2^15 + 5 2^14) or 128 (2 2^15 + 2^14),
//    is below 2^24, an exact integer, drained (exact float -> int) into 64-bit fixed point,
//    acc += g << shift(s + t).  Digit pairs whose weight is below the kept
//    precision are not issued.  The result is acc scaled by
//    2^(e_row + f_col + base): FP64 complex, no intermediate in global memory.
//  * f32 mode (FP32-accurate products): x = x0 + x1 + x2 (three BF16 pieces
//    of an FP32 value, 24 bits); of the six pairs with weight >= 2^-16 the leading
//    one has an accumulator of its own, where products of 16 bits lose little, and
//    the five below share one (the tensor cores cut off what lies below the last
//    place of the sum, a bias towards zero where small terms meet a large sum: all
//    six in one accumulator were off by 3e-7 of like-signed sums, 1e-8 so).  Both
//    collect kF32Span K-blocks and are drained into register sums; C = alpha D + beta C.
//
// GPU safety: every mbarrier wait is bounded by wall time (%globaltimer);
// on expiry the thread records an error code, the other roles see it and
// stop, the producer waits (bounded) for its copies in flight and the
// allocating warp frees TMEM before the CTA exits.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "olc_common.h"
#include "olc_tcgemm.h"

namespace olc {
namespace tc {

namespace {

constexpr int BM = 128;            // rows per tile (TMEM lanes)
constexpr int BK = 64;             // K per stage: 64 BF16 = one 128-byte swizzle row
constexpr int MAX_SLOTS = 8;       // plane slots per operand
constexpr int kEpiWarps = 16;      // loads in flight for the drains; 96 registers hold 32 64-bit sums
constexpr int kThreads = (kEpiWarps + 2) * 32;
// accumulators: four of 128 columns (fixed mode), two of 256 (f32 mode)
template <int MODE>
constexpr int num_acc() { return MODE == 0 ? 4 : 2; }
constexpr int kTmemCols = 512;
constexpr int kF32Span = 4;        // K-blocks an accumulator of the f32 mode collects
constexpr long long kWaitNs = 2000000000LL;   // 2 s per wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for the phase of `parity`; false when the wait expired or
// another role of the CTA gave up (error word set).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* cta_err,
                                          int* gerr, int code) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = now_ns();
  for (;;) {
    if (mbar_try(bar, parity)) return true;
    if (*cta_err) return false;
    if ((long long)(now_ns() - t0) > kWaitNs) {
      *cta_err = code;
      atomicExch(gerr, code);
      return false;
    }
  }
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
      "[%2];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row atoms of
// 1024 bytes (stride byte offset), descriptor version 1.  lo: the address
// field (bytes / 16) with kDescLo.
constexpr uint32_t kDescLo = 1u << 16, kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint64_t sdesc(uint32_t lo) { return ((uint64_t)kDescHi << 32) | lo; }
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
  return one != 0;
}
// Instruction descriptor of kind::f16: BF16 A and B, FP32 D, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void umma(uint32_t dt, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dt),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// 16 consecutive 32-bit TMEM columns of this thread's lane
__device__ __forceinline__ void tmem_ld16(uint32_t ta, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(ta));
}
__device__ __forceinline__ void tmem_ld8(uint32_t ta, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(ta));
}
// Waits for every load issued so far; r, the values about to be used, passes
// through so that no use of it moves ahead of the wait.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
               :
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Tile of a CTA: grouped raster (GM row tiles at a time) so that the CTAs in
// flight share operand panels in L2.
__device__ __forceinline__ void tile_of(int t, int nmt, int nnt, int& mt, int& nt) {
  constexpr int GM = 8;
  const int per_group = GM * nnt;
  const int g = t / per_group, first = g * GM;
  const int gsize = min(GM, nmt - first);
  const int r = t % per_group;
  mt = first + r % gsize;
  nt = r / gsize;
}

constexpr int kTileBytesA = BM * BK * 2;
template <int MODE>
constexpr int tile_bytes_b() { return (MODE == 0 ? 128 : 256) * BK * 2; }
// planes' slots, barriers, alignment slack
inline int smem_total(int mode, int slots_a, int slots_b) {
  return slots_a * kTileBytesA + slots_b * (mode == 0 ? tile_bytes_b<0>() : tile_bytes_b<1>()) + 512 + 1024;
}

}  // namespace

// ---------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------
// What bounds it: in the fixed mode the copies from L2 and the MMAs one after the
// other: a K-block's 14 tiles of 16 KB fill shared memory and are all in use
// for half of its pairs, the copies run at the 5.4 TB/s that all SMs together
// reach, and what is left of the 34 pairs hides about a third of them.  In the
// f32 mode the copies' latency at the K-steps' ends.  Measured: FP64-accurate
// product of order 1248 1025 -> 818 us; FP32-accurate ones with their slices 75 -> 72
// (order 832, the kernel alone 55 -> 60) and 362 -> 325 us (2000, 274 -> 277); a mixed
// pass over 64 matrices of order 832: FP64-accurate products 22.7 -> 18.8 ms,
// FP32-accurate ones (as then formed) 18.5 -> 14.2 ms, now 11.5.
// MODE 0 (fixed): BN = 128, four accumulators of 128 columns, int64 drains,
//   FP64 complex output.  Epilogue warp w owns TMEM lanes 32 (w % 4) .. +31
//   and columns 32 (w / 4) .. +31 of the tile (16 complex columns).
// MODE 1 (f32):   BN = 256, two accumulators, FP32 complex output with
//   alpha, beta; warp w owns columns 64 (w / 4) .. +63 (32 complex).

template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
    tc_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ TcParams p) {
  constexpr int BN = MODE == 0 ? 128 : 256;
  constexpr int NACC = num_acc<MODE>();
  constexpr uint32_t IDESC = idesc_bf16(BM, BN);
  constexpr int TB = tile_bytes_b<MODE>();
  constexpr int PRODUCER_WARP = kEpiWarps, MMA_WARP = PRODUCER_WARP + 1;
  constexpr int CW = 4 * BN / kEpiWarps;      // columns of an epilogue warp
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint8_t* sA = smem;
  uint8_t* sB = smem + p.slots_a * kTileBytesA;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sB + p.slots_b * TB);
  uint64_t* fullA = bars;                    // [slot] TMA -> MMA
  uint64_t* emptyA = fullA + MAX_SLOTS;      // [slot] MMA -> TMA
  uint64_t* fullB = emptyA + MAX_SLOTS;
  uint64_t* emptyB = fullB + MAX_SLOTS;
  uint64_t* accfull = emptyB + MAX_SLOTS;    // [NACC] MMA -> epilogue
  uint64_t* accempty = accfull + 4;          // [NACC] epilogue -> MMA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accempty + 4);
  volatile int* cta_err = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.y;
  int mt, nt;
  tile_of(blockIdx.x, p.nmt, p.nnt, mt, nt);
  const int m0 = mt * BM, n0 = nt * BN;     // n0: first real column of D
  // Hermitian result: a tile whose complex columns all lie left of its first
  // row is wholly below the diagonal (filled afterwards from the upper part)
  if (p.herm_upper && (n0 >> 1) + BN / 2 - 1 < m0) return;
  // lower part wanted: a tile whose complex columns all lie right of its last
  // row is wholly above the diagonal
  if (p.lower_only && (n0 >> 1) > m0 + BM - 1) return;
  // triangular operands (f32 mode): the complex K range [kmin, kmax) this
  // tile needs; a K-block is run when it meets that range in the real or the
  // imaginary half of K' (every role skips the same blocks)
  int kmin = 0, kmax = p.kp;
  if (p.tri_a_upper) kmin = m0;
  if (p.tri_a_lower) kmax = min(kmax, m0 + BM);
  if (p.tri_b_upper) kmax = min(kmax, (n0 >> 1) + BN / 2);
  const bool tri = kmin > 0 || kmax < p.kp;
  auto kb_needed = [&](int kb) {
    if (!tri) return true;
    const int lo = kb * BK, hi = lo + BK;
    return (lo < kmax && hi > kmin) || (lo < p.kp + kmax && hi > p.kp + kmin);
  };
  // K-blocks that run, of which kF32Span share the accumulators (f32 mode)
  int needed = p.kblocks;
  if (MODE == 1 && tri) {
    needed = 0;
    for (int kb = 0; kb < p.kblocks; ++kb) needed += kb_needed(kb);
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_SLOTS; ++s) {
      mbar_init(&fullA[s], 1);
      mbar_init(&emptyA[s], 1);
      mbar_init(&fullB[s], 1);
      mbar_init(&emptyB[s], 1);
    }
    for (int s = 0; s < NACC; ++s) {
      mbar_init(&accfull[s], 1);
      mbar_init(&accempty[s], kEpiWarps);
    }
    *cta_err = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == PRODUCER_WARP) {
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB) : "memory");
      int basea = 0, baseb = 0;         // slots of this K-step's tile 0
      uint32_t pha = 0, phb = 0;        // their wrap-around parities
      const int span = p.kspan - 1;     // 0 or 1
      uint32_t seen[2] = {0u, 0u}, par[2] = {0u, 0u};   // slots in use and the parities of their last copies
      bool ok = true;
      for (int kb = 0; kb < p.kblocks && ok; ++kb) {
        if (!kb_needed(kb)) continue;
        for (int i = 0; i < p.nload; ++i) {
          const int ld = p.load[i];
          if (ld >= 0) {
            int s = basea + ld;
            uint32_t ph = pha;
            while (s >= p.slots_a) { s -= p.slots_a; ph ^= 1u; }
            if (!mbar_wait(&emptyA[s], ph ^ 1u, cta_err, p.err, 1)) { ok = false; break; }
            mbar_expect_tx(&fullA[s], (uint32_t)kTileBytesA);
            const int pl = MODE == 0 ? ld >> span : ld, k0 = MODE == 0 ? (kb << span) + (ld & span) : kb;
            tma_load_3d(sA + s * kTileBytesA, &tmA, &fullA[s], k0 * BK, m0, b * p.planes_a + pl);
            seen[0] |= 1u << s;
            par[0] = (par[0] & ~(1u << s)) | (ph << s);
          } else {
            const int t = -1 - ld;
            int s = baseb + t;
            uint32_t ph = phb;
            while (s >= p.slots_b) { s -= p.slots_b; ph ^= 1u; }
            if (!mbar_wait(&emptyB[s], ph ^ 1u, cta_err, p.err, 1)) { ok = false; break; }
            mbar_expect_tx(&fullB[s], (uint32_t)TB);
            // f32 mode: B's planes from the last to the first
            const int pl = MODE == 0 ? t >> span : p.planes_b - 1 - t, k0 = MODE == 0 ? (kb << span) + (t & span) : kb;
            tma_load_3d(sB + s * TB, &tmB, &fullB[s], k0 * BK, n0, b * p.planes_b + pl);
            seen[1] |= 1u << s;
            par[1] = (par[1] & ~(1u << s)) | (ph << s);
          }
        }
        basea += p.planes_a * p.kspan;
        while (basea >= p.slots_a) { basea -= p.slots_a; pha ^= 1u; }
        baseb += p.planes_b * p.kspan;
        while (baseb >= p.slots_b) { baseb -= p.slots_b; phb ^= 1u; }
      }
      if (!ok) {
        // wait (bounded) for the copies still in flight before the CTA exits
        for (int s = 0; s < 2 * MAX_SLOTS; ++s) {
          const int o = s / MAX_SLOTS, q = s % MAX_SLOTS;
          if (!(seen[o] >> q & 1u)) continue;
          const unsigned long long t0 = now_ns();
          while (!mbar_try(o ? &fullB[q] : &fullA[q], par[o] >> q & 1u) && (long long)(now_ns() - t0) < kWaitNs) {
          }
        }
      }
    }
  } else if (warp == MMA_WARP) {
    // the whole warp runs the schedule, so that slots and descriptors stay in
    // uniform registers; one elected lane issues
    const bool leader = elect_one();
    const uint32_t a_lo = (smem_u32(sA) >> 4) | kDescLo, b_lo = (smem_u32(sB) >> 4) | kDescLo;
    int basea = 0, baseb = 0;           // slots of this K-step's tile 0
    uint32_t pha = 0, phb = 0;
    bool ok = true;
    int buf = 0;                        // accumulator of the current group and its wrap-around parity
    uint32_t phacc = 1;
    TcPair pr = p.pairs[0];             // the next pair is read while this one is issued
    int nth = 0;                        // K-steps run before this one
    for (int kb = 0; kb < p.kblocks && ok; ++kb) {
      if (!kb_needed(kb)) continue;
      // f32 mode: first and last K-block of the accumulators
      const bool opens = MODE == 0 || nth % kF32Span == 0;
      const bool closes = MODE == 0 || nth % kF32Span == kF32Span - 1 || nth == needed - 1;
      if (MODE == 1) ++nth;
      for (int i = 0; i < p.npairs; ++i) {
        const int all = pr.flags;
        const int flags = MODE == 0 ? all : all & ~((opens ? 0 : kPairStart) | (closes ? 0 : kPairEnd));
        int sa = basea + pr.pa, sb = baseb + pr.pb;
        pr = p.pairs[i + 1 < p.npairs ? i + 1 : 0];
        uint32_t fa = pha, fb = phb;
#pragma unroll
        for (int w = 0; w < 2; ++w) {   // a step has fewer tiles than two turns of the ring
          if (sa >= p.slots_a) { sa -= p.slots_a; fa ^= 1u; }
          if (sb >= p.slots_b) { sb -= p.slots_b; fb ^= 1u; }
        }
        if (flags & (kPairStart | kPairFirstA | kPairFirstB)) {
          if (flags & kPairStart) ok = mbar_wait(&accempty[buf], phacc, cta_err, p.err, 2);
          if (ok && (flags & kPairFirstA)) ok = mbar_wait(&fullA[sa], fa, cta_err, p.err, 3);
          if (ok && (flags & kPairFirstB)) ok = mbar_wait(&fullB[sb], fb, cta_err, p.err, 3);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          tc_fence_after();
        }
        const uint32_t dt = tmem + (uint32_t)(buf * BN);
        const uint32_t al = a_lo + sa * (kTileBytesA >> 4), bl = b_lo + sb * (TB >> 4);
        if (leader) {
          umma(dt, sdesc(al), sdesc(bl), IDESC, (flags & kPairStart) ? 0u : 1u);
#pragma unroll
          for (int k = 1; k < BK / 16; ++k)
            // +32 bytes of K per instruction: +2 in the descriptor's address field
            umma(dt, sdesc(al + 2 * k), sdesc(bl + 2 * k), IDESC, 1u);
          if (flags & kPairLastA) umma_commit(&emptyA[sa]);
          if (flags & kPairLastB) umma_commit(&emptyB[sb]);
          if (flags & kPairEnd) umma_commit(&accfull[buf]);
        }
        if (all & kPairEnd) {
          if (++buf == NACC) {
            buf = 0;
            if (MODE == 0 || closes) phacc ^= 1u;
          }
        }
      }
      __syncwarp();
      basea += p.planes_a * p.kspan;
      while (basea >= p.slots_a) { basea -= p.slots_a; pha ^= 1u; }
      baseb += p.planes_b * p.kspan;
      while (baseb >= p.slots_b) { baseb -= p.slots_b; phb ^= 1u; }
    }
  } else {
    // ---------------- epilogue warps ----------------
    const int q = warp & 3, h = warp >> 2;
    const int row = m0 + 32 * q + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(32 * q) << 16);
    bool ok = true;
    int g = 0;
    if (MODE == 0) {
      long long acc[CW];
#pragma unroll
      for (int j = 0; j < CW; ++j) acc[j] = 0;
      for (int kb = 0; kb < p.kblocks && ok; ++kb) {
        if (!kb_needed(kb)) continue;
        for (int i = 0; i < p.ngroups; ++i, ++g) {
          const int buf = g % NACC;
          ok = __all_sync(0xffffffffu, mbar_wait(&accfull[buf], (uint32_t)(g / NACC) & 1u, cta_err, p.err, 4));
          if (!ok) break;
          tc_fence_after();
          const int sh = p.shift[i];
          const uint32_t col = lane_addr + (uint32_t)(buf * BN + CW * h);
          const auto drain = [&](auto add) {
            // the next eight columns are under way while the last are added
            uint32_t rr[2][8];
            tmem_ld8(col, rr[0]);
#pragma unroll
            for (int part = 0; part < CW / 8; ++part) {
              tmem_ld_wait(rr[part & 1]);
              if (part < CW / 8 - 1) {
                tmem_ld8(col + 8 * (part + 1), rr[(part + 1) & 1]);
              } else {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&accempty[buf]);
              }
#pragma unroll
              for (int j = 0; j < 8; ++j) add(acc[8 * part + j], __float2int_rn(__uint_as_float(rr[part & 1][j])));
            }
          };
          if (sh > 30) {
            drain([sh](long long& x, int v) { x += (long long)v << sh; });
          } else if (sh >= 0) {
            // one 32 x 32 + 64-bit multiply-add per sum
            const int mul = 1 << sh;
            drain([mul](long long& x, int v) { x += (long long)v * mul; });
          } else {
            // low-order digit groups: rounded to the accumulator's unit (a
            // plain arithmetic shift would floor, a bias of half a unit per
            // drain that adds up over long K)
            const int half = 1 << (-sh - 1);
            drain([sh, half](long long& x, int v) { x += (v + half) >> (-sh); });
          }
        }
      }
      if (ok && row < p.m) {
        const int er = p.ea[(size_t)b * p.m + row] + p.base;
        const int c0 = (n0 >> 1) + CW / 2 * h;     // first complex column of this warp
        double2* out = reinterpret_cast<double2*>(p.c64) + (size_t)b * p.stride_c;
#pragma unroll
        for (int j = 0; j < CW / 2; ++j) {
          const int c = c0 + j;
          if (c < p.ncols) {
            const int e = er + p.fb[(size_t)b * p.ncols + c];
            out[(size_t)c * p.ldc + row] =
                make_double2(scalbn(__ll2double_rn(acc[2 * j]), e), scalbn(__ll2double_rn(acc[2 * j + 1]), e));
          }
        }
      }
    } else {
      // the sums of every kF32Span K-blocks are drained into register
      // accumulators with round-to-nearest adds, so that long sums of
      // like-signed terms are not left to the tensor core's accumulator alone
      float acc[CW];
#pragma unroll
      for (int j = 0; j < CW; ++j) acc[j] = 0.f;
      for (int kb = 0; kb < needed && ok; kb += kF32Span) {
        for (int i = 0; i < p.ngroups; ++i, ++g) {
          const int buf = g % NACC;
          ok = __all_sync(0xffffffffu, mbar_wait(&accfull[buf], (uint32_t)(g / NACC) & 1u, cta_err, p.err, 4));
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int part = 0; part < CW / 16; ++part) {
            uint32_t r[16];
            tmem_ld16(lane_addr + (uint32_t)(buf * BN + CW * h + 16 * part), r);
            tmem_ld_wait();
            if (part == CW / 16 - 1) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&accempty[buf]);
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[16 * part + j] += __uint_as_float(r[j]);
          }
        }
      }
      if (ok && row < p.m) {
        float2* out = reinterpret_cast<float2*>(p.c32) + (size_t)b * p.stride_c;
        const int cbase = (n0 >> 1) + CW / 2 * h;
#pragma unroll
        for (int j = 0; j < CW / 2; ++j) {
          const int c = cbase + j;
          if (c < p.ncols) {
            float2 v = make_float2(p.alpha * acc[2 * j], p.alpha * acc[2 * j + 1]);
            float2* o = out + (size_t)c * p.ldc + row;
            if (p.beta != 0.f) {
              const float2 old = *o;
              v.x += p.beta * old.x;
              v.y += p.beta * old.y;
            }
            *o = v;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
  }
}

// ---------------------------------------------------------------------------
// operand preparation
// ---------------------------------------------------------------------------
namespace {

__device__ __forceinline__ int expo_field(double x) { return (int)((__double_as_longlong(x) >> 52) & 0x7ff); }
__device__ __forceinline__ int expo_field(float x) { return (int)((__float_as_uint(x) >> 23) & 0xff); }
// smallest e with |x| < 2^e over a maximum exponent field E (normal numbers)
__device__ __forceinline__ int bound_expo(double, int E) { return E ? E - 1022 : -100000; }
__device__ __forceinline__ int bound_expo(float, int E) { return E ? E - 126 : -100000; }

// trunc(|x| 2^(W - e)) for |x| < 2^e, W <= 62; subnormals count as zero
__device__ __forceinline__ unsigned long long fixed_bits(double x, int e, int W) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffULL;
  const int E = (int)(u >> 52);
  if (E == 0) return 0ULL;
  const unsigned long long mant = (u & 0xfffffffffffffULL) | (1ULL << 52);
  const int sh = E - 1075 + W - e;
  if (sh >= 0) return mant << sh;
  if (sh <= -64) return 0ULL;
  return mant >> (-sh);
}
__device__ __forceinline__ unsigned long long fixed_bits(float x, int e, int W) {
  const unsigned u = __float_as_uint(x) & 0x7fffffffu;
  const int E = (int)(u >> 23);
  if (E == 0) return 0ULL;
  const unsigned long long mant = (unsigned long long)((u & 0x7fffffu) | (1u << 23));
  const int sh = E - 150 + W - e;
  if (sh >= 0) return mant << sh;
  if (sh <= -64) return 0ULL;
  return mant >> (-sh);
}

// Exponents of the lines (rows of op(A) or columns of B) that lie contiguous
// in the source: warp per line.
template <class T>
__global__ void line_expo_kernel(const T* __restrict__ src, long long sstride, int ld, int len, int lines, int nb,
                                 int* __restrict__ expo) {
  const size_t gw = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= (size_t)lines * nb) return;
  const int b = (int)(gw / lines), line = (int)(gw % lines);
  const T* s = src + (size_t)b * sstride + 2 * (size_t)line * ld;
  int E = 0;
  for (int i = lane; i < 2 * len; i += 32) E = max(E, expo_field(s[i]));
  for (int o = 16; o; o >>= 1) E = max(E, __shfl_xor_sync(0xffffffffu, E, o));
  if (lane == 0) expo[gw] = bound_expo(T(0), E);
}

// Exponents of the rows of a column-major source: block of 32 rows, the
// columns spread over its warps.
template <class T>
__global__ void __launch_bounds__(256) row_expo_kernel(const T* __restrict__ src, long long sstride, int ld, int rows,
                                                       int cols, int* __restrict__ expo) {
  __shared__ int part[8][32];
  const int b = blockIdx.y, r = blockIdx.x * 32 + threadIdx.x;
  const T* s = src + (size_t)b * sstride;
  int E = 0;
  if (r < rows) {
#pragma unroll 8
    for (int c = threadIdx.y; c < cols; c += 8) {
      E = max(E, expo_field(s[2 * ((size_t)c * ld + r)]));
      E = max(E, expo_field(s[2 * ((size_t)c * ld + r) + 1]));
    }
  }
  part[threadIdx.y][threadIdx.x] = E;
  __syncthreads();
  if (threadIdx.y == 0 && r < rows) {
#pragma unroll
    for (int w = 1; w < 8; ++w) E = max(E, part[w][threadIdx.x]);
    expo[(size_t)b * rows + r] = bound_expo(T(0), E);
  }
}

// x as signed fixed point (W bits of magnitude, truncated) plus the bias that
// turns its base-256 digits into balanced ones: digit 0 = biased >> 8 (np - 1),
// in [-256, 256], digit pl = ((biased >> 8 (np - 1 - pl)) & 255) - 128.
template <class T>
__device__ __forceinline__ long long biased_fixed(T x, int e, int nplanes) {
  const long long m = (long long)fixed_bits(x, e, nplanes * kBeta);
  long long bias = 0;
  for (int q = 0; q < nplanes - 1; ++q) bias = (bias << kBeta) + 128;
  return (x < T(0) ? -m : m) + bias;
}
__device__ __forceinline__ float digit_of(long long biased, int nplanes, int pl) {
  const int sh = kBeta * (nplanes - 1 - pl);
  return pl == 0 ? (float)(int)(biased >> sh) : (float)((int)((unsigned long long)biased >> sh & 255u) - 128);
}

// Plane values of one real number, plane after plane: digits, or the BF16
// pieces of an FP32 value.
template <class T>
struct PlaneValue {
  long long biased;
  float rest;
  __device__ __forceinline__ PlaneValue(T x, int e, int nplanes, bool digits)
      : biased(digits ? biased_fixed(x, e, nplanes) : 0), rest((float)x) {}
  __device__ __forceinline__ __nv_bfloat16 next(int nplanes, int pl, bool digits) {
    if (digits) return __float2bfloat16_rn(digit_of(biased, nplanes, pl));
    const __nv_bfloat16 v = __float2bfloat16_rn(rest);
    rest -= __bfloat162float(v);
    return v;
  }
};

// Left operand planes: out[b][pl][r][Kp] with columns [0, k) = Re op(A)(r, .),
// [kp, kp + k) = Im op(A)(r, .), zero elsewhere (Kp = 2 kp).  op(A) = src or
// src^H; tiles of 32 rows by 64 of K through shared memory so that reads and
// writes (two BF16 a lane) coalesce in both cases.
template <class T>
__global__ void __launch_bounds__(256) slice_a_kernel(const T* __restrict__ src, long long sstride, int ld, bool conj,
                                                      int m, int k, int kp, const int* __restrict__ ea,
                                                      int nplanes, bool digits, __nv_bfloat16* __restrict__ out) {
  __shared__ T tre[32][65], tim[32][65];
  const int b = blockIdx.z;
  const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 64;   // rows of op(A), K columns
  const int tx = threadIdx.x, ty = threadIdx.y;
  const T* s = src + (size_t)b * sstride;
  // tre[r][c] = op(A)(r0 + r, c0 + c)
  if (!conj) {
    for (int j = ty; j < 64; j += 8) {
      const int r = r0 + tx, c = c0 + j;
      const bool in = r < m && c < k;
      const size_t at = 2 * ((size_t)c * ld + r);
      tre[tx][j] = in ? s[at] : T(0);
      tim[tx][j] = in ? s[at + 1] : T(0);
    }
  } else {
    for (int j = ty; j < 32; j += 8)
      for (int x = tx; x < 64; x += 32) {
        const int r = r0 + j, c = c0 + x;
        const bool in = r < m && c < k;
        const size_t at = 2 * ((size_t)r * ld + c);
        tre[j][x] = in ? s[at] : T(0);
        tim[j][x] = in ? -s[at + 1] : T(0);
      }
  }
  __syncthreads();
  const size_t Kp = 2 * (size_t)kp;
  for (int j = ty; j < 32; j += 8) {
    const int r = r0 + j, c = c0 + 2 * tx;
    if (r >= m || c >= kp) continue;
    const int e = digits ? ea[(size_t)b * m + r] : 0;
    PlaneValue<T> x0(tre[j][2 * tx], e, nplanes, digits), x1(tre[j][2 * tx + 1], e, nplanes, digits);
    PlaneValue<T> y0(tim[j][2 * tx], e, nplanes, digits), y1(tim[j][2 * tx + 1], e, nplanes, digits);
    for (int pl = 0; pl < nplanes; ++pl) {
      __nv_bfloat16* o = out + (((size_t)b * nplanes + pl) * m + r) * Kp + c;
      *reinterpret_cast<__nv_bfloat162*>(o) = __nv_bfloat162(x0.next(nplanes, pl, digits), x1.next(nplanes, pl, digits));
      *reinterpret_cast<__nv_bfloat162*>(o + kp) =
          __nv_bfloat162(y0.next(nplanes, pl, digits), y1.next(nplanes, pl, digits));
    }
  }
}

// Right operand planes: out[b][pl][2c + (0|1)][Kp]: row 2c = [Re B(., c) | -Im B(., c)],
// row 2c+1 = [Im B(., c) | Re B(., c)]; thread per column and two K indices.
template <class T>
__global__ void slice_b_kernel(const T* __restrict__ src, long long sstride, int ld, int k, int n, int kp,
                               const int* __restrict__ fb, int nplanes, bool digits, int nb,
                               __nv_bfloat16* __restrict__ out) {
  const int half = kp >> 1;
  const size_t per = (size_t)half * n, total = per * nb;
  const size_t Kp = 2 * (size_t)kp;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int b = (int)(idx / per);
    const size_t q = idx - (size_t)b * per;
    const int c = (int)(q / half), r = 2 * (int)(q - (size_t)c * half);
    const T* s = src + (size_t)b * sstride + 2 * ((size_t)c * ld + r);
    const T v[4] = {r < k ? s[0] : T(0), r < k ? s[1] : T(0), r + 1 < k ? s[2] : T(0), r + 1 < k ? s[3] : T(0)};
    const int e = digits ? fb[(size_t)b * n + c] : 0;
    PlaneValue<T> x0(v[0], e, nplanes, digits), y0(v[1], e, nplanes, digits);
    PlaneValue<T> x1(v[2], e, nplanes, digits), y1(v[3], e, nplanes, digits);
    for (int pl = 0; pl < nplanes; ++pl) {
      const __nv_bfloat162 re(x0.next(nplanes, pl, digits), x1.next(nplanes, pl, digits));
      const __nv_bfloat162 im(y0.next(nplanes, pl, digits), y1.next(nplanes, pl, digits));
      __nv_bfloat162* o =
          reinterpret_cast<__nv_bfloat162*>(out + (((size_t)b * nplanes + pl) * 2 * n + 2 * (size_t)c) * Kp + r);
      o[0] = re;
      o[half] = __hneg2(im);
      o[kp] = im;
      o[kp + half] = re;
    }
  }
}

// Right operand planes of B = src^H (src n x k, column-major), FP32 pieces: the
// rows of slice_b_kernel, 32 x 32 tiles through shared memory.
__global__ void __launch_bounds__(256) slice_bh_kernel(const float* __restrict__ src, long long sstride, int ld, int k,
                                                       int n, int kp, __nv_bfloat16* __restrict__ out) {
  __shared__ float2 tile[32][33];                         // [column of B][K index]
  const int b = blockIdx.z, c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const float2* s = reinterpret_cast<const float2*>(src + (size_t)b * sstride);
  for (int j = ty; j < 32; j += 8) {
    const int c = c0 + tx, r = r0 + j;
    tile[tx][j] = (c < n && r < k) ? s[(size_t)r * ld + c] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const size_t Kp = 2 * (size_t)kp;
  for (int j = ty; j < 32; j += 8) {
    const int c = c0 + j, r = r0 + tx;
    if (c >= n || r >= kp) continue;
    float vr = tile[j][tx].x, vi = -tile[j][tx].y;
    for (int pl = 0; pl < 3; ++pl) {
      const __nv_bfloat16 pr = __float2bfloat16_rn(vr), pi = __float2bfloat16_rn(vi);
      __nv_bfloat16* o = out + (((size_t)b * 3 + pl) * 2 * n + 2 * (size_t)c) * Kp;
      o[r] = pr;
      o[kp + r] = __float2bfloat16_rn(-__bfloat162float(pi));
      o[Kp + r] = pi;
      o[Kp + kp + r] = pr;
      vr -= __bfloat162float(pr);
      vi -= __bfloat162float(pi);
    }
  }
}

int grid_of(size_t n) { return (int)std::min<size_t>((n + 255) / 256, 152 * 16); }

// C(r, c) = conj(C(c, r)) for r > c: the strict lower triangle of a
// Hermitian batch [nb][n][n] (complex FP64, column-major) from its upper one.
__global__ void mirror_lower_kernel(double2* __restrict__ C, int n, int nb) {
  __shared__ double2 tile[32][33];
  const int b = blockIdx.z;
  const int bx = blockIdx.x, by = blockIdx.y;   // tile (rows by, columns bx) of the lower part
  if (bx > by) return;
  double2* Cb = C + (size_t)b * n * n;
  const int tx = threadIdx.x, ty = threadIdx.y;
  // read the upper tile (rows bx, columns by), write its conjugate transpose
  for (int j = ty; j < 32; j += 8) {
    const int r = bx * 32 + tx, c = by * 32 + j;
    if (r < n && c < n) tile[j][tx] = Cb[(size_t)c * n + r];
  }
  __syncthreads();
  for (int j = ty; j < 32; j += 8) {
    const int r = by * 32 + tx, c = bx * 32 + j;     // lower element (r, c) = conj(upper (c, r))
    if (r < n && c < n && r > c) {
      const double2 u = tile[tx][j];
      Cb[(size_t)c * n + r] = make_double2(u.x, -u.y);
    }
  }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against libcuda).
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(p);
  });
  return fn;
}

// 3-D BF16 tensor [planes][rows][Kp] (K contiguous), box 64 x box_rows x 1,
// 128-byte swizzle; rows past `rows` read as zero.
int make_map(CUtensorMap* map, const void* base, size_t Kp, size_t rows, size_t planes, int box_rows) {
  EncodeFn fn = encode_fn();
  if (!fn) return fail(OLC_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (Kp * 2) % 16)
    return fail(OLC_ERR_CUDA, "tensor map operand not 16-byte aligned");
  const cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, (cuuint64_t)planes};
  const cuuint64_t strides[2] = {(cuuint64_t)(Kp * 2), (cuuint64_t)(Kp * 2 * rows)};
  const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(OLC_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  return OLC_OK;
}

int* g_err = nullptr;   // device error word shared by the launches of this process
std::mutex g_err_mu;

// First / last uses of the tiles, the tile slots and the staging order.  The
// slots fill 224 KB: fixed mode 14 of 16 KB, a slot per tile where a K-step has
// no more tiles than that (7 + 7 digits), else rings (3 + 6 digits in two
// K-blocks: the three-digit operand's six tiles live throughout, a window of
// six of the other's); f32 mode rings of 6 of 16 KB and 4 of 32 KB.
constexpr int kFixedSlots = 14;
// the most a launch of either mode takes: the limit every launch sets (a limit set
// to the launch's own need could be lowered by another thread before it)
constexpr int kSmemMax = kFixedSlots * kTileBytesA + 512 + 1024;
void plan_pairs(TcParams& p, int mode) {
  for (int i = 0; i < p.npairs; ++i) {
    TcPair& pr = p.pairs[i];
    bool firstA = true, firstB = true, lastA = true, lastB = true;
    for (int j = 0; j < p.npairs; ++j) {
      if (j < i) {
        firstA &= p.pairs[j].pa != pr.pa;
        firstB &= p.pairs[j].pb != pr.pb;
      } else if (j > i) {
        lastA &= p.pairs[j].pa != pr.pa;
        lastB &= p.pairs[j].pb != pr.pb;
      }
    }
    pr.flags = (int16_t)((pr.flags & (kPairStart | kPairEnd)) | (firstA ? kPairFirstA : 0) | (firstB ? kPairFirstB : 0) |
                         (lastA ? kPairLastA : 0) | (lastB ? kPairLastB : 0));
  }
  if (p.kspan == 2) p.kblocks = (p.kblocks + 1) / 2;     // a step past K' reads zeros
  const int ta = p.planes_a * p.kspan, tb = p.planes_b * p.kspan;
  const bool resident = mode == 0 && ta + tb <= kFixedSlots && ta <= MAX_SLOTS && tb <= MAX_SLOTS;
  if (resident) {
    p.slots_a = ta;
    p.slots_b = tb;
  } else if (mode == 0) {
    p.slots_a = p.planes_a < p.planes_b ? 6 : p.planes_a > p.planes_b ? 8 : 7;
    p.slots_b = kFixedSlots - p.slots_a;
  } else {
    p.slots_a = 6;
    p.slots_b = 4;
  }
  // staging order: a slot per tile is free again after its tile's last use in
  // the step before; slots in rings are filled in the order of first use
  p.nload = 0;
  const int want = resident ? kPairLastA : kPairFirstA, wantb = resident ? kPairLastB : kPairFirstB;
  for (int i = 0; i < p.npairs; ++i) {
    if (p.pairs[i].flags & want) p.load[p.nload++] = p.pairs[i].pa;
    if (p.pairs[i].flags & wantb) p.load[p.nload++] = (int8_t)(-1 - p.pairs[i].pb);
  }
}

int launch(olc_context* ctx, int mode, const void* dA, const void* dB, int planes_a, int planes_b, size_t Kp,
           int m, int nreal, int nb, TcParams p, int stage) {
  cudaStream_t st = ctx->stream;
  int s;
  {
    std::lock_guard<std::mutex> lk(g_err_mu);
    if (!g_err) {
      if ((s = cuda_check(cudaMalloc(&g_err, sizeof(int)), "tc error word"))) return s;
      if ((s = cuda_check(cudaMemset(g_err, 0, sizeof(int)), "tc error word"))) return s;
    }
  }
  const int BN = mode == 0 ? 128 : 256;
  CUtensorMap ta, tb;
  if ((s = make_map(&ta, dA, Kp, (size_t)m, (size_t)planes_a * nb, BM))) return s;
  if ((s = make_map(&tb, dB, Kp, (size_t)nreal, (size_t)planes_b * nb, BN))) return s;
  p.planes_a = planes_a;
  p.planes_b = planes_b;
  p.nmt = (m + BM - 1) / BM;
  p.nnt = (nreal + BN - 1) / BN;
  p.kblocks = (int)(Kp / BK);
  p.kp = (int)(Kp / 2);
  p.err = g_err;
  plan_pairs(p, mode);
  const dim3 grid((unsigned)(p.nmt * p.nnt), (unsigned)nb);
  const int smem = smem_total(mode, p.slots_a, p.slots_b);     // at most kSmemMax
  if (mode == 0) {
    if ((s = cuda_check(cudaFuncSetAttribute(tc_gemm_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax),
                        "tc smem")))
      return s;
    tc_gemm_kernel<0><<<grid, kThreads, smem, st>>>(ta, tb, p);
  } else {
    if ((s = cuda_check(cudaFuncSetAttribute(tc_gemm_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax),
                        "tc smem")))
      return s;
    tc_gemm_kernel<1><<<grid, kThreads, smem, st>>>(ta, tb, p);
  }
  count_launch();
  double frac = 1.0;
  if (p.herm_upper || p.lower_only) {
    long long done = 0;
    for (int mt = 0; mt < p.nmt; ++mt)
      for (int nt = 0; nt < p.nnt; ++nt)
        done += p.herm_upper ? ((nt * BN) / 2 + BN / 2 - 1 >= mt * BM) : ((nt * BN) / 2 <= mt * BM + BM - 1);
    frac = (double)done / ((double)p.nmt * p.nnt);
  }
  add_work(ctx, stage, 2.0 * m * (double)nreal * (double)Kp * (p.npairs / p.kspan) * nb * frac, 0.0);
  return cuda_check(cudaGetLastError(), "tc_gemm launch");
}

}  // namespace

// Kept-digit plan of a fixed-point product: na / nb digits of A / B,
// pairs (s, t) with s + t <= T kept, T the smallest with the dropped part
// below 2^-(prec + 2) of the scale product.
void fixed_plan(int bits_a, int bits_b, int prec, int* na, int* nbd, int* T) {
  *na = (bits_a + kBeta - 1) / kBeta;
  *nbd = (bits_b + kBeta - 1) / kBeta;
  // dropped pairs with s + t >= T + 1 weigh at most ~4 * 2^(-beta (T + 1))
  int t = 0;
  while (kBeta * (t + 1) - 2 < prec + 2) ++t;
  *T = std::min(t, *na + *nbd - 2);
}

int read_error(int* code) {
  *code = 0;
  if (!g_err) return OLC_OK;
  int s = cuda_check(cudaMemcpy(code, g_err, sizeof(int), cudaMemcpyDeviceToHost), "tc error read");
  if (!s && *code) cudaMemset(g_err, 0, sizeof(int));
  return s;
}

template <class TA, class TB>
int zgemm_fixed(olc_context* ctx, int m, int n, int k, const TA* A, long long sA, int lda, bool conjA, int bits_a,
                const TB* B, long long sB, int ldb, int bits_b, double* C, int nb, int stage, bool hermitian) {
  if (hermitian && m != n) return fail(OLC_ERR_ARG, "hermitian product must be square");
  cudaStream_t st = ctx->stream;
  int na, nbd, T;
  // the product is wanted to the precision of the wider operand (the
  // narrower one is represented exactly or as a consistent basis change)
  fixed_plan(bits_a, bits_b, std::max(bits_a, bits_b), &na, &nbd, &T);
  const int kp = (k + 31) & ~31;
  const size_t Kp = 2 * (size_t)kp;
  TcParams plan{};
  // 64-bit fixed point: unit 2^(L - beta (T + 2)) of the scale product
  const double mag = kBeta * T + 2 * kBeta + std::log2(1.03 * (double)Kp);
  const int L = std::max(0, (int)std::ceil(mag - 62.0));
  // Up to three pairs a weight, the group's sum stays an exact integer over two
  // K-blocks (128 (2 2^15 + 2^14) < 2^24): half the drains, which bound this mode
  // (a drain of the 128 x 128 tile takes the epilogue 1600 clocks, three pairs of
  // one K-block the tensor cores 950).
  plan.kspan = std::min(na, nbd) <= 3 ? 2 : 1;
  // One group per weight s + t = d <= T.  Where every tile of a K-step has a slot of
  // its own, from the highest weight down and its pairs from the middle out: the
  // low-order tiles retire first and the tiles that the next step begins with long
  // before its first pair (from weight 0 up all tiles retired in the last group and
  // every step began with a wait for its copies).  In
  // rings the pairs run from weight 0 up, A's new plane first and B's last, so that
  // tiles are used in the order 0, 1, ..
  const bool down = (na + nbd) * plan.kspan <= kFixedSlots && std::max(na, nbd) * plan.kspan <= MAX_SLOTS;
  for (int g = 0; g <= T; ++g) {
    const int d = down ? T - g : g, first = plan.npairs;
    int order[32], cnt = 0;
    for (int q = std::min(d, na - 1); q >= 0 && d - q < nbd; --q) order[cnt++] = q;
    if (down)
      std::stable_sort(order, order + cnt, [d](int x, int y) { return std::abs(2 * x - d) < std::abs(2 * y - d); });
    for (int j = 0; j < cnt; ++j)
      for (int q = 0; q < plan.kspan; ++q) {
        if (plan.npairs == kMaxPairs || plan.ngroups == kMaxGroups)
          return fail(OLC_ERR_UNSUPPORTED, "fixed-point product: too many digit pairs");
        plan.pairs[plan.npairs++] =
            TcPair{(int8_t)(plan.kspan * order[j] + q), (int8_t)(plan.kspan * (d - order[j]) + q), 0};
      }
    if (plan.npairs == first) continue;
    plan.pairs[first].flags |= kPairStart;
    plan.pairs[plan.npairs - 1].flags |= kPairEnd;
    // a group's sum is below 2^24, so that a shift to the right by 26 and more gives
    // 0, and one past 30 (K of a million) may stop there: half a unit fits 32 bits
    plan.shift[plan.ngroups++] = (int16_t)std::max(kBeta * (T - d) - L, -30);
  }
  // batch chunk: digit planes below ~8 GB
  const size_t per_b = 2 * Kp * ((size_t)na * m + (size_t)nbd * 2 * n);
  const int chunk = (int)std::max<size_t>(1, std::min<size_t>(nb, (8ULL << 30) / std::max<size_t>(per_b, 1)));
  __nv_bfloat16 *wa = nullptr, *wb = nullptr;
  int *ea = nullptr, *fb = nullptr;
  int s;
  if ((s = cuda_check(ctx_malloc(ctx, (void**)&wa, 2 * Kp * na * (size_t)m * chunk, st), "malloc digits A")))
    return s;
  if ((s = cuda_check(ctx_malloc(ctx, (void**)&wb, 2 * Kp * nbd * 2 * (size_t)n * chunk, st), "malloc digits B")))
    return s;
  if ((s = cuda_check(ctx_malloc(ctx, (void**)&ea, 4ULL * chunk * m, st), "malloc ea"))) return s;
  if ((s = cuda_check(ctx_malloc(ctx, (void**)&fb, 4ULL * chunk * n, st), "malloc fb"))) return s;
  StageScope scope(ctx, stage, 0);
  for (int b0 = 0; b0 < nb; b0 += chunk) {
    const int cb = std::min(chunk, nb - b0);
    const TA* Ab = A + (size_t)b0 * sA;
    const TB* Bb = B + (size_t)b0 * sB;
    if (conjA)
      line_expo_kernel<TA><<<(int)(((size_t)m * cb * 32 + 255) / 256), 256, 0, st>>>(Ab, sA, lda, k, m, cb, ea);
    else
      row_expo_kernel<TA><<<dim3((m + 31) / 32, cb), dim3(32, 8), 0, st>>>(Ab, sA, lda, m, k, ea);
    line_expo_kernel<TB><<<(int)(((size_t)n * cb * 32 + 255) / 256), 256, 0, st>>>(Bb, sB, ldb, k, n, cb, fb);
    slice_a_kernel<TA><<<dim3((m + 31) / 32, (kp + 63) / 64, cb), dim3(32, 8), 0, st>>>(
        Ab, sA, lda, conjA, m, k, kp, ea, na, true, wa);
    slice_b_kernel<TB><<<grid_of((size_t)kp / 2 * n * cb), 256, 0, st>>>(Bb, sB, ldb, k, n, kp, fb, nbd, true, cb, wb);
    scope.add_launches(5);
    TcParams p = plan;
    p.m = m;
    p.ncols = n;
    p.ldc = m;
    p.stride_c = (long long)m * n;
    p.c64 = C + 2 * (size_t)b0 * m * n;
    p.ea = ea;
    p.fb = fb;
    p.base = L - kBeta * (T + 2);
    p.herm_upper = hermitian ? 1 : 0;
    if ((s = launch(ctx, 0, wa, wb, na, nbd, Kp, m, 2 * n, cb, p, stage))) return s;
    if (hermitian) {
      StageScope ms(ctx, stage, 1);
      mirror_lower_kernel<<<dim3((n + 31) / 32, (n + 31) / 32, cb), dim3(32, 8), 0, st>>>(
          reinterpret_cast<double2*>(C + 2 * (size_t)b0 * m * n), n, cb);
    }
  }
  cudaFreeAsync(wa, st);
  cudaFreeAsync(wb, st);
  cudaFreeAsync(ea, st);
  cudaFreeAsync(fb, st);
  return cuda_check(cudaGetLastError(), "fixed-point tensor-core product");
}

int cgemm_f32(olc_context* ctx, int m, int n, int k, const float* A, long long sA, int lda, bool conjA,
              const float* B, long long sB, int ldb, float alpha, float beta, float* C, long long sC, int ldc,
              int nb, int stage, bool lower, int tri, bool conjB) {
  cudaStream_t st = ctx->stream;
  const int kp = (k + 31) & ~31;
  const size_t Kp = 2 * (size_t)kp;
  // the six piece pairs of weight 2^-16 and above, and with OLC_F32_PAIRS=9 the
  // three below as well: one plane of B (the wide tile) after the other, the
  // low-order one first, so that a slot of B is free again after its own pairs
  // (the second index counts B's planes from the last: pairs (a, 2 - b)); the
  // leading pair last, a group of its own
  static const int8_t six[6][2] = {{0, 0}, {0, 1}, {1, 1}, {1, 2}, {2, 2}, {0, 2}};
  static const int8_t nine[9][2] = {{0, 0}, {1, 0}, {2, 0}, {0, 1}, {1, 1}, {2, 1}, {1, 2}, {2, 2}, {0, 2}};
  TcParams plan{};
  const char* pv = std::getenv("OLC_F32_PAIRS");
  plan.npairs = pv && std::atoi(pv) == 9 ? 9 : 6;
  for (int i = 0; i < plan.npairs; ++i) {
    const int8_t* q = plan.npairs == 9 ? nine[i] : six[i];
    plan.pairs[i] = TcPair{q[0], q[1], 0};
  }
  plan.pairs[0].flags |= kPairStart;
  plan.pairs[plan.npairs - 2].flags |= kPairEnd;
  plan.pairs[plan.npairs - 1].flags |= kPairStart | kPairEnd;
  plan.ngroups = num_acc<1>();     // one accumulator each: a group's stays its own over K-blocks
  plan.kspan = 1;
  const size_t per_b = 2 * Kp * 3 * ((size_t)m + 2 * (size_t)n);
  const int chunk = (int)std::max<size_t>(1, std::min<size_t>(nb, (8ULL << 30) / std::max<size_t>(per_b, 1)));
  __nv_bfloat16 *wa = nullptr, *wb = nullptr;
  int s;
  if ((s = cuda_check(ctx_malloc(ctx, (void**)&wa, 2 * Kp * 3 * (size_t)m * chunk, st), "malloc pieces A")))
    return s;
  if ((s = cuda_check(ctx_malloc(ctx, (void**)&wb, 2 * Kp * 3 * 2 * (size_t)n * chunk, st), "malloc pieces B")))
    return s;
  StageScope scope(ctx, stage, 0);
  for (int b0 = 0; b0 < nb; b0 += chunk) {
    const int cb = std::min(chunk, nb - b0);
    const float* Ab = A + (size_t)b0 * sA;
    const float* Bb = B + (size_t)b0 * sB;
    slice_a_kernel<float><<<dim3((m + 31) / 32, (kp + 63) / 64, cb), dim3(32, 8), 0, st>>>(
        Ab, sA, lda, conjA, m, k, kp, nullptr, 3, false, wa);
    if (conjB)
      slice_bh_kernel<<<dim3((n + 31) / 32, (kp + 31) / 32, cb), dim3(32, 8), 0, st>>>(Bb, sB, ldb, k, n, kp, wb);
    else
      slice_b_kernel<float><<<grid_of((size_t)kp / 2 * n * cb), 256, 0, st>>>(Bb, sB, ldb, k, n, kp, nullptr, 3, false,
                                                                              cb, wb);
    scope.add_launches(2);
    TcParams p = plan;
    p.m = m;
    p.ncols = n;
    p.ldc = ldc;
    p.stride_c = sC / 2;
    p.c32 = C + (size_t)b0 * sC;
    p.alpha = alpha;
    p.beta = beta;
    p.lower_only = lower ? 1 : 0;
    p.tri_a_upper = (tri & kTriAUpper) != 0;
    p.tri_a_lower = (tri & kTriALower) != 0;
    p.tri_b_upper = (tri & kTriBUpper) != 0;
    if ((s = launch(ctx, 1, wa, wb, 3, 3, Kp, m, 2 * n, cb, p, stage))) return s;
  }
  cudaFreeAsync(wa, st);
  cudaFreeAsync(wb, st);
  return cuda_check(cudaGetLastError(), "FP32-accurate tensor-core product");
}

template int zgemm_fixed<double, float>(olc_context*, int, int, int, const double*, long long, int, bool, int,
                                        const float*, long long, int, int, double*, int, int, bool);
template int zgemm_fixed<float, double>(olc_context*, int, int, int, const float*, long long, int, bool, int,
                                        const double*, long long, int, int, double*, int, int, bool);
template int zgemm_fixed<double, double>(olc_context*, int, int, int, const double*, long long, int, bool, int,
                                         const double*, long long, int, int, double*, int, int, bool);

}  // namespace tc
}  // namespace olc
