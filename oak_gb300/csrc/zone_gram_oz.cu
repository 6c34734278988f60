// The plain (FP64) form's products on the tensor cores, ensembles of up to 64 members: K1 + K2
// (selection and the Gram, k_zone_gram_oz) and E4 of the eigensolve (the square-root transform
// T = U (I+L)^-1/2 U^T Omega, k_zone_tsym_oz, further below).
//
// Selection and weights are those of zone_gram.cu (assimilation.F90:3683-3771): the relevance
// decisions of the tensor-core mixed kernel (FP32 distances away from the thresholds, the
// reference's FP64 evaluation near them; the selected set is identical to the plain form's),
// and for every selected observation the FP64 weight w of zone_gram.cu (FP64 distance,
// exp(-(d/L)^2) or locfun(d/L)). The Gram matrix G = HS_sel^T diag(c) HS_sel (rrsqrt.F90:135,
// c = w (w / r), DCDCovar of rrsqrt.F90:395) is formed as X^T X with X = diag(|w| / sqrt(r))
// HS_sel, in FP64, as an exact integer product on the FP16 tensor cores (the slice splitting
// of Ozaki et al., "Error-free transformations of matrix multiplication by using fast routines
// of matrix multiplication and its applications", Numer. Algorithms 59 (2012)):
//
//   Column a of X gets a fixed exponent E_a with |X_qa| <= 2^E_a for every observation q (from
//   max_q |HS_qa| / sqrt(r_q), once per call), so F_qa = round(X_qa 2^(54 - E_a)) is
//   an integer below 2^54 in magnitude, taken from the FP64 bit pattern with integer
//   operations. F is written in 7 balanced base-256 digits, F = sum_p d_p 256^(6-p) with
//   d_0 in [-64, 64] and d_1..d_6 in [-128, 127] (the bytes of F + 0x80808080808080 minus 128);
//   every digit is exact in FP16.
//   Then G_ab = 2^(E_a + E_b - 12) sum_L 256^-L level_L(a, b), level_L = sum_{p+q=L} D_p^T D_q
//   (D_p the digit-p matrix of the zone's rows), for levels 0..7. Levels 8..12 are left out: a
//   row adds at most 5 x 2^14 x 256^4 = 1.25 x 2^48 to level 8 against 2^108 = F_a F_b at the
//   column bounds, 2^-59.7 of 2^(E_a + E_b).
//   A K-tile of 64 observations is staged as 7 digit slices (64 members x 64 observations of
//   FP16, K-major, 128-byte swizzle), the buffer's eighth slice is zero (D_7), and each K-step of
//   16 observations issues tcgen05.mma kind::f16 (FP16 x FP16 -> FP32) with A = [D_p ; D_(p+1)]
//   (M = 128), p = 0, 2, 4, 6, and B = D_0 .. D_(7-p) into the column blocks p .. 7: block L then
//   holds level L's products with even p in lanes 0-63 and level L + 1's with odd p in lanes
//   64-127. Both halves of every MMA are used: 20 block columns a K-step, 7 MMAs of up to 256.
//   Exactness: a digit product is at most 2^14 (2^13 with d_0) and a half sums at most 4 a row,
//   so the FP32 sums stay exact integers up to 2^24 over 256 observations; the accumulators are
//   read every 4 K-tiles and added into two 64-bit integer sums, levels 0..3 and levels 4..7 (in
//   units of level 6: level 7 is rounded there, 2^-60 of 2^(E_a + E_b) a read). At the end of
//   the zone G = 2^(E_a + E_b - 36) v_hi + 2^(E_a + E_b - 60) v_lo, each converted once to FP64.
//   The error of G is therefore the rounding of X to the fixed point (2^-54 of its column scale)
//   and the last addition, not the length of the sums (the CPU model of these steps,
//   tests/test_slice_products_model.py, checks the bound and the budgets of the scheme that
//   stops one level earlier).
//
// The innovation projection g = X^T (sqrt(c) d) (rrsqrt.F90:142) is accumulated in FP64 by the
// staging threads (one FMA per staged element).
//
// What bounds it: the worker warps' integer work and FP64 pipe, in turn with each other, not
// the tensor cores (busy under 15% of the time) and not memory. The CTA (one per SM: its shared
// memory and the 512 tensor-memory columns admit no second one) is split by role:
//   16 worker warps   candidates are tested 512 at a time (a zone's cell-row ranges flattened
//                     into one index space); selected observations go to a ring, their FP64
//                     weights are computed one thread an entry (|w| / sqrt(r) as significand and
//                     exponent, so that staging is one 64 x 64-bit integer product a value;
//                     w^2 / r (yo - Hxf)); full K-tiles are staged into two shared buffers;
//   the issuer warp   waits for a staged buffer, issues its 28 MMAs and the commit, so no worker
//                     spends its time on descriptors;
//   the scout warp    takes the next zone from the counter and evaluates its FP64 set-up
//                     (projection, length scales, cell range) while the workers are at this one.
// Measured on 64,800 zones of a 360 x 180 global grid, N = 50, 3,000 observations, against the
// same kernel with levels 0..6 in 44 MMAs of which half of each was unused, issued by a worker,
// the set-up in line and the FP64 multiply-and-split staging: 24.5 ms before, 20.9 ms now; 7,200
// zones with N = 64: 2.55 ms before, 2.13 ms now. Of about 95,000 cycles a zone 28,000 are staging, 25,000
// accumulator reads, 24,000 selection and ranges, 10,000 FP64 weights. Reading the accumulators
// every 8 K-tiles instead of 4 measured the same.
// Every wait for the tensor core is bounded; on expiry the kernel records ZST_TIMEOUT, stops taking
// zones, waits (bounded) for its MMAs and frees its tensor memory.
#include <cuda_runtime.h>
#include <math.h>

#include "oakg_internal.cuh"
#include "oz_slices.cuh"
#include "selection.cuh"

namespace oakg {

namespace {

constexpr int kThreads = 512;
constexpr int NB = 64;                 // padded ensemble width
constexpr int KT = 64;                 // observations per K-tile (128 bytes of FP16 a row)
constexpr int kRing = 1024;            // selected-observation ring (power of two)
constexpr uint32_t kSliceBytes = 64u * 128u;         // one digit slice of a K-tile
constexpr uint32_t kBufBytes = 8 * kSliceBytes;  // one K-tile buffer: the digits and a zero slice
constexpr uint32_t kTmemCols = 512;
constexpr int kFlushTiles = 4;         // K-tiles between accumulator reads (256 observations)
constexpr int kTri = NB * (NB + 1) / 2;
constexpr int kLdG = NB + 1;
constexpr int kStageGroups = kThreads / NB;  // threads a member in the staging (8-obs chunks)
static_assert(KT == 8 * kStageGroups, "a chunk of 8 observations a thread");
// dynamic shared memory: alignment slack, two K-tile buffers, the integer level sums (lower
// triangle) and the FP64 innovation partials
constexpr size_t kDynSmem = 1024 + 2 * (size_t)kBufBytes + 2 * (size_t)kTri * sizeof(long long) +
                            kStageGroups * NB * sizeof(double);

// a zone's set-up, by the scout warp
struct OzZone {
  double zu, zv, L, Rmax, iL;
  sel::ZoneCell32 zc;  // the zone's cell-relative FP32 coordinates (read by broadcast)
  sel::ScanRange sr;   // the zone's cell range
  int32_t w, zl, z;
};

struct OzShared {
  int32_t ring_q[kRing];
  unsigned long long ring_m[kRing];  // |w| / sqrt(r_q): significand << 11 (0 for a zero)
  int32_t ring_e[kRing];             // and its biased exponent
  double ring_t[kRing];  // w^2 / r_q (yo - Hxf)_q
  OzZone zone[2];
  unsigned long long done[2];           // a buffer's MMAs complete
  int32_t first[2];                     // the buffer's tile starts the accumulators
  int32_t warp_cnt[kThreads / 32];
  int32_t rlo[kThreads];   // first observation of each candidate range of a block of ranges
  int32_t roff[kThreads];  // exclusive prefix of the ranges' lengths
  int32_t wpre[kThreads / 32];
  int32_t rtotal;
  int32_t E[NB];         // column exponents
  uint32_t tmem_base;
  int32_t nrel, bad, stop;
};

// round(s h 2^(54 - E)) for s >= 0 (|s h| <= 2^E), from the FP64 bit patterns with integer
// arithmetic: the product of the two 53-bit significands is exact in 128 bits and rounded once
// (half away from zero) at the fixed-point position; no FP64 operation. *bad is set for a
// non-finite factor or a product above the bound.
__device__ __forceinline__ long long fixed_prod(double s, double h, int E, int& bad) {
  const unsigned long long sb = (unsigned long long)__double_as_longlong(s);
  const unsigned long long hb = (unsigned long long)__double_as_longlong(h);
  const int es = (int)((sb >> 52) & 0x7FFu), eh = (int)((hb >> 52) & 0x7FFu);
  if (es == 0x7FF || eh == 0x7FF) {
    bad = 1;
    return 0;
  }
  if (es == 0 || eh == 0) return 0;  // a zero or subnormal factor (far under the column scale)
  const unsigned long long ms = (sb & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const unsigned long long mh = (hb & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  // s h 2^(54 - E) = ms mh 2^(es + eh - 2150 + 54 - E) = P 2^-r, P = ms mh < 2^106
  const int r = 2096 + E - es - eh;
  if (r >= 107) return 0;  // below half a unit of the fixed point
  if (r < 50) {            // at least 2^54: above the bound
    bad = 1;
    return 0;
  }
  unsigned long long lo = ms * mh, hi = __umul64hi(ms, mh);
  // P + 2^(r-1), then >> r
  if (r - 1 < 64) {
    const unsigned long long add = 1ull << (r - 1);
    const unsigned long long lo2 = lo + add;
    hi += (lo2 < lo) ? 1ull : 0ull;
    lo = lo2;
  } else {
    hi += 1ull << (r - 1 - 64);
  }
  const unsigned long long F = (r < 64) ? ((hi << (64 - r)) | (lo >> r)) : (hi >> (r - 64));
  if (F > (1ull << 54)) {
    bad = 1;
    return 0;
  }
  return (hb >> 63) ? -(long long)F : (long long)F;
}

// round(s h 2^(54 - E)) for s = m 2^(es - 1086) >= 0 (m its significand << 11): the upper 64 of the
// product's 106 bits are shifted to the fixed point once (the bits below weigh 2^-9 of its unit).
// The observation's half of the work is done once for all members: 28 integer instructions an
// element where fixed_prod takes 60.
__device__ __forceinline__ long long fixed_row(unsigned long long m, int es, double h, int E,
                                               int& bad) {
  const unsigned long long hb = (unsigned long long)__double_as_longlong(h);
  const int eh = (int)(hb >> 52) & 0x7FF;
  const unsigned long long mh = ((hb & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << 10;
  // s h 2^(54 - E) = P 2^-(2096 + E - es - eh), P = (m >> 11) (mh >> 10); top = P >> 43
  const int r = 2053 + E - es - eh;
  // non-finite, or above the bound (to 2^56 units: what seven digits do not hold, stage_digits finds)
  if (eh == 0x7FF || (r < 7 && m != 0ull && eh != 0)) {
    bad = 1;
    return 0;
  }
  const unsigned long long top = __umul64hi(m, mh);
  const unsigned long long F = (r < 64 && eh != 0) ? (top + (1ull << (r - 1))) >> r : 0ull;
  return (hb >> 63) ? -(long long)F : (long long)F;
}

// A zone whose largest element is 2^lx in a call whose largest is 2^em holds its Gram matrix to about
// 2^(em + lx - 54) an observation. Where that exceeds 2^(kCoarseBits - 54) of the larger of the zone's
// own products (2^(2 lx)) and the identity that is added to them, FP64 products of the zone's rows
// would be more exact, and a caller that asks for it has such zones marked (one observation with an
// error variance of 1e-12 beside others of 1e-2 would cost them 17 bits). Ordinary data are within 2
// bits: no zone of the 2,400 seeded ones of the adjoint over 64,800 zones is marked.
constexpr int kCoarseBits = 4;
constexpr int kNoExponent = -100000;  // of a call without a non-zero element

// 64-bit-integer lower-triangle index of (row j, column c <= j)
__device__ __forceinline__ int tri(int j) { return j * (j + 1) / 2; }

// barrier of the worker warps; with the scout warp
__device__ __forceinline__ void bar_workers() {
  asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
}
__device__ __forceinline__ void bar_zone() {
  asm volatile("bar.sync 2, %0;" ::"n"(kThreads + 32) : "memory");
}
// buffer b's tile staged: the workers arrive, the issuer warp waits. A hardware barrier, as it waits
// for the workers' progress: a run of zones that select nothing stages no tile, however long it is,
// and only a wait for the tensor core may expire.
__device__ __forceinline__ void tile_arrive(uint32_t b) {
  if (b)
    asm volatile("bar.arrive 4, %0;" ::"n"(kThreads + 32) : "memory");
  else
    asm volatile("bar.arrive 3, %0;" ::"n"(kThreads + 32) : "memory");
}
__device__ __forceinline__ void tile_wait(uint32_t b) {
  if (b)
    asm volatile("bar.sync 4, %0;" ::"n"(kThreads + 32) : "memory");
  else
    asm volatile("bar.sync 3, %0;" ::"n"(kThreads + 32) : "memory");
}

// kCoarse: mark the zones whose fixed point is too coarse for them (kCoarseBits)
template <bool kCoarse>
__global__ void __launch_bounds__(kThreads + 64, 1)
    k_zone_gram_oz(CellGrid g, SortedObs so, int N, LocParams lp, int32_t z0, int32_t nzc,
                   const double* __restrict__ zone_xyzt, const double* __restrict__ corr_len,
                   const double* __restrict__ max_len, const int32_t* __restrict__ col_exp,
                   const double* __restrict__ isr, double* __restrict__ G,
                   double* __restrict__ gv, int32_t* __restrict__ nobs, int brute,
                   int32_t* __restrict__ work, int32_t* __restrict__ err,
                   const int32_t* __restrict__ order, const int32_t* __restrict__ zlist,
                   OzCoarse coarse) {
  extern __shared__ __align__(16) unsigned char dyn_raw[];
  __shared__ __align__(16) OzShared ts;
  __shared__ unsigned long long s_used[kCoarse ? NB : 1];  // the zone's |F| of each member, or-ed
  const uint32_t raw_addr = smem_u32(dyn_raw);
  const uint32_t pad = ((raw_addr + 1023u) & ~1023u) - raw_addr;
  unsigned char* tiles = dyn_raw + pad;  // 2 x kBufBytes (7 slices and a zero slice), 1024-aligned
  const uint32_t tile_addr = raw_addr + pad;
  long long* acc_hi = reinterpret_cast<long long*>(tiles + 2 * kBufBytes);  // levels 0..3
  long long* acc_lo = acc_hi + kTri;                                       // levels 4..7
  double* gpart = reinterpret_cast<double*>(acc_lo + kTri);  // [kStageGroups][NB]
  // the halves' exchange overlays the K-tile buffers' digits (free at a read): [64 columns][64 rows]
  // of levels 0..3 in the first, of levels 4..7 in the second
  long long* xch = reinterpret_cast<long long*>(tiles);
  long long* xcl = reinterpret_cast<long long*>(tiles + kBufBytes);
  double* Gs = reinterpret_cast<double*>(tiles);  // and then the zone's G, [64][kLdG]

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t done0 = smem_u32(&ts.done[0]);
  if (tid == 0) {
#pragma unroll
    for (int b = 0; b < 2; b++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(done0 + 8 * b));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    ts.stop = 0;
  }
  if (tid < NB) ts.E[tid] = (tid < N) ? col_exp[tid] : 0;
  // the zero slices past the digits
  for (uint32_t i = tid; i < 2 * kSliceBytes / 16; i += kThreads + 64)
    reinterpret_cast<uint4*>(tiles + (i / (kSliceBytes / 16)) * kBufBytes + 7 * kSliceBytes)
        [i % (kSliceBytes / 16)] = make_uint4(0, 0, 0, 0);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&ts.tmem_base)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = ts.tmem_base;
  const int64_t ncells = (int64_t)g.nu * g.nv;
  const int full_scan = brute || !lp.localise;
  bool late = false;  // a bounded wait of this thread expired

  if (warp == kThreads / 32) {
    // ---- issuer: every complete K-tile to the tensor core, so that no staging warp waits for the
    // tensor core's queue (28 MMAs a tile: p = 0, 2, 4, 6, [D_p ; D_(p+1)] by D_0 .. D_(7-p))
    for (uint32_t n = 0;; n++) {
      const uint32_t b = n & 1u;
      tile_wait(b);
      if (*(volatile int32_t*)&ts.stop) break;
      if (lane == 0) {
        const uint32_t acc0 = *(volatile int32_t*)&ts.first[b] ? 0u : 1u;
        fence_after();
        const uint32_t B = tile_addr + b * kBufBytes;
#pragma unroll 1
        for (int kk = 0; kk < KT / 16; kk++) {
          const uint32_t ko = kk * 32, acc = kk > 0 ? 1u : acc0;
          const uint64_t b0 = make_desc(B + ko), b4 = make_desc(B + 4 * kSliceBytes + ko);
          mma_f16(tmem, b0, b0, idesc_f16(256), acc);        // p = 0, q = 0..3: blocks 0..3
          mma_f16(tmem + 256, b0, b4, idesc_f16(192), acc);  // q = 4..6: blocks 4..6
          uint64_t a = make_desc(B + 2 * kSliceBytes + ko);
          mma_f16(tmem + 128, a, b0, idesc_f16(256), 1u);    // p = 2, q = 0..3: blocks 2..5
          mma_f16(tmem + 384, a, b4, idesc_f16(64), 1u);     // q = 4: block 6
          mma_f16(tmem + 448, a, make_desc(B + 5 * kSliceBytes + ko), idesc_f16(64), acc);
          mma_f16(tmem + 256, b4, b0, idesc_f16(256), 1u);   // p = 4, q = 0..3: blocks 4..7
          a = make_desc(B + 6 * kSliceBytes + ko);
          mma_f16(tmem + 384, a, b0, idesc_f16(128), 1u);    // p = 6, q = 0, 1: blocks 6, 7
        }
        mma_commit(done0 + 8 * b);
      }
      __syncwarp();
    }
  } else if (warp == kThreads / 32 + 1) {
    // ---- scout: picks the next zone and forms its FP64 set-up (divisions, floors: some 10,000
    // cycles on one thread) while the workers are at the present one
    for (int par = 0;; par ^= 1) {
      int32_t w = 0;
      if (lane == 0) {
        OzZone& s = ts.zone[par];
        w = atomicAdd(work, 1);  // pick number; zone order[z0 + w] when a pick order is given
        s.w = w;
        if (w < nzc) {
          const int32_t zl = order ? order[z0 + w] : w;
          const int32_t z = zlist ? zlist[w] : z0 + zl;  // a list's zones: slots in list order
          s.zl = zl;
          s.z = z;
          const double zx = zone_xyzt[4 * (int64_t)z + 0], zy = zone_xyzt[4 * (int64_t)z + 1];
          const double zzc = zone_xyzt[4 * (int64_t)z + 2], ztc = zone_xyzt[4 * (int64_t)z + 3];
          s.zu = (lp.loctype == 1) ? zx : (lp.loctype == 2 ? zzc : ztc);
          s.zv = (lp.loctype == 1) ? zy : 0.0;
          s.L = corr_len[z];
          s.Rmax = max_len[z];
          s.zc = sel::zone_cell32(g, s.zu, s.zv, s.Rmax);
          s.iL = 1.0 / s.L;
          if (full_scan) {
            s.sr.cu0 = 0;
            s.sr.cu1 = g.nu - 1;
            s.sr.cv0 = 0;
            s.sr.cv1 = g.nv - 1;
            s.sr.all_u = 1;
          } else {
            s.sr = sel::zone_scan_range(g, lp.metric, lp.loctype, s.zu, s.zv, s.Rmax);
          }
        }
      }
      w = __shfl_sync(0xffffffffu, w, 0);
      bar_zone();  // the zone handed over; the workers are past the one before the last
      if (w >= nzc || *(volatile int32_t*)&ts.stop) break;
    }
  } else {
    // ---- workers
    const int a = tid & (NB - 1), kq = tid >> 6;  // staging: member a, 8-observation chunk kq
    const int Ea = ts.E[a];
    const bool fast = (lp.loctype != 1) || (lp.metric == OAKG_METRIC_CARTESIAN);
    uint32_t phd[2] = {0u, 0u};      // parity of the buffer's next completion
    bool pend[2] = {false, false};   // buffer handed over, its completion not yet waited for
    uint32_t nt = 0;                 // K-tiles handed over so far (buffer nt & 1)
    bool abort = false;

    auto wait_done = [&](int b) {
      if (pend[b]) {
        if (!mbar_wait(done0 + 8 * b, phd[b])) late = true;
        phd[b] ^= 1u;
        pend[b] = false;
      }
    };
    // Add the accumulators into the level sums (first: they start them; last: the zone's G goes to
    // Gs instead). Level L's even-digit part is in lanes 0-63 of column block L, its odd part in
    // lanes 64-127 of block L - 1. A part sums up to 4 products of at most 2^14 a row, so over 256
    // rows every level is an exact integer (at most 2^24).
    // Row j keeps columns c <= j; a thread of each half gives the partner half of its columns and
    // keeps the other.
    auto flush = [&](bool first, bool last, bool zbad) {
      wait_done(0);
      wait_done(1);
      fence_after();
      bar_workers();  // every warp has seen its completions: the buffers take the exchange
      const int q = warp & 3, cg = warp >> 2;
      const bool odd = q >= 2;
      const int j = 32 * (q & 1) + lane, gi = 2 * cg + (odd ? 1 : 0), gg = 2 * cg + (odd ? 0 : 1);
      const bool act = 16 * cg < 32 * ((q & 1) + 1);  // columns of the rows' lower triangle
      const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
      // four levels' 8 columns: four loads, one wait
      auto read4 = [&](uint32_t ta, uint32_t (&r)[32]) {
#pragma unroll
        for (int i = 0; i < 4; i++)
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
              : "=r"(r[8 * i]), "=r"(r[8 * i + 1]), "=r"(r[8 * i + 2]), "=r"(r[8 * i + 3]),
                "=r"(r[8 * i + 4]), "=r"(r[8 * i + 5]), "=r"(r[8 * i + 6]), "=r"(r[8 * i + 7])
              : "r"(ta + 64u * i));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int p = 0; p < 32; p += 16)
          asm volatile(""
                       : "+r"(r[p]), "+r"(r[p + 1]), "+r"(r[p + 2]), "+r"(r[p + 3]),
                         "+r"(r[p + 4]), "+r"(r[p + 5]), "+r"(r[p + 6]), "+r"(r[p + 7]),
                         "+r"(r[p + 8]), "+r"(r[p + 9]), "+r"(r[p + 10]), "+r"(r[p + 11]),
                         "+r"(r[p + 12]), "+r"(r[p + 13]), "+r"(r[p + 14]), "+r"(r[p + 15])
                       :
                       : "memory");
      };
      auto read = [&](int c0, long long (&hi)[8], long long (&lo)[8]) {
        uint32_t r[32];
        // integers: below 2^22 the bits of x + 1.5 2^23 are 0x4B400000 + x (data); a conversion else
        auto ints = [&]() {
          float mx = 0.f;
#pragma unroll
          for (int i = 0; i < 32; i++) mx = fmaxf(mx, fabsf(__uint_as_float(r[i])));
          if (__any_sync(0xffffffffu, !(mx < 4194304.f))) {
#pragma unroll
            for (int i = 0; i < 32; i++) r[i] = (uint32_t)__float2int_rn(__uint_as_float(r[i]));
          } else {
#pragma unroll
            for (int i = 0; i < 32; i++)
              r[i] = __float_as_uint(__uint_as_float(r[i]) + 12582912.f) - 0x4B400000u;
          }
        };
        auto level = [&](int i) { return (long long)(int32_t)r[i]; };
        // odd digits: levels 1..3 are in blocks 0..2 (level 0 has none), levels 4..7 in blocks 3..6
        read4(tl + c0, r);
        ints();
#pragma unroll
        for (int t = 0; t < 8; t++)
          hi[t] = odd ? level(t) * 65536 + level(8 + t) * 256 + level(16 + t)
                      : level(t) * 16777216 + level(8 + t) * 65536 + level(16 + t) * 256 + level(24 + t);
        read4(tl + (odd ? 192u : 256u) + c0, r);
        ints();
#pragma unroll
        for (int t = 0; t < 8; t++)  // in units of level 6
          lo[t] = level(t) * 65536 + level(8 + t) * 256 + level(16 + t) + ((level(24 + t) + 128) >> 8);
      };
      long long hi[8], lo[8];
      if (act) {
        read(8 * gg, hi, lo);
#pragma unroll
        for (int t = 0; t < 8; t++) {
          xch[(8 * gg + t) * NB + j] = hi[t];
          xcl[(8 * gg + t) * NB + j] = lo[t];
        }
        read(8 * gi, hi, lo);
      }
      fence_before();
      bar_workers();  // exchanged; tensor memory read
      if (act) {
        const int tj = tri(j);
#pragma unroll
        for (int t = 0; t < 8; t++) {
          const int c = 8 * gi + t;
          if (c <= j) {
            hi[t] += xch[c * NB + j];
            lo[t] += xcl[c * NB + j];
            if (!first) {
              hi[t] += acc_hi[tj + c];
              lo[t] += acc_lo[tj + c];
            }
            if (!last) {
              acc_hi[tj + c] = hi[t];
              acc_lo[tj + c] = lo[t];
            }
          }
        }
      }
      bar_workers();  // the exchange is read: the buffers take G or tiles
      if (last) {
        if (act) {
#pragma unroll
          for (int t = 0; t < 8; t++) {
            const int c = 8 * gi + t;
            if (c <= j) {
              // each sum is exact in FP64 (below 2^53 for up to 2^17 observations); the addition
              // rounds
              const int ex = ts.E[j] + ts.E[c];
              double val = scaled_i64(hi[t], ex - 36) + scaled_i64(lo[t], ex - 60);
              if (zbad) val = __longlong_as_double(0x7FF8000000000000ll);  // NaN: non-finite input
              Gs[j * kLdG + c] = val;
              Gs[c * kLdG + j] = val;
            }
          }
        }
        bar_workers();
      }
    };

    for (int par = 0; !abort; par ^= 1) {
      bar_zone();
      const OzZone& zn = ts.zone[par];
      if (zn.w >= nzc) break;
      const int32_t zl = zn.zl, z = zn.z;
      const double zu = zn.zu, zv = zn.zv, L = zn.L, Rmax = zn.Rmax;
      // the FP32 distance (relative error < 1e-6, sel::ZoneCell32) decides outside a 3e-6 band
      const float r_lo = (float)Rmax * (1.f - 3e-6f), r_hi = (float)Rmax * (1.f + 3e-6f);
      const bool fastz = fast && zn.zc.ok && !brute;  // brute force: one cell, no local offsets
      const double iL = zn.iL, iL2 = iL * iL;
      const float iL32 = (float)iL;
      if (tid == 0) {
        ts.nrel = 0;
        ts.bad = 0;
      }
      if (kCoarse && tid < NB) s_used[tid] = 0ull;  // (barriers below come before its first use)
      unsigned long long used = 0ull;
      int head = 0, tail = 0, ntile = 0, ctile = 0, nflush = 0, nrel_local = 0, bad = 0;
      double gsum = 0.0, gsum1 = 0.0;

      // stage ring entries [head, head + rows) as one K-tile and hand it to the issuer
      auto do_tile = [&](int rows) {
        if (ctile == kFlushTiles) {
          flush(nflush == 0, false, false);
          nflush++;
          ctile = 0;
        }
        const int b = (int)(nt & 1u);
        wait_done(b);
        unsigned char* tb = tiles + b * kBufBytes;
        // the chunk's 8 elements loaded first (independent loads in flight together)
        double hv[8];
        const bool in = a < N;
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int k = 8 * kq + i;
          hv[i] = (k < rows && in)
                      ? so.HSt[(int64_t)ts.ring_q[(head + k) & (kRing - 1)] * N + a] : 0.0;
        }
        long long F[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int idx = (head + 8 * kq + i) & (kRing - 1);
          const bool ok = 8 * kq + i < rows;
          F[i] = fixed_row(ok ? ts.ring_m[idx] : 0ull, ts.ring_e[idx], hv[i], Ea, bad);
          if (kCoarse) used |= (unsigned long long)(F[i] < 0 ? -F[i] : F[i]);
          // the innovation projection (two accumulators: shorter FMA chains)
          const double tq = ok ? ts.ring_t[idx] : 0.0;
          if (i & 1)
            gsum1 = fma(hv[i], tq, gsum1);
          else
            gsum = fma(hv[i], tq, gsum);
        }
        if (!stage_digits<kSliceBytes>(F, tb, tile_off(a, kq))) bad = 1;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        fence_before();
        if (tid == 0) ts.first[b] = ctile == 0;
        __syncwarp();
        tile_arrive((uint32_t)b);
        pend[b] = true;
        nt++;
        ntile++;
        ctile++;
        head += rows;
      };

      const sel::ScanRange sr = zn.sr;
      // The zone's candidates are the observations of cell rows cv0..cv1, each row one or (a
      // periodic u axis wrapping) two contiguous ranges of the cell-sorted order. Range ri is
      // (row cv0 + ri / 2, part ri % 2); blocks of kThreads ranges are flattened into one index
      // space (exclusive prefix of their lengths), so that a pass of kThreads threads takes
      // kThreads candidates across rows in the order of the rows. The order, and so the ring
      // and the selection, are those of a row-by-row scan.
      const int nranges = 2 * (sr.cv1 - sr.cv0 + 1);
      for (int rbase = 0; rbase < nranges; rbase += kThreads) {
        {
          const int ri = rbase + tid;
          int32_t rq0 = 0, rlen = 0;
          if (ri < nranges) {
            const int cv = sr.cv0 + (ri >> 1), part = ri & 1;
            int cu_a = 0, cu_b = -1;
            if (sr.all_u) {
              if (!part) cu_b = g.nu - 1;
            } else if (!g.periodic_u) {
              if (!part) {
                cu_a = sr.cu0;
                cu_b = sr.cu1;
              }
            } else {
              const int a0 = sr.cu0, b0 = sr.cu1;
              if (a0 < 0) {
                cu_a = part ? 0 : a0 + g.nu;
                cu_b = part ? b0 : g.nu - 1;
              } else if (b0 >= g.nu) {
                cu_a = part ? 0 : a0;
                cu_b = part ? b0 - g.nu : g.nu - 1;
              } else if (!part) {
                cu_a = a0;
                cu_b = b0;
              }
            }
            const int64_t c_lo = (int64_t)cu_a + (int64_t)g.nu * cv;
            const int64_t c_hi = (int64_t)cu_b + (int64_t)g.nu * cv;
            if (c_lo <= c_hi && c_lo >= 0 && c_hi < ncells) {
              rq0 = so.cell_start[c_lo];
              rlen = so.cell_start[c_hi + 1] - rq0;
            }
          }
          int incl = rlen;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
          }
          if (lane == 31) ts.warp_cnt[warp] = incl;
          bar_workers();
          if (warp == 0) {
            const int wsum = (lane < kThreads / 32) ? ts.warp_cnt[lane] : 0;
            int winc = wsum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const int t = __shfl_up_sync(0xffffffffu, winc, o);
              if (lane >= o) winc += t;
            }
            if (lane < kThreads / 32) ts.wpre[lane] = winc - wsum;
            if (lane == 31) ts.rtotal = winc;
          }
          bar_workers();
          ts.rlo[tid] = rq0;
          ts.roff[tid] = ts.wpre[warp] + incl - rlen;
          bar_workers();
        }
        const int32_t ncand = ts.rtotal;
        const int nr = min(kThreads, nranges - rbase);
        for (int32_t gb = 0; gb < ncand; gb += kThreads) {
          const int32_t gi = gb + tid;
          int32_t q = 0;
          int cv = sr.cv0;
          const bool valid = gi < ncand;
          if (valid) {
            // the last range starting at or before gi (empty ranges share the next one's start)
            int lo_i = 0, hi_i = nr - 1;
            while (lo_i < hi_i) {
              const int mid = (lo_i + hi_i + 1) >> 1;
              if (ts.roff[mid] <= gi) lo_i = mid;
              else hi_i = mid - 1;
            }
            q = ts.rlo[lo_i] + (gi - ts.roff[lo_i]);
            cv = sr.cv0 + ((rbase + lo_i) >> 1);
          }
          int sel = 0, rel = 0;
          if (valid) {
            // FP32 decisions away from the thresholds, the reference's FP64 evaluation near them
            bool done = false;
            if (fastz) {
              const float d32 = sel::cell_distance32(zn.zc, so, q, cv, lp.loctype == 1);
              const int inside = (d32 <= r_lo) ? 1 : ((d32 >= r_hi) ? 0 : -1);
              if (inside >= 0) {
                const float r32 = d32 * iL32;
                if (lp.weight == OAKG_WEIGHT_GAUSS_CUTOFF) {
                  rel = inside;
                  done = true;
                } else if (r32 >= 2.f + 1e-5f) {  // locfun = 0
                  rel = 0;
                  done = true;
                } else if (r32 <= 2.f - 1e-3f) {  // locfun > 3e-13, far above its FP64 rounding
                  rel = inside;
                  done = true;
                }
              }
            }
            if (!done) {
              double d;
              if (lp.loctype == 1)
                d = sel::distance(so.u[q], so.v[q], zu, zv, lp.metric);
              else
                d = fabs(__dsub_rn(so.u[q], zu));
              if (lp.weight == OAKG_WEIGHT_GAUSS_CUTOFF) {
                rel = (d <= Rmax);
              } else {
                rel = (d <= Rmax) && (sel::locfun(d / L) != 0.0);
              }
            }
            sel = rel || !lp.localise;
          }
          nrel_local += rel;
          const unsigned ball = __ballot_sync(0xffffffffu, sel);
          if (lane == 0) ts.warp_cnt[warp] = __popc(ball);
          bar_workers();
          int before = 0, total = 0;
#pragma unroll
          for (int w2 = 0; w2 < kThreads / 32; w2++) {
            const int cnt = ts.warp_cnt[w2];
            before += (w2 < warp) ? cnt : 0;
            total += cnt;
          }
          if (sel) {
            const int slot = (tail + before + __popc(ball & ((1u << lane) - 1u))) & (kRing - 1);
            ts.ring_q[slot] = q;
          }
          bar_workers();
          // the plain form's FP64 weights of the new entries (zone_gram.cu), one thread an
          // entry, so that the FP64 work runs with full warps: sqrt(c) = |w| / sqrt(r)
          // (c = w (w / r), DCDCovar, covariance.F90:612-619) and c (yo - Hxf). The values
          // (not the decisions, made above with the reference's rounding) are evaluated with
          // fewer FP64 operations for the Cartesian and 1-D distances: exp(-d^2 / L^2) needs
          // no square root or division, locfun(sqrt(d^2) / L) takes 1/L once a zone.
          if (tid < total) {
            const int slot = (tail + tid) & (kRing - 1);
            const int32_t qs = ts.ring_q[slot];
            double w64;
            if (fast) {
              const double du = so.u[qs] - zu;
              double D2 = du * du;
              if (lp.loctype == 1) {
                const double dv = so.v[qs] - zv;
                D2 = fma(dv, dv, D2);
              }
              w64 = (lp.weight == OAKG_WEIGHT_GAUSS_CUTOFF) ? exp(-(D2 * iL2))
                                                            : sel::locfun_value(sqrt(D2) * iL);
            } else {
              double d;
              if (lp.loctype == 1)
                d = sel::distance(so.u[qs], so.v[qs], zu, zv, lp.metric);
              else
                d = fabs(__dsub_rn(so.u[qs], zu));
              if (lp.weight == OAKG_WEIGHT_GAUSS_CUTOFF) {
                const double t = d / L;
                w64 = exp(-(t * t));
              } else {
                w64 = sel::locfun(d / L);
              }
            }
            const double sc = fabs(w64) * isr[qs];
            const unsigned long long sb = (unsigned long long)__double_as_longlong(sc);
            const int es = (int)(sb >> 52) & 0x7FF;
            ts.ring_m[slot] = es ? ((sb & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull) << 11 : 0ull;
            ts.ring_e[slot] = es;
            if (es == 0x7FF) bad = 1;  // (sc >= 0: no sign)
            ts.ring_t[slot] = sc * sc * so.innov[qs];
          }
          tail += total;
          bar_workers();  // the new entries and their weights are visible
          while (tail - head >= KT) do_tile(KT);
        }
        bar_workers();  // the block's ranges consumed before the next block overwrites them
      }
      if (tail > head) do_tile(tail - head);
      // relevant-observation count of the zone
      for (int o = 16; o > 0; o >>= 1) nrel_local += __shfl_xor_sync(0xffffffffu, nrel_local, o);
      if (lane == 0) atomicAdd(&ts.nrel, nrel_local);
      if (bad) atomicOr(&ts.bad, 1);
      if (kCoarse) atomicOr(&s_used[a], used);
      gpart[kq * NB + a] = gsum + gsum1;
      bar_workers();  // nrel, bad and the partials published
      const int nrel = ts.nrel;
      if (tid == 0) nobs[z] = nrel;
      if (kCoarse && warp == 0) {
        // 2^em bounds the call's elements, 2^lx the zone's (all rounded to zero: by half a unit)
        const int em = col_exp[NB];
        int lx = em - 54;
        for (int c = lane; c < N; c += 32)
          if (s_used[c]) lx = max(lx, ts.E[c] + 10 - __clzll((long long)s_used[c]));
        lx = __reduce_max_sync(0xffffffffu, lx);
        const bool c = nrel > 0 && (ts.bad || (em > kNoExponent &&
                                               em + lx > kCoarseBits + max(0, 2 * lx)));
        if (lane == 0) {
          coarse.zone[zl] = c;
          if (c) atomicAdd(coarse.count, 1);
        }
      }
      if (ctile > 0) flush(nflush == 0, true, ts.bad != 0);
      if (nrel > 0 && ntile > 0) {
        double* Gz = G + (int64_t)zl * N * N;
        for (int idx = tid; idx < N * NB; idx += kThreads) {
          const int j = idx >> 6, c = idx & (NB - 1);
          if (c < N) Gz[j * N + c] = Gs[j * kLdG + c];
        }
        if (tid < N) {
          double gs = 0.0;
#pragma unroll
          for (int p = 0; p < kStageGroups; p++) gs += gpart[p * NB + tid];
          gv[(int64_t)zl * N + tid] = gs;
        }
      }
      // uniform: a wait that expired in any thread ends the workers
      int any;
      asm volatile(
          "{\n.reg .pred p, q;\nsetp.ne.s32 p, %1, 0;\nbar.red.or.pred q, 1, %2, p;\n"
          "selp.s32 %0, 1, 0, q;\n}\n"
          : "=r"(any)
          : "r"((int)late), "n"(kThreads)
          : "memory");
      abort = any != 0;
    }
    // release the issuer, and after an expired wait the scout
    if (tid == 0) ts.stop = 1;
    __syncwarp();
    bar_workers();
    tile_arrive(nt & 1u);
    if (abort) bar_zone();
    wait_done(0);
    wait_done(1);
  }
  // teardown: no MMA may still write tensor memory when it is freed
  if (late) atomicOr(err, ZST_TIMEOUT);
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols));
}

// isr_q = r_q^-1/2 and the column exponents: E_a with max_q |HS_qa| isr_q (1 + 2^-20) <= 2^E_a
// (|w| <= 1, so every |X_qa| of every zone is below it). The maxima of non-negative FP64
// values are taken on their bit patterns (ordered like the values). Non-finite values and
// r <= 0 are left out: the zones that select such an observation get a non-finite weight or
// element, which marks their G as NaN (as the CUDA-core products would propagate it); the
// other zones keep the scale of the finite data.
__global__ void k_oz_colmax(int64_t m, int N, const double* __restrict__ HSt,
                            const double* __restrict__ r, unsigned long long* __restrict__ mx,
                            double* __restrict__ isr) {
  __shared__ unsigned long long smax[NB];
  if (threadIdx.x < NB) smax[threadIdx.x] = 0ull;
  __syncthreads();
  const int a = threadIdx.x & (NB - 1);
  unsigned long long loc = 0ull;
  if (a < N) {
    for (int64_t q = blockIdx.x * (int64_t)(blockDim.x / NB) + threadIdx.x / NB; q < m;
         q += (int64_t)gridDim.x * (blockDim.x / NB)) {
      const double rq = r[q];
      const double iq = rsqrt(rq);
      if (a == 0) isr[q] = iq;
      if (!(rq > 0.0) || !(rq < INFINITY)) continue;
      const double v = fabs(HSt[q * N + a]) * iq;
      const unsigned long long vb = (unsigned long long)__double_as_longlong(v);
      if (vb < 0x7FF0000000000000ull) loc = vb > loc ? vb : loc;
    }
    atomicMax(&smax[a], loc);
  }
  __syncthreads();
  if (threadIdx.x < N) atomicMax(&mx[threadIdx.x], smax[threadIdx.x]);
}

__global__ void k_oz_exponents(int N, const unsigned long long* __restrict__ mx,
                               int32_t* __restrict__ E) {
  const int a = threadIdx.x;  // NB threads
  __shared__ int top[NB / 32];
  const double vmax = a < N ? __longlong_as_double((long long)mx[a]) : 0.0;
  int e;
  if (vmax == 0.0) {
    e = 0;  // an all-zero column (or no usable observation)
  } else {
    const double v = vmax * (1.0 + 0x1p-20);
    if (!(v < INFINITY)) {
      e = -4000;  // beyond the FP64 range: every nonzero element is out of range (G is NaN)
    } else {
      // v in [2^(k-1), 2^k) with k = biased exponent - 1022 (normal v)
      const int be = (int)(((unsigned long long)__double_as_longlong(v) >> 52) & 0x7FF);
      e = (be == 0) ? -1022 : be - 1022;
    }
  }
  if (a < N) E[a] = e;
  // the largest of all, at E[NB]
  const int t = __reduce_max_sync(0xffffffffu, vmax == 0.0 ? kNoExponent : e);
  if ((a & 31) == 0) top[a >> 5] = t;
  __syncthreads();
  if (a == 0) E[NB] = max(top[0], top[1]);
}

// ------------------------------------------------------------------ square-root transform
// The plain form's T_sym = U diag((1 + lambda)^-1/2) U^T (rrsqrt.F90:162-169) as the Gram X^T X
// of X_ka = q_k U_ak, q_k = (1 + lambda_k)^-1/4: row k of X is eigenvector k scaled, so a zone
// is one K-tile of 64 rows and the slice products of k_zone_gram_oz apply unchanged. With one
// K-tile every level (at most 7 x 64 x 2^14 < 2^23 in magnitude) is exact in its FP32
// accumulator, and one read of the tensor memory gives T_sym = 2^(E_a + E_b - 36) (v + V456 /
// 256), recombined here as the integer v 2^16 + round(256 V456) (below 2^62) with one
// conversion to FP64. Column exponents come from the exponent fields: a normal x lies below
// 2^(e(x) - 1022) (e the biased exponent), so E_a = max_k (e(q_k) + e(U_ak)) - 2044 bounds
// |X_ka| (at most two bits above the column's maximum) and every product fits the fixed point.
//
// T = T_sym Omega (rrsqrt.F90:171-185) follows in FP64. Omega = P_v P_w + (1 - s_v s_w) v w^T
// with P_x = I - u_x u_x^T / c_x, u_x = x + s_x e_N, c_x = 1 + |x_N| (matoper.F90:509-535;
// w = N^-1/2 1, s_w = 1), so T = T_sym - a u_v^T - g u_w^T + b w^T is a rank-three update
// with a = T_sym u_v / c_v, g = (T_sym u_w - (u_v . u_w) a) / c_w and b = (1 - s_v) T_sym v.
// T_sym v and the row sums (T_sym u_w = w rowsum + T_sym e_N) are accumulated while T_sym is
// formed; the update is then one FMA and one add an element.
// Pipeline per CTA (one of 512 threads per SM, zones strided): while zone i's MMAs run, zone
// i + 1's U and scalings are copied into shared memory (cp.async); after zone i's accumulator
// read, zone i + 1 is split and its MMAs issued, and zone i's rotation and T write run beside
// them. The levels are recombined into FP64 by integer operations (the FP64 pipe carries only
// the rotation's sums and update). The shared-memory request keeps a second CTA (which would
// wait for the tensor memory) off the SM.
constexpr int kTsLd = NB + 1;
constexpr size_t kTsData = 1024 + (size_t)kBufBytes +
                           (size_t)NB * kTsLd * sizeof(double) + (size_t)NB * NB * sizeof(double) +
                           18 * NB * sizeof(double);
constexpr size_t kTsDynSmem = (size_t)148 * 1024;
static_assert(kTsData <= kTsDynSmem, "square-root transform shared memory");

struct TsShared {
  unsigned long long mbar;
  uint32_t tmem_base;
  int32_t emax[NB];  // max_k e(q_k) + e(U_ak) of the zone being split
  int32_t E[NB];     // column exponents of the zone in the accumulators
  int32_t flag;
  int32_t bad[2];    // non-finite input, by zone parity
  double uvuw;       // u_v . u_w of the current zone
};

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// the seven levels' 8 columns at c0 of this warp's 32 lanes: seven loads, one wait; the empty
// asm statements tie the registers' uses to the wait
__device__ __forceinline__ void tmem_ld7x8(uint32_t ta, int c0, uint32_t (&r)[56]) {
  const uint32_t cols[7] = {0u, 64u, 128u, 192u, 256u, 320u, 384u};
#pragma unroll
  for (int L = 0; L < 7; L++)
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r[8 * L]), "=r"(r[8 * L + 1]), "=r"(r[8 * L + 2]), "=r"(r[8 * L + 3]),
          "=r"(r[8 * L + 4]), "=r"(r[8 * L + 5]), "=r"(r[8 * L + 6]), "=r"(r[8 * L + 7])
        : "r"(ta + cols[L] + (uint32_t)c0));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < 56; q += 14)
    asm volatile(""
                 : "+r"(r[q]), "+r"(r[q + 1]), "+r"(r[q + 2]), "+r"(r[q + 3]), "+r"(r[q + 4]),
                   "+r"(r[q + 5]), "+r"(r[q + 6]), "+r"(r[q + 7]), "+r"(r[q + 8]),
                   "+r"(r[q + 9]), "+r"(r[q + 10]), "+r"(r[q + 11]), "+r"(r[q + 12]),
                   "+r"(r[q + 13])
                 :
                 : "memory");
}

__global__ void __launch_bounds__(kThreads, 1)
    k_zone_tsym_oz(int N, int32_t nzc, double* __restrict__ GT, const double* __restrict__ aux,
                   const double* __restrict__ Zg, const int32_t* __restrict__ nobs, int rotate,
                   int32_t* status, const int32_t* __restrict__ retries) {
  if (retries && *retries == 0) return;
  extern __shared__ __align__(16) unsigned char dyn_raw[];
  __shared__ __align__(16) TsShared ts;
  const uint32_t raw_addr = smem_u32(dyn_raw);
  const uint32_t pad = ((raw_addr + 1023u) & ~1023u) - raw_addr;
  unsigned char* tile = dyn_raw + pad;  // the 7 slices and the zero slice past them
  const uint32_t tile_addr = raw_addr + pad;
  double* Ts = reinterpret_cast<double*>(tile + kBufBytes);  // [NB][kTsLd]
  double* Upre = Ts + NB * kTsLd;  // next zone's U slot, as stored (U_ak at k N + a)
  double* qpre = Upre + NB * NB;   // next zone's (1 + lambda)^-1/4
  double* vpre = qpre + NB;        // next zone's v
  double* vvb = vpre + NB;         // [2][NB] v by zone parity
  double* uv = vvb + 2 * NB;       // u_v of the current zone
  double* pv = uv + NB;            // [4][NB] partial T_sym v (column groups)
  double* ps = pv + 4 * NB;        // [4][NB] partial row sums
  double* ar = ps + 4 * NB;        // a
  double* cr = ar + NB;            // (b - g) w
  double* gr = cr + NB;            // g
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int a = tid & (NB - 1), kq = tid >> 6;  // member a; rows 8 kq .. 8 kq + 7 of X
  const uint32_t mbar = smem_u32(&ts.mbar);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    ts.flag = 0;
  }
  if (tid < NB) ts.emax[tid] = 0;
  // rows 64-127 of the last digit's A operand: read by the MMA, never read back
  for (uint32_t i = tid; i < kSliceBytes / 16; i += kThreads)
    reinterpret_cast<uint4*>(tile + 7 * kSliceBytes)[i] = make_uint4(0, 0, 0, 0);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&ts.tmem_base)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = ts.tmem_base;
  const double wv = 1.0 / sqrt((double)N);
  const double cw = 1.0 + wv, icw = 1.0 / cw;
  // this CTA's next zone from z on
  auto next_zone = [&](int32_t z) {
    while (z < nzc && (nobs[z] == 0 || (retries && !(status[z] & ZST_RETRY)))) z += gridDim.x;
    return z;
  };
  uint32_t ph = 0;
  bool pending = false;  // an MMA group whose completion was not observed (timeout)

  // zone zn into Upre / qpre / vpre (asynchronous copies)
  auto prefetch = [&](int32_t zn) {
    const double* src = Zg + (int64_t)zn * N * N;
    for (int idx = tid; idx < N * N; idx += kThreads) cp_async8(Upre + idx, src + idx);
    const double* axn = aux + (int64_t)zn * (5 * N + 2);
    if (tid < N) {
      cp_async8(qpre + tid, axn + 4 * N + tid);
      cp_async8(vpre + tid, axn + tid);
    }
  };
  // split the prefetched zone (parity par) into the slices and issue its MMAs; its copies
  // have landed and are visible (a barrier since this thread's cp_async_wait_all)
  auto stage_issue = [&](int par) {
    double hv[8], sv[8];
    int em = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int k = 8 * kq + i;
      hv[i] = (a < N && k < N) ? Upre[k * N + a] : 0.0;
      sv[i] = (k < N) ? qpre[k] : 0.0;
      const int es = (int)(((unsigned long long)__double_as_longlong(sv[i]) >> 52) & 0x7FFu);
      const int eh = (int)(((unsigned long long)__double_as_longlong(hv[i]) >> 52) & 0x7FFu);
      if (es != 0 && eh != 0 && es != 0x7FF && eh != 0x7FF) em = max(em, es + eh);
    }
    if (em > 0) atomicMax(&ts.emax[a], em);
    if (tid == 0) ts.bad[par] = 0;
    if (tid < NB) vvb[par * NB + tid] = (rotate && tid < N) ? vpre[tid] : 0.0;
    __syncthreads();  // maxima complete; the previous zone's exponents no longer read
    const int ema = ts.emax[a];
    const int Ea = (ema > 0) ? ema - 2044 : 0;
    if (tid < NB) ts.E[tid] = Ea;  // a == tid
    int bad = 0;
    uint32_t pk[kDigits][4];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      unsigned long long Ub[2];
#pragma unroll
      for (int u = 0; u < 2; u++)
        Ub[u] = (unsigned long long)fixed_prod(sv[i + u], hv[i + u], Ea, bad) + kDigitBias;
      uint32_t d[kDigits];
      digit_pairs(Ub[0], Ub[1], d);
#pragma unroll
      for (int p = 0; p < kDigits; p++) pk[p][i >> 1] = d[p];
    }
#pragma unroll
    for (int p = 0; p < kDigits; p++)
      *reinterpret_cast<uint4*>(tile + p * kSliceBytes + tile_off(a, kq)) =
          make_uint4(pk[p][0], pk[p][1], pk[p][2], pk[p][3]);
    if (bad) atomicOr(&ts.bad[par], 1);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();  // slices staged; Upre, qpre, vpre and the maxima read
    if (tid < NB) ts.emax[tid] = 0;
    if (tid == 0) {
      fence_after();
#pragma unroll 1
      for (int kk = 0; kk < KT / 16; kk++) {
        const uint32_t ko = kk * 32;
        const uint32_t acc0 = kk > 0 ? 1u : 0u;
        // levels 0..3 in columns 64 L: A = [D_p ; D_p+1], B = D_0 .. D_(3-p)
#pragma unroll
        for (int p = 0; p < 4; p++)
          mma_f16(tmem + 64 * p, make_desc(tile_addr + p * kSliceBytes + ko),
                   make_desc(tile_addr + ko), idesc_f16(64u * (4 - p)), p == 0 ? acc0 : 1u);
        // levels 4..6 in columns 256 + 64 (L - 4): B = D_qlo .. D_qhi, q = L - p
#pragma unroll
        for (int p = 0; p < kDigits; p++) {
          const int qlo = (4 - p > 0) ? 4 - p : 0;
          const int qhi = (6 - p < kDigits - 1) ? 6 - p : kDigits - 1;
          const int off = qlo - (4 - p);
          mma_f16(tmem + 256 + 64 * off, make_desc(tile_addr + p * kSliceBytes + ko),
                   make_desc(tile_addr + qlo * kSliceBytes + ko),
                   idesc_f16(64u * (qhi - qlo + 1)), p == 0 ? acc0 : 1u);
        }
      }
      mma_commit(mbar);
    }
  };

  int32_t zl = next_zone((int32_t)blockIdx.x), zn = nzc;  // in the accumulators; prefetched
  if (zl < nzc) {
    prefetch(zl);
    cp_async_wait_all();
    __syncthreads();
    stage_issue(0);
    zn = next_zone(zl + gridDim.x);
    if (zn < nzc) prefetch(zn);
  }
  for (int par = 0; zl < nzc; par ^= 1) {
    if (tid == 0 && !mbar_wait(mbar, ph)) ts.flag = 1;
    ph ^= 1u;
    __syncthreads();  // MMA completion (or the timeout) published
    if (ts.flag) {
      pending = true;
      if (tid == 0) atomicOr(&status[zl], ZST_TIMEOUT);
      break;
    }
    fence_after();
    const double* vv = vvb + par * NB;
    // T_sym from the accumulators: lanes 0-63 (rows j) are read by warps 0, 1, 4, 5, 8, 9,
    // 12, 13; warp group cg takes columns 16 cg .. 16 cg + 15 of all seven levels, and its
    // partial sums of T_sym v and of the row. Warp 2 forms u_v and u_v . u_w meanwhile.
    if ((warp & 3) < 2) {
      const int qd = warp & 3, cg = warp >> 2;
      const int j = 32 * qd + lane;
      const uint32_t ta = tmem + ((uint32_t)(32 * qd) << 16);
      const bool zbad = ts.bad[par] != 0;
      const int Ej = ts.E[j];
      double sv_part = 0.0, sr_part = 0.0;
#pragma unroll 1
      for (int h8 = 0; h8 < 2; h8++) {
        const int c0 = 16 * cg + 8 * h8;
        uint32_t r[56];
        tmem_ld7x8(ta, c0, r);
#pragma unroll
        for (int t = 0; t < 8; t++) {
          const int c = c0 + t;
          const long long v =
              (((long long)__float2int_rn(__uint_as_float(r[t])) * 256 +
                __float2int_rn(__uint_as_float(r[8 + t]))) * 256 +
               __float2int_rn(__uint_as_float(r[16 + t]))) * 256 +
              __float2int_rn(__uint_as_float(r[24 + t]));
          // 256 V456 is below 2^31 in magnitude (level 4 below 5 x 64 x 2^14)
          const float f456 = fmaf(__uint_as_float(r[48 + t]), 1.f / 65536.f,
                                  fmaf(__uint_as_float(r[40 + t]), 1.f / 256.f,
                                       __uint_as_float(r[32 + t])));
          const long long vt = v * 65536 + (long long)__float2int_rn(f456 * 256.f);
          double val = scaled_i64(vt, Ej + ts.E[c] - 52);
          if (zbad) val = __longlong_as_double(0x7FF8000000000000ll);  // NaN: non-finite input
          Ts[j * kTsLd + c] = val;
          if (rotate) {
            sv_part = fma(val, vv[c], sv_part);
            sr_part += (c < N) ? val : 0.0;
          }
        }
      }
      if (rotate) {
        pv[cg * NB + j] = sv_part;
        ps[cg * NB + j] = sr_part;
      }
    } else if (warp == 2 && rotate) {  // u_v and u_v . u_w, u_w = w 1 + e_N
      const double sgv = signbit(vv[N - 1]) ? -1.0 : 1.0;
      double sdot = 0.0;
      for (int jj = lane; jj < NB; jj += 32) {
        const double u = (jj < N) ? vv[jj] + ((jj == N - 1) ? sgv : 0.0) : 0.0;
        uv[jj] = u;
        sdot = fma(u, wv + ((jj == N - 1) ? 1.0 : 0.0), sdot);
      }
      for (int o = 16; o > 0; o >>= 1) sdot += __shfl_xor_sync(0xffffffffu, sdot, o);
      if (lane == 0) ts.uvuw = sdot;
    }
    const int32_t znn = zn < nzc ? next_zone(zn + gridDim.x) : nzc;
    if (zn < nzc) cp_async_wait_all();  // the next zone's copies (this thread's)
    fence_before();
    __syncthreads();  // T_sym, sums, u_v published; tensor memory read; next zone landed
    if (zn < nzc) {
      stage_issue(par ^ 1);  // the next zone's MMAs run beside this zone's rotation
      if (znn < nzc) prefetch(znn);
    }
    double* Gz = GT + (int64_t)zl * N * N;
    if (rotate) {
      const double sgv = signbit(vv[N - 1]) ? -1.0 : 1.0;
      if (tid < N) {
        const int r = tid;
        const double tvi = (pv[r] + pv[NB + r]) + (pv[2 * NB + r] + pv[3 * NB + r]);  // T_sym v
        const double rsi = (ps[r] + ps[NB + r]) + (ps[2 * NB + r] + ps[3 * NB + r]);
        const double tlast = Ts[r * kTsLd + N - 1];
        const double ai = fma(sgv, tlast, tvi) / (1.0 + fabs(vv[N - 1]));  // T_sym u_v / c_v
        const double gi = fma(-ts.uvuw, ai, fma(wv, rsi, tlast)) * icw;
        ar[r] = ai;
        gr[r] = gi;
        cr[r] = ((1.0 - sgv) * tvi - gi) * wv;
      }
      __syncthreads();
      for (int idx = tid; idx < N * N; idx += kThreads) {
        const int r = idx / N, c = idx - r * N;
        double t = fma(-ar[r], uv[c], Ts[r * kTsLd + c]) + cr[r];
        if (c == N - 1) t -= gr[r];
        Gz[idx] = t;
      }
    } else {
      for (int idx = tid; idx < N * N; idx += kThreads) {
        const int r = idx / N, c = idx - r * N;
        Gz[idx] = Ts[r * kTsLd + c];
      }
    }
    if (retries && tid == 0) status[zl] &= ~ZST_RETRY;
    zl = zn;
    zn = znn;
  }
  // teardown: no MMA may still write tensor memory when it is freed, no copy still land
  cp_async_wait_all();
  if (pending && tid == 0) mbar_wait(mbar, ph ^ 1u);
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols));
}

}  // namespace

int gram_oz_max_n() { return NB; }

size_t gram_oz_scratch_bytes(int64_t m) {
  return NB * sizeof(unsigned long long) + (NB + 2) * sizeof(int32_t) + (size_t)m * sizeof(double);
}

cudaError_t zone_gram_oz(const CellGrid& g, const SortedObs& so, int64_t m, int N, LocParams lp,
                         int32_t z0, int32_t nzc, const double* zone_xyzt, const double* corr_len,
                         const double* max_len, double* d_G, double* d_g, int32_t* d_nobs,
                         int brute, int32_t* d_work, int32_t* d_err, void* d_scratch,
                         cudaStream_t st, const int32_t* order, const int32_t* zlist,
                         OzCoarse coarse) {
  if (N < 1 || N > NB || !so.HSt || !so.r || !d_scratch) return cudaErrorInvalidValue;
  unsigned long long* mx = reinterpret_cast<unsigned long long*>(d_scratch);
  int32_t* E = reinterpret_cast<int32_t*>(mx + NB);
  double* isr = reinterpret_cast<double*>(E + NB + 2);  // 8-byte aligned: E's 66 int32 are 264 bytes
  cudaError_t e = cudaMemsetAsync(mx, 0, NB * sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (m > 0) {
    const int64_t per = kThreads / NB;
    int64_t blocks = (m + per - 1) / per;
    if (blocks > 4 * (int64_t)sms) blocks = 4 * (int64_t)sms;
    k_oz_colmax<<<(unsigned)(blocks > 0 ? blocks : 1), kThreads, 0, st>>>(m, N, so.HSt, so.r, mx, isr);
    count_launches(1);
  }
  k_oz_exponents<<<1, NB, 0, st>>>(N, mx, E);
  count_launches(1);
  const auto kernel = coarse.zone ? k_zone_gram_oz<true> : k_zone_gram_oz<false>;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDynSmem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  // the shared-memory size admits one CTA per SM (it holds all 512 tensor-memory columns)
  int grid = sms;
  if (grid > nzc) grid = nzc > 0 ? nzc : 1;
  e = cudaMemsetAsync(d_work, 0, sizeof(int32_t), st);
  if (e != cudaSuccess) return e;
  kernel<<<grid, kThreads + 64, kDynSmem, st>>>(g, so, N, lp, z0, nzc, zone_xyzt, corr_len, max_len, E,
                                                isr, d_G, d_g, d_nobs, brute, d_work, d_err, order,
                                                zlist, coarse);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t zone_tsym_oz(int N, int32_t nzc, double* d_GT, const double* d_aux,
                         const double* d_Z, const int32_t* d_nobs, int rotate,
                         int32_t* d_status, cudaStream_t st, const int32_t* d_retries) {
  if (N < 1 || N > NB) return cudaErrorInvalidValue;
  if (nzc <= 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k_zone_tsym_oz, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kTsDynSmem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_zone_tsym_oz, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = sms < nzc ? sms : nzc;
  k_zone_tsym_oz<<<grid, kThreads, kTsDynSmem, st>>>(N, nzc, d_GT, d_aux, d_Z, d_nobs, rotate,
                                                     d_status, d_retries);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace oakg
