// The plain (FP64) form's square-root transform from FP32 eigenpairs, ensembles of 17..64
// members: T_sym = A^(-1/2), A = I + G, by a Newton iteration whose residual is formed by exact
// slice products on the FP16 tensor cores. The outputs are functions of A alone
// (rrsqrt.F90:136-185; lambda >= 0 because G is a Gram matrix): T = A^(-1/2) Omega,
// ampl = A^-1 g, v = A^(1/2) w / |A^(1/2) w|, so no FP64 eigenvectors are needed.
//
// Start. V, lambda are the FP32 eigenpairs of G (zone_eig32.cu), s_k = (1 + lambda_k)^(1/2), and
//   Y_0 = V diag(1 / s) V^T. R = I - Y_0 A Y_0 has entries of 2e-5 at lambda_max ~ 10^3.
// Step. The correction E of Y + E solves E (A Y) + (Y A) E = R to first order; A Y is A^(1/2) to
//   first order, in V's basis diag(s) + X, and X is known from the first residual: R' = V^T R V
//   gives X_kl = -s_k R'_kl s_l / (s_k + s_l) and s_k (1 - R'_kk / 2) for s_k. So
//   E' = R' / (s_k + s_l), from the second step on less (E' X + X E') / (s_k + s_l), E = V E' V^T.
//   The residual falls from 2e-5 to 1e-9 (the basis is off by 4 rho_0) to 1e-15 (by 7 rho_0^2 and
//   by the 22 bits of the FP16 x 2 products with V): two steps, a third for 2 % of the zones of
//   the 64,800-zone case. Clusters of eigenvalues do not matter (s_k + s_l >= 2) and V need
//   not be exact. A zone whose R does not fall (eigenvalues from about 10^6, non-finite entries)
//   goes to the FP64 eigensolve (ZST_RETRY), with G intact.
// Acceptance. The residual after the last correction is not formed but predicted: the last one
//   formed times the factor by which a step reduces it, as expected and, with a margin, as the
//   worst zones show it (kAccept). In a sweep of 43,200 zones (20, 40 and 64 members, lambda_max
//   1 to 10^8, six shapes of spectrum, among them clusters and one dominant eigenvalue) the
//   residual formed once more after acceptance was at most 0.46 max(2e-14, u (1 + lambda_max)),
//   u = 2^-53: below what rounding A's entries to FP64 does. With the expected factor alone it
//   was up to 1.7 times that; 0.8 % of the zones take a step more for it.
// Arithmetic. Y is a 64-bit fixed-point number (2^-60), kept a multiple of 2^-54 while it enters
//   products; A has a power-of-two scale a row (54 bits below the row's maximum: finer than the
//   FP64 entries themselves). Z = A Y and Y Z are exact slice products as in zone_gram_oz.cu,
//   seven balanced base-256 digits an operand, all levels 0..7 (level 8 and beyond weigh 2^-61
//   of the row and column scales for data): level L sums D_p B_q over p + q = L. The operand
//   [D_p ; D_(p+1)], p = 0, 2, 4, 6 (M = 128, a zero slice as D_7) times D_0 .. D_(7-p) puts level
//   L's even-p part into lanes 0-63 of column block L and its odd-p part into lanes 64-127 of
//   block L - 1: the eight blocks of 64 columns are the whole tensor memory and no row is
//   computed twice. Every level sum is an integer below 2^22 and exact in FP32; the two halves
//   meet as 64-bit integers through shared memory. Z is bounded by the square root of A's
//   diagonal, which fixes its column scale before it is known. The small vectors (A^-1 g, A^(1/2)
//   1, the rotation's terms) are 64-bit fixed point as well: the FP64 pipe runs two FMAs a
//   cycle and SM.
//
// One CTA of 512 threads per SM (222 KB of shared memory and all tensor memory), zones strided;
// the next zone's G and V are copied in while a zone finishes. Every mbarrier wait is bounded
// (ZST_TIMEOUT).
//
// Measured, 64,800 zones of 64 members: 20 ms (18 and 85,000 cycles a zone without the amplitudes'
// refinement; a level product ~2,700 of tensor time, its staging ~2,000 and its read ~2,900, a
// step's four products with V ~9,000: bound by the latency of that chain with one zone in flight),
// and 13 ms for the FP32 stages.
// The FP64 eigensolve and its tensor-core transform took 146 ms (FP64 pipe at 85-90 %). Errors
// against long double on a zone: 1e-15, where an FP64 eigensolve has 1e-14 to 1e-13.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>

#include "oakg_internal.cuh"
#include "oz_slices.cuh"

namespace oakg {

namespace {

constexpr int kThreads = 512;
constexpr int NB = 64;  // padded ensemble width
constexpr uint32_t kSlice = 64u * 128u;
constexpr uint32_t kTmemCols = 512;
// dynamic shared memory (1024-aligned): A (7 digit slices and a zero slice), Y (likewise), V
// member-major (hi, lo) and vector-major (hi, lo), the work area (7 slices of Z; the exchange,
// correction operands and partial sums otherwise). An M = 128 operand of 64 rows reads the slice
// after it into accumulator lanes 64-127, which are then not read back; the work area is last
// and no such operand starts in its last slice.
constexpr uint32_t kOffA = 0, kOffY = 8 * kSlice, kOffVa = 16 * kSlice, kOffVk = 18 * kSlice,
                   kOffW = 20 * kSlice;
constexpr uint32_t kOffX1 = kOffW, kOffX2 = kOffW + 2 * kSlice;  // correction operands (hi, lo)
constexpr uint32_t kOffE = kOffW + 4 * kSlice;                   // FP32 [64][65]
constexpr uint32_t kOffPd = kOffE + 64 * 65 * 4;                 // FP64 [8][64] partial sums
constexpr uint32_t kOffPf = kOffPd + 8 * 64 * 8;                 // FP32 [8][64]
static_assert(kOffPf + 8 * 64 * 4 <= 27 * kSlice, "work area");
constexpr size_t kIsqSmem = 1024 + 27 * (size_t)kSlice;
constexpr int kMaxSteps = 6;
// Predicted residual that a zone may keep: kAccept by the expected factor of a step; by its worst
// case kAccept or u (1 + lambda_max)
constexpr float kAccept = 2e-14f;
constexpr int kLdE = 65;

constexpr float kVScale = 128.f;  // V's FP16 slices hold 128 V (their low parts stay normal)

struct IsqShared {
  long long zpart[8][NB];  // partial row sums of Z = A Y, units 2^(E_row - 60)
  long long gi[NB];        // g in units 2^(eg - 62)
  long long t1[NB];        // Y g, then u_v in units 2^-61
  long long ar[NB], cr[NB], gr[NB];  // T_sym u_v / c_v (2^-61), and the row terms (2^-60)
  double vj[NB], tl[NB];
  double red[2][2];
  unsigned long long mbar;
  float s[NB];   // (1 + lambda)^(1/2)
  float es[NB];  // row sums of the last correction
  float rf[NB], tf[NB];  // the amplitudes' residual in units 2^Eg, Y times it
  float rmax[kThreads / 32];
  float lmax[2];  // 1 + lambda_max, a half each
  int32_t emax[NB];  // largest exponent of A's rows
  int32_t fj[NB];    // column exponents of Z
  uint32_t tmax[2];  // high word of max |Y g|
  int32_t emaxg[2];  // largest exponent of g
  uint32_t tmem_base;
  int32_t bad, nan;
};

// cp.async of B bytes (4, 8 or 16, aligned)
template <int B>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(B)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// 16 consecutive accumulator columns of this warp's 32 tensor-memory lanes
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// two floats as packed FP16 (first in the low half)
__device__ __forceinline__ uint32_t pack_f16(float a, float b) {
  const __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// 8 consecutive K elements of an operand row as FP16 slices hi, lo (22 bits together)
__device__ __forceinline__ void stage_f16(const float (&x)[8], unsigned char* slices, uint32_t off) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    h[i] = pack_f16(x[2 * i], x[2 * i + 1]);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h[i]));
    l[i] = pack_f16(x[2 * i] - f.x, x[2 * i + 1] - f.y);
  }
  *reinterpret_cast<uint4*>(slices + off) = make_uint4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<uint4*>(slices + kSlice + off) = make_uint4(l[0], l[1], l[2], l[3]);
}

// (by integer operations, as fixed_of in oz_slices.cuh) x 2^sh towards zero, |x 2^sh| < 2^62
__device__ __forceinline__ long long fixed_of(float x, int sh) {
  const uint32_t b = __float_as_uint(x);
  const int e = (int)((b >> 23) & 255u);
  const unsigned long long m = e ? (b & 0x7FFFFFu) | 0x800000u : 0u;
  const int s = e - 150 + sh;
  const unsigned long long F = s >= 0 ? m << (s < 39 ? s : 39) : (s > -24 ? m >> (-s) : 0ull);
  return (b >> 31) ? -(long long)F : (long long)F;
}

// v to 24 bits, towards zero
__device__ __forceinline__ float float_of(long long v) {
  const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  if (a == 0) return 0.f;
  const int lz = __clzll((long long)a);
  const uint32_t m = (uint32_t)((a << lz) >> 40) & 0x7FFFFFu;
  return __uint_as_float((v < 0 ? 0x80000000u : 0u) | ((uint32_t)(190 - lz) << 23) | m);
}

// x to 24 bits, towards zero; |x| in FP32's normal range or taken as 0
__device__ __forceinline__ float float_of(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const uint32_t hi = (uint32_t)(b >> 32), lo = (uint32_t)b, ae = (hi & 0x7FFFFFFFu) >> 20;
  if (ae <= 896u) return 0.f;
  return __uint_as_float((hi & 0x80000000u) |
                         ((((hi & 0x7FFFFFFFu) - (896u << 20)) << 3) | (lo >> 29)));
}

__global__ void __launch_bounds__(kThreads, 1)
    k_zone_isqrt_oz(int N, int32_t nzc, double* __restrict__ GT, const float* __restrict__ Zv,
                    const float* __restrict__ aux32, int aux_stride, const double* __restrict__ gv,
                    const int32_t* __restrict__ nobs, int rotate, double* __restrict__ ampl,
                    int32_t* __restrict__ status, int32_t* __restrict__ retries) {
  extern __shared__ __align__(16) unsigned char dyn_raw[];
  __shared__ __align__(16) IsqShared ts;
  const uint32_t raw_addr = smem_u32(dyn_raw);
  const uint32_t pad = ((raw_addr + 1023u) & ~1023u) - raw_addr;
  unsigned char* sm = dyn_raw + pad;
  const uint32_t sa = raw_addr + pad;
  long long* xch = reinterpret_cast<long long*>(sm + kOffW);  // [64 columns][64 rows]
  float* Eb = reinterpret_cast<float*>(sm + kOffE);           // [64][kLdE]
  long long* pd = reinterpret_cast<long long*>(sm + kOffPd);  // [8][64]
  long long* py = reinterpret_cast<long long*>(sm + kOffX1);  // [8][64]
  float* pf = reinterpret_cast<float*>(sm + kOffPf);          // [8][64]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // tensor-memory lane quarter q: rows 32 (q & 1) .. + 31, odd digits for q >= 2. The thread
  // owns row j, columns 8 gi .. 8 gi + 7 of every matrix
  const int q = warp & 3, cg = warp >> 2;
  const bool odd = q >= 2;
  const int j = 32 * (q & 1) + lane, gi = 2 * cg + (odd ? 1 : 0), c0 = 8 * gi;
  const int gi_give = 2 * cg + (odd ? 0 : 1);  // the group of the other half's thread
  const uint32_t own_off = tile_off(j, gi);
  const uint32_t mbar = smem_u32(&ts.mbar);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the zero slices past the digits of A and Y; the work area holds finite values before any
  // of it is an operand row that is not read back
  for (uint32_t i = tid; i < kSlice / 16; i += kThreads) {
    reinterpret_cast<uint4*>(sm + kOffA + 7 * kSlice)[i] = make_uint4(0, 0, 0, 0);
    reinterpret_cast<uint4*>(sm + kOffY + 7 * kSlice)[i] = make_uint4(0, 0, 0, 0);
  }
  for (uint32_t i = tid; i < 7 * kSlice / 16; i += kThreads)
    reinterpret_cast<uint4*>(sm + kOffW)[i] = make_uint4(0, 0, 0, 0);
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
  const uint32_t tlane = tmem + ((uint32_t)(32 * q) << 16);
  const double wv = 1.0 / sqrt((double)N);
  const double icw = 1.0 / (1.0 + wv);
  uint32_t ph = 0;
  bool timeout = false;

  bool late = false;  // a bounded wait of this thread expired
  // operands complete in shared memory and visible to the tensor core; false (uniform) when a
  // wait expired
  auto publish = [&]() -> bool {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    fence_before();
    return __syncthreads_or(late) == 0;
  };
  // all MMAs of the last commit complete
  auto finish = [&]() {
    if (!mbar_wait(mbar, ph)) late = true;
    ph ^= 1u;
    fence_after();
  };
  // thread 0: the level products of operands X (rows) and B (columns), 7 digits each
  auto issue_levels = [&](uint32_t X, uint32_t B) {
    fence_after();
#pragma unroll 1
    for (int kk = 0; kk < 4; kk++) {
      const uint32_t ko = kk * 32, acc = kk > 0 ? 1u : 0u;
      const uint64_t b0 = make_desc(B + ko), b4 = make_desc(B + 4 * kSlice + ko);
      uint64_t a = make_desc(X + ko);
      mma_f16(tmem, a, b0, idesc_f16(256), acc);           // p = 0, q = 0..3: blocks 0..3
      mma_f16(tmem + 256, a, b4, idesc_f16(192), acc);     // q = 4..6: blocks 4..6
      a = make_desc(X + 2 * kSlice + ko);
      mma_f16(tmem + 128, a, b0, idesc_f16(256), 1u);      // p = 2, q = 0..3: blocks 2..5
      mma_f16(tmem + 384, a, b4, idesc_f16(64), 1u);       // q = 4: block 6
      mma_f16(tmem + 448, a, make_desc(B + 5 * kSlice + ko), idesc_f16(64), acc);  // block 7
      a = make_desc(X + 4 * kSlice + ko);
      mma_f16(tmem + 256, a, b0, idesc_f16(256), 1u);      // p = 4, q = 0..3: blocks 4..7
      a = make_desc(X + 6 * kSlice + ko);
      mma_f16(tmem + 384, a, b0, idesc_f16(128), 1u);      // p = 6, q = 0, 1: blocks 6, 7
    }
    mma_commit(mbar);
  };
  // thread 0: X B^T of two-slice FP16 operands into lanes 0-63 of columns 0..63
  auto issue_pair = [&](uint32_t X, uint32_t B) {
    fence_after();
#pragma unroll 1
    for (int kk = 0; kk < 4; kk++) {
      const uint32_t ko = kk * 32;
      const uint64_t xh = make_desc(X + ko), bh = make_desc(B + ko);
      mma_f16(tmem, xh, bh, idesc_f16(64), kk > 0 ? 1u : 0u);
      mma_f16(tmem, xh, make_desc(B + kSlice + ko), idesc_f16(64), 1u);
      mma_f16(tmem, make_desc(X + kSlice + ko), bh, idesc_f16(64), 1u);
    }
    mma_commit(mbar);
  };
  // both halves of the level products: v = the thread's 8 columns of its row
  auto gather_levels = [&](long long (&v)[8]) {
    read_levels<64, 0>(tlane + 8 * gi_give, odd, v);
#pragma unroll
    for (int t = 0; t < 8; t++) xch[(8 * gi_give + t) * NB + j] = v[t];
    read_levels<64, 0>(tlane + c0, odd, v);
    fence_before();
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 8; t++) v[t] += xch[(c0 + t) * NB + j];
  };
  // 16 columns of a pair product (lanes 0-63) into Eb
  auto product_to_E = [&]() -> bool {
    if (!odd) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        float v[8];
        tmem_ld8(tlane + 16 * cg + 8 * h, v);
#pragma unroll
        for (int t = 0; t < 8; t++) Eb[j * kLdE + 16 * cg + 8 * h + t] = v[t];
      }
    }
    fence_before();
    return __syncthreads_or(late) == 0;
  };

  // a zone's G and V are copied into Y's slices (free once the last product is done) while the
  // previous zone finishes
  const double* Graw = reinterpret_cast<const double*>(sm + kOffY);
  const float* Vraw = reinterpret_cast<const float*>(sm + kOffY + 4 * kSlice);
  double gg = 0.0;
  float lam = 0.f;
  auto next_zone = [&](int32_t z) {
    while (z < nzc && nobs[z] == 0) z += gridDim.x;
    return z;
  };
  auto load = [&](int32_t z) {
    const char* gp = reinterpret_cast<const char*>(GT + (int64_t)z * N * N);
    const char* vp = reinterpret_cast<const char*>(Zv + (int64_t)z * N * N);
    if (N % 2 == 0) {  // slots of a multiple of 16 bytes
      const int ng = N * N / 2, nv = N * N / 4;
      for (int i = tid; i < ng; i += kThreads) cp_async<16>(sm + kOffY + 16 * i, gp + 16 * i);
      for (int i = tid; i < nv; i += kThreads)
        cp_async<16>(sm + kOffY + 4 * kSlice + 16 * i, vp + 16 * i);
    } else {
      for (int i = tid; i < N * N; i += kThreads) {
        cp_async<8>(sm + kOffY + 8 * i, gp + 8 * i);
        cp_async<4>(sm + kOffY + 4 * kSlice + 4 * i, vp + 4 * i);
      }
    }
    if (tid < NB) {
      lam = (tid < N) ? aux32[(int64_t)z * aux_stride + 3 * N + tid] : 0.f;
      gg = (tid < N) ? gv[(int64_t)z * N + tid] : 0.0;
    }
  };

  int32_t zl = next_zone(blockIdx.x);
  if (zl < nzc) load(zl);
  for (; zl < nzc;) {
    const int32_t zn = next_zone(zl + gridDim.x);
    double* Gz = GT + (int64_t)zl * N * N;
    cp_async_wait_all();
    __syncthreads();  // the zone has landed; the previous zone's shared values are consumed
    if (tid < NB) {
      ts.emax[tid] = 0;
      ts.s[tid] = sqrtf(1.f + fmaxf(lam, 0.f));
      const uint32_t l = __reduce_max_sync(0xffffffffu, __float_as_uint(1.f + fmaxf(lam, 0.f)));
      if (lane == 0) ts.lmax[warp] = __uint_as_float(l);
      int eg = (int)(((unsigned long long)__double_as_longlong(gg) >> 52) & 0x7FFu);
      for (int o = 16; o > 0; o >>= 1) eg = max(eg, __shfl_xor_sync(0xffffffffu, eg, o));
      if (lane == 0) ts.emaxg[warp] = eg;
    }
    if (tid == 0) {
      ts.bad = 0;
      ts.nan = 0;
    }
    // A = I + G (identity on the padding); columns along the lanes (G is symmetric)
    double ga[8];
    int em = 0;
#pragma unroll
    for (int t = 0; t < 8; t++) {
      const int c = c0 + t;
      ga[t] = ((j < N && c < N) ? Graw[c * N + j] : 0.0) + (j == c ? 1.0 : 0.0);
      em = max(em, (int)(((unsigned long long)__double_as_longlong(ga[t]) >> 52) & 0x7FFu));
    }
    {  // V vector-major: row k, K = member (four rows a warp, eight lanes a row)
      const int k = 4 * warp + (lane >> 3), ch = lane & 7;
      float x[8];
      if (N == NB) {
        const float4 a = *reinterpret_cast<const float4*>(Vraw + k * NB + 8 * ch);
        const float4 b = *reinterpret_cast<const float4*>(Vraw + k * NB + 8 * ch + 4);
        x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w;
        x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
      } else {
#pragma unroll
        for (int t = 0; t < 8; t++)
          x[t] = (k < N && 8 * ch + t < N) ? Vraw[k * N + 8 * ch + t] : (k == 8 * ch + t ? 1.f : 0.f);
      }
#pragma unroll
      for (int t = 0; t < 8; t++) x[t] *= kVScale;
      stage_f16(x, sm + kOffVk, tile_off(k, ch));
    }
    __syncthreads();  // emax cleared; s, emaxg set
    atomicMax(&ts.emax[j], em);
    if (em == 0x7FF) ts.bad = 1;  // non-finite
    if ((j >> 3) == gi) {         // the diagonal: |(A^(1/2))_ij| <= A_jj^(1/2)
      double ajj = 1.0;
#pragma unroll
      for (int t = 0; t < 8; t++) ajj = (j == c0 + t) ? ga[t] : ajj;
      const int e = (int)(((unsigned long long)__double_as_longlong(ajj) >> 52) & 0x7FFu);
      ts.fj[j] = (e - 1021) >> 1;
      // beyond 2^40 FP32 eigenpairs are no start
      if (!(ajj >= 1.0) || e > 1023 + 40) ts.bad = 1;
    }
    const int emaxg = max(ts.emaxg[0], ts.emaxg[1]), Eg = emaxg - 1022;
    if (tid < NB) ts.gi[tid] = (emaxg < 0x7FF) ? fixed_of<62>(gg, Eg) : 0;
    {  // V member-major (row a, K = vector) and W = V diag(s^(-1/2)) for Y_0
      float x[8], w[8];
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const int c = c0 + t;
        x[t] = kVScale * ((j < N && c < N) ? Vraw[c * N + j] : (j == c ? 1.f : 0.f));
        w[t] = x[t] * rsqrtf(ts.s[c]);
      }
      stage_f16(x, sm + kOffVa, own_off);
      stage_f16(w, sm + kOffW, own_off);
    }
    if (!publish()) {
      timeout = true;
      break;
    }
    const int Ei = ts.emax[j] - 1022;
    if (ts.bad) {
      if (tid == 0) {
        status[zl] = ZST_RETRY;
        atomicAdd(retries, 1);
      }
      zl = zn;
      if (zl < nzc) load(zl);  // Y's slices are read: publish() was a barrier
      continue;
    }
    if (tid == 0) issue_pair(sa + kOffW, sa + kOffW);  // Y_0 = W W^T
    {                                                  // A's digits beside the product
      long long F[8];
#pragma unroll
      for (int t = 0; t < 8; t++) F[t] = fixed_of<54>(ga[t], Ei);
      stage_digits<kSlice>(F, sm + kOffA, own_off);
    }
    long long Y[8];
    float esum = 0.f;
    finish();
    if (!product_to_E()) {
      timeout = true;
      break;
    }
#pragma unroll
    for (int t = 0; t < 8; t++) {
      const float y = Eb[j * kLdE + c0 + t] + Eb[(c0 + t) * kLdE + j];
      Y[t] = fixed_of(y, 59 - 14);  // half the sum, 128^2 taken out
    }

    float rho_prev = 0.f, rho0 = 0.f;
    uint32_t xp[8];  // (lanes 0-63) row j of the second-order part of A^(1/2) in V's basis, FP16
    float xscale = 0.f;
    bool ok = false;
#pragma unroll 1
    for (int it = 0; it < kMaxSteps; it++) {
      {  // Y rounded to 2^-54 and staged (symmetric: rows serve as rows and as columns)
        long long F[8];
#pragma unroll
        for (int t = 0; t < 8; t++) {
          F[t] = (Y[t] + 32) >> 6;
          Y[t] = F[t] * 64;
        }
        stage_digits<kSlice>(F, sm + kOffY, own_off);
      }
      if ((timeout = !publish())) break;
      if (tid == 0) issue_levels(sa + kOffA, sa + kOffY);  // Z = A Y
      finish();
      long long v[8];
      gather_levels(v);
      {  // row sums of Z, units 2^(Ei - 60) (|Y_ij| <= 1; the row's norm is A_jj^(1/2))
        long long zs = 0;
#pragma unroll
        for (int t = 0; t < 8; t++) zs += v[t];
        ts.zpart[gi][j] = zs;
      }
      __syncthreads();  // the exchange is read: Z's slices may overwrite it
      {  // Z in fixed point below its column bounds, staged with row = column (K = this row)
        unsigned long long U[8];
#pragma unroll
        for (int t = 0; t < 8; t++) {
          const int sh = 6 + ts.fj[c0 + t] - Ei;  // F = v 2^-sh
          const long long F = sh > 0 ? (v[t] + (1ll << (sh - 1))) >> sh : v[t] << (-sh);
          U[t] = (unsigned long long)F + kDigitBias;
        }
        // lanes 2i, 2i + 1 exchange columns t, t + 4, so that a lane stores pairs of K elements
        // (rows 4 apart: different banks in the swizzled layout)
#pragma unroll
        for (int t = 0; t < 4; t++) {
          const unsigned long long mine = (lane & 1) ? U[t + 4] : U[t];
          const unsigned long long give = (lane & 1) ? U[t] : U[t + 4];
          const unsigned long long got = __shfl_xor_sync(0xffffffffu, give, 1);
          uint32_t d[kDigits];
          digit_pairs((lane & 1) ? got : mine, (lane & 1) ? mine : got, d);
          const int row = c0 + t + 4 * (lane & 1);
          unsigned char* w = sm + kOffW + tile_off(row, j >> 3) + (j & 6) * 2;
#pragma unroll
          for (int p = 0; p < kDigits; p++) *reinterpret_cast<uint32_t*>(w + p * kSlice) = d[p];
        }
      }
      if ((timeout = !publish())) break;
      if (tid == 0) issue_levels(sa + kOffY, sa + kOffW);  // Y Z
      finish();
      gather_levels(v);
      float r[8];
      {
        float rm = 0.f;
#pragma unroll
        for (int t = 0; t < 8; t++) {
          const int fc = ts.fj[c0 + t];
          const long long one = (j == c0 + t) ? (1ll << (60 - fc)) : 0ll;
          r[t] = float_of(one - v[t]) * __int_as_float((fc - 60 + 127) << 23);
          rm = fmaxf(rm, fabsf(r[t]));
        }
        // non-negative floats order as their bits
        const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(rm));
        if (lane == 0) ts.rmax[warp] = __uint_as_float(m);
      }
      __syncthreads();  // the exchange is read: the correction's operands may overwrite it
      float rho = 0.f;
#pragma unroll
      for (int k = 0; k < kThreads / 32; k++) rho = fmaxf(rho, ts.rmax[k]);
      if (!(rho < 0.25f)) break;  // no start
      // a power of two sig = 2^se near 1 / rho keeps the FP16 operands in range
      const int se = 126 - (int)((__float_as_uint(fmaxf(rho, 0x1p-80f)) >> 23) & 255u);
      const float sig = __int_as_float((127 + se) << 23), isig = __int_as_float((127 - se) << 23);
#pragma unroll
      for (int t = 0; t < 8; t++) r[t] *= sig;
      stage_f16(r, sm + kOffX1, own_off);
      if ((timeout = !publish())) break;
      // lanes 0-63 hold each product's rows: 16 columns a thread
      auto stage_rows = [&](uint32_t dst) -> bool {
        if (!odd) {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            float x[8];
            tmem_ld8(tlane + 16 * cg + 8 * h, x);
#pragma unroll
            for (int t = 0; t < 8; t++) x[t] *= 1.f / kVScale;
            stage_f16(x, sm + dst, tile_off(j, 2 * cg + h));
          }
        }
        return publish();
      };
      if (tid == 0) issue_pair(sa + kOffVk, sa + kOffX1);  // [k][i] = sum_a V_ak R_ia
      finish();
      if ((timeout = !stage_rows(kOffX2))) break;
      if (tid == 0) issue_pair(sa + kOffX2, sa + kOffVk);  // R'[k][l]
      finish();
      {
        float e[16];
        if (!odd) {
          tmem_ld16(tlane + 16 * cg, e);
#pragma unroll
          for (int t = 0; t < 16; t++) e[t] *= 1.f / kVScale;
        }
        if (it == 0) {
          // the eigenvalues that R'_kk = 1 - (V^T A V)_kk / s_k^2 shows, and V^T A^(1/2) V =
          // diag(s) + X to first order: X_kl = -s_k R'_kl s_l / (s_k + s_l), k /= l
          if (!odd && cg == (j >> 4)) {
            float d = 0.f;
#pragma unroll
            for (int t = 0; t < 16; t++) d = (j == 16 * cg + t) ? e[t] : d;
            ts.s[j] *= 1.f - 0.5f * d * isig;
          }
          __syncthreads();
          rho0 = rho;
          xscale = 16.f * isig;
          if (!odd) {
            const float sj = ts.s[j];
#pragma unroll
            for (int t = 0; t < 16; t += 2) {
              float x[2];
#pragma unroll
              for (int u = 0; u < 2; u++) {
                const int l = 16 * cg + t + u;
                const float sl = ts.s[l];
                e[t + u] = __fdividef(e[t + u], sj + sl);
                x[u] = (j == l) ? 0.f : fminf(fmaxf(-0.0625f * sj * e[t + u] * sl, -6e4f), 6e4f);
              }
              xp[t / 2] = pack_f16(x[0], x[1]);
            }
            stage_f16(reinterpret_cast<float(&)[8]>(e[0]), sm + kOffX1, tile_off(j, 2 * cg));
            stage_f16(reinterpret_cast<float(&)[8]>(e[8]), sm + kOffX1, tile_off(j, 2 * cg + 1));
          }
          if ((timeout = !publish())) break;
        } else {
          // E' - (E' X + X E') / (s_k + s_l)
          if (!odd) {
            const float sj = ts.s[j];
#pragma unroll
            for (int t = 0; t < 16; t++) e[t] = __fdividef(e[t], sj + ts.s[16 * cg + t]);
            stage_f16(reinterpret_cast<float(&)[8]>(e[0]), sm + kOffX1, tile_off(j, 2 * cg));
            stage_f16(reinterpret_cast<float(&)[8]>(e[8]), sm + kOffX1, tile_off(j, 2 * cg + 1));
            *reinterpret_cast<uint4*>(sm + kOffE + tile_off(j, 2 * cg)) =
                make_uint4(xp[0], xp[1], xp[2], xp[3]);
            *reinterpret_cast<uint4*>(sm + kOffE + tile_off(j, 2 * cg + 1)) =
                make_uint4(xp[4], xp[5], xp[6], xp[7]);
          }
          if ((timeout = !publish())) break;
          if (tid == 0) {
            fence_after();
#pragma unroll 1
            for (int kk = 0; kk < 4; kk++) {
              const uint64_t eh = make_desc(sa + kOffX1 + kk * 32), xh = make_desc(sa + kOffE + kk * 32);
              mma_f16(tmem, eh, xh, idesc_f16(64), kk > 0 ? 1u : 0u);
              mma_f16(tmem, xh, eh, idesc_f16(64), 1u);
            }
            mma_commit(mbar);
          }
          finish();
          if (!odd) {
            const float sj = ts.s[j];
            float x[16];
            tmem_ld16(tlane + 16 * cg, x);
#pragma unroll
            for (int t = 0; t < 16; t++) {
              x[t] = e[t] - __fdividef(x[t] * xscale, sj + ts.s[16 * cg + t]);
              x[t] = fminf(fmaxf(x[t], -4e3f), 4e3f);  // finite whatever X is
            }
            stage_f16(reinterpret_cast<float(&)[8]>(x[0]), sm + kOffX1, tile_off(j, 2 * cg));
            stage_f16(reinterpret_cast<float(&)[8]>(x[8]), sm + kOffX1, tile_off(j, 2 * cg + 1));
          }
          if ((timeout = !publish())) break;
        }
      }
      if (tid == 0) issue_pair(sa + kOffVa, sa + kOffX1);  // [a][l] = sum_k V_ak E'_lk
      finish();
      if ((timeout = !stage_rows(kOffX2))) break;
      if (tid == 0) issue_pair(sa + kOffX2, sa + kOffVa);  // E[a][b]
      finish();
      if ((timeout = !product_to_E())) break;
      esum = 0.f;
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const float e = Eb[j * kLdE + c0 + t] + Eb[(c0 + t) * kLdE + j];
        esum += e;
        Y[t] += fixed_of(e, 59 - 7 - se);  // half the sum, 128 and 2^se taken out
      }
      esum *= (0.5f / kVScale) * isig;
      // what the correction leaves of rho: the square, the first step's basis (~ 4 rho0), with X
      // its square (~ 7 rho0^2), then as the step before, and the 22-bit products
      const float left = it == 0   ? 16.f * rho
                         : it == 1 ? fmaxf(16.f * rho0 * rho0, 0x1p-19f)
                                   : fmaxf(rho / rho_prev, 0x1p-19f);
      // at most (clustered and linear spectra: rho0 / 2 after the second step, from there on 5 times
      // the step before)
      const float most = it == 0   ? left
                         : it == 1 ? fmaxf(left, 0.5f * rho0)
                                   : fmaxf(8.f * rho / rho_prev, 0x1p-19f);
      const float lmax = fmaxf(ts.lmax[0], ts.lmax[1]);
      if (rho * left < kAccept && rho * most < fmaxf(kAccept, 0x1p-53f * lmax)) {
        ok = true;
        break;
      }
      if (it > 0 && rho > 0.5f * rho_prev) break;  // not converging
      rho_prev = rho;
    }
    if (timeout) break;
    if (!ok) {  // uniform: the FP64 eigensolve takes the zone (G is intact)
      if (tid == 0) {
        status[zl] = ZST_RETRY;
        atomicAdd(retries, 1);
      }
      zl = zn;
      if (zl < nzc) load(zl);
      continue;
    }
    if (zn < nzc) load(zn);  // on its way while this zone finishes
    // T_sym = Y. t1 = Y g, ampl = Y t1 (= A^-1 g), refined below; A^(1/2) w = w (A Y) 1 =
    // w (Z 1 + A (E 1)) with Z of the last residual and E the correction after it. Sums in 64-bit
    // fixed point: the FP64 pipe would take a cycle for two multiply-adds an SM
    {
      long long pa = 0, ys = 0;
#pragma unroll
      for (int t = 0; t < 8; t++) {
        pa += __mul64hi(Y[t] * 2, ts.gi[c0 + t]);  // units 2^(Eg - 59): |Y g| <= 8 max |g|
        ys += Y[t];
      }
      pd[gi * NB + j] = pa;
      py[gi * NB + j] = ys >> 2;
      pf[gi * NB + j] = esum;
    }
    if (N - 1 >= c0 && N - 1 < c0 + 8) {
      long long l = 0;
#pragma unroll
      for (int t = 0; t < 8; t++) l = (c0 + t == N - 1) ? Y[t] : l;
      ts.tl[j] = scaled_i64(l, -60);  // T_sym e_N
    }
    __syncthreads();
    if (tid < NB) {
      long long s = 0;
      float e = 0.f;
#pragma unroll
      for (int k = 0; k < 8; k++) {
        s += pd[k * NB + tid];
        e += pf[k * NB + tid];
      }
      ts.t1[tid] = s;
      ts.es[tid] = e;
      uint32_t m = (uint32_t)((unsigned long long)(s < 0 ? -s : s) >> 32);
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) ts.tmax[warp] = m;
    }
    __syncthreads();
    // t1 scaled up to 62 bits
    const int st = max(0, __clz((int)max(ts.tmax[0], ts.tmax[1])) - 2);
    double gd[8];  // G once more
#pragma unroll
    for (int t = 0; t < 8; t++) gd[t] = (j < N && c0 + t < N) ? Gz[(c0 + t) * N + j] : 0.0;
    {
      long long pa = 0;
#pragma unroll
      for (int t = 0; t < 8; t++) pa += __mul64hi(Y[t] * 2, ts.t1[c0 + t] << st);  // 2^(Eg - 56 - st)
      pd[gi * NB + j] = pa;
    }
    __syncthreads();
    long long s0 = 0;  // A^-1 g
    if (tid < NB) {
#pragma unroll
      for (int k = 0; k < 8; k++) s0 += pd[k * NB + tid];
      ts.t1[tid] = s0;
      uint32_t m = (uint32_t)((unsigned long long)(s0 < 0 ? -s0 : s0) >> 32);
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) ts.tmax[warp] = m;
    }
    __syncthreads();
    // One step of refinement: acceptance lets Y's residual be 2e-14, and the amplitudes, of which |g|
    // is up to lambda_max times the size, show it. r = g - A a in fixed point (modulo 2^64: the sum's
    // terms cancel) and a + Y (Y r), r and Y in FP32. Without it the increments at the observations
    // were up to 7 times as far off as an FP64 eigensolve's (geometric mean over 300 zones of 64
    // members with a linear spectrum), the mean of 26 dense cases 1.28 times (3.0 at most); with it
    // 0.03 and 0.70 (1.09). 64,800 zones of 64 members: 31.0 -> 32.8 ms with the FP32 stages.
    const int sa2 = max(0, __clz((int)max(ts.tmax[0], ts.tmax[1])) - 2);
    float yf[8];
    {
      long long ra = 4;  // __mul64hi rounds down
      float pe = 0.f;
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const int c = c0 + t;
        ra += __mul64hi(fixed_of<62>(gd[t], Ei), ts.t1[c] << sa2);  // 2^(Ei + Eg - 54 - st - sa2)
        pe = fmaf(float_of(gd[t]), ts.es[c], pe);
        yf[t] = float_of(Y[t]) * 0x1p-60f;
      }
      pd[gi * NB + j] = ra;
      pf[gi * NB + j] = pe;
    }
    __syncthreads();
    float eg1 = 0.f;  // G (E 1)
    if (tid < NB) {  // (j = tid)
      unsigned long long r = 0;
#pragma unroll
      for (int k = 0; k < 8; k++) {
        r -= (unsigned long long)pd[k * NB + tid];
        eg1 += pf[k * NB + tid];
      }
      const int k = st + sa2 - 8 - Ei;
      const long long gk = ts.gi[tid];
      r += (unsigned long long)(k >= 0 ? (k < 64 ? gk << k : 0) : gk >> min(-k, 63));
      r -= (unsigned long long)((s0 << sa2) >> min(Ei + 2, 63));  // the identity's part of A
      ts.rf[tid] = float_of((long long)r) * __int_as_float((127 + Ei - 54 - st - sa2) << 23);
    }
    __syncthreads();
    auto mul_y = [&](const float* x) {
      float p = 0.f;
#pragma unroll
      for (int t = 0; t < 8; t++) p = fmaf(yf[t], x[c0 + t], p);
      pf[gi * NB + j] = p;
      __syncthreads();
      float s = 0.f;
      if (tid < NB) {
#pragma unroll
        for (int k = 0; k < 8; k++) s += pf[k * NB + tid];
      }
      return s;
    };
    {
      const float t = mul_y(ts.rf);
      if (tid < NB) ts.tf[tid] = t;
      __syncthreads();
    }
    const float da = mul_y(ts.tf);
    double vj = 0.0;
    if (tid < NB) {
      if (tid < N) {
        // (Eg may be near the ends of FP64's exponents)
        const int h = Eg / 2;
        double a = scaled_i64(s0, Eg - 56 - st) +
                   (double)da * __longlong_as_double((long long)(h + 1023) << 52) *
                       __longlong_as_double((long long)(Eg - h + 1023) << 52);
        if (emaxg == 0x7FF) a = __longlong_as_double(0x7FF8000000000000ll);  // non-finite g
        ampl[(int64_t)zl * N + tid] = a;
        if (!(a == a) || isinf(a)) ts.nan = 1;
      }
      if (rotate) {
        long long z = 0;
        const float e = ts.es[tid] + eg1;  // (I + G) (E 1)
#pragma unroll
        for (int k = 0; k < 8; k++) z += ts.zpart[k][tid];
        // Ei is row j's exponent and j = tid for threads 0-63
        vj = (tid < N) ? (scaled_i64(z, ts.emax[tid] - 1022 - 60) + (double)e) * wv : 0.0;
        double a = vj * vj, b = vj;
        for (int o = 16; o > 0; o >>= 1) {
          a += __shfl_xor_sync(0xffffffffu, a, o);
          b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (lane == 0) {
          ts.red[warp][0] = a;
          ts.red[warp][1] = b;
        }
        ts.vj[tid] = vj;
      }
    }
    if (rotate) {
      __syncthreads();
      // Omega = P_v P_w + (1 - s_v) v w^T (zone_gram_oz.cu): T = T_sym - a u_v^T - g u_w^T + b w^T;
      // T_sym v = w / |A^(1/2) w|. |a|, |u_v| <= 2
      if (tid < NB) {
        const double inv = rsqrt(ts.red[0][0] + ts.red[1][0]);
        const double vs = (ts.red[0][1] + ts.red[1][1]) * inv, vN = ts.vj[N - 1] * inv;
        const double sgv = signbit(vN) ? -1.0 : 1.0;
        const double uvuw = fma(wv, vs, vN) + sgv * (1.0 + wv);
        const double tv = wv * inv;
        long long rs = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) rs += py[k * NB + tid];
        const double tlast = ts.tl[tid];
        const double ai = fma(sgv, tlast, tv) / (1.0 + fabs(vN));
        const double gw = fma(-uvuw, ai, fma(wv, scaled_i64(rs, -58), tlast)) * icw;
        ts.ar[tid] = __double2ll_rn(ai * 0x1p61);
        ts.gr[tid] = __double2ll_rn(gw * 0x1p60);
        ts.cr[tid] = __double2ll_rn(((1.0 - sgv) * tv - gw) * wv * 0x1p60);
        ts.t1[tid] = __double2ll_rn(fma(vj, inv, (tid == N - 1) ? sgv : 0.0) * 0x1p61);  // u_v
      }
      __syncthreads();
      const long long a = ts.ar[j], cj = ts.cr[j];
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const int c = c0 + t;
        Y[t] += cj - 4 * __mul64hi(a, ts.t1[c]);
        if (c == N - 1) Y[t] -= ts.gr[j];
      }
    }
    // T through A's slices (free), 16-byte units swizzled, so that rows leave coalesced
    if (N == NB) {
#pragma unroll
      for (int t = 0; t < 8; t += 2)
        *reinterpret_cast<double2*>(sm + kOffA + 512 * j + 16 * ((4 * gi + t / 2) ^ (j & 31))) =
            make_double2(scaled_i64(Y[t], -60), scaled_i64(Y[t + 1], -60));
    } else {
#pragma unroll
      for (int t = 0; t < 8; t++)
        if (j < N && c0 + t < N) Gz[j * N + c0 + t] = scaled_i64(Y[t], -60);
    }
    __syncthreads();  // T staged; ts.nan
    if (N == NB)
      for (int i = tid; i < NB * NB / 2; i += kThreads)
        reinterpret_cast<double2*>(Gz)[i] = *reinterpret_cast<const double2*>(
            sm + kOffA + 512 * (i >> 5) + 16 * ((i & 31) ^ ((i >> 5) & 31)));
    if (tid == 0) status[zl] = ts.nan ? ZST_NAN : 0;
    zl = zn;
  }
  cp_async_wait_all();
  if (timeout && tid == 0) {
    atomicOr(&status[zl], ZST_TIMEOUT);
    mbar_wait(mbar, ph ^ 1u);
  }
  // teardown: no MMA may still write tensor memory when it is freed
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols));
}

}  // namespace

int isqrt_oz_max_n() { return NB; }

cudaError_t zone_isqrt_oz(int N, int32_t nzc, double* d_GT, const float* d_V, const float* d_aux32,
                          const double* d_g, const int32_t* d_nobs, int rotate, double* d_ampl,
                          int32_t* d_status, int32_t* d_retries, cudaStream_t st) {
  if (N < 2 || N > NB) return cudaErrorInvalidValue;
  if (nzc <= 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k_zone_isqrt_oz, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kIsqSmem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_zone_isqrt_oz, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = sms < nzc ? sms : nzc;
  k_zone_isqrt_oz<<<grid, kThreads, kIsqSmem, st>>>(N, nzc, d_GT, d_V, d_aux32, (int)zone_eig_aux(N), d_g, d_nobs, rotate,
                                                    d_ampl, d_status, d_retries);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace oakg
