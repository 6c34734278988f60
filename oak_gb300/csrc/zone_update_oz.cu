// K5 of the plain (FP64) form on the tensor cores, ensembles of up to 64 members:
//   Sa(i1:i2,:) = Sf(i1:i2,:) T,  xa(i1:i2) = xf(i1:i2) + Sf(i1:i2,:) ampl
// (rrsqrt.F90:151,165-185,462-464) with the product as exact slices (oz_slices.cuh). T's columns
// are the first operand ([D_p ; D_(p+1)] of 64 members: M = 128 without padding, staged once a
// zone), the zone's state rows the second one in tiles of RT rows, so that a short zone costs a
// short product: Sa^T = T^T Sf^T. Column c of T and row r of Sf get a power of two each (54 bits
// below their largest element); all levels 0..7 are summed as in zone_isqrt_oz.cu, and an
// element of Sa is formed in units of 2^(E_c + F_r - 57) and rounded once to FP64. The mean is one
// FP64 multiply-add an element.
//
// RT = 32: 256 threads and 256 tensor-memory columns, two CTAs an SM, one staging while the other
// multiplies. Tiles of 64 rows (512 threads, one CTA an SM) were never ahead: 16,200 zones of 20
// rows 1.25 against 0.68 ms, of 64 rows 1.98 against 1.65, 5,000 of 1,000 rows 9.12 against 8.91,
// one of 324,000 rows 0.33 against 0.27. Reads and writes are in place safe (a tile is read before
// it is written; Sa may alias Sf, xa may alias xf). Every mbarrier wait is bounded (ZST_TIMEOUT).
// Errors: 2^-54 of a row's largest element times a column's of T, an element, which T's own absolute
// accuracy amounts to; an element of Sf far below its row's largest is not held to its own last bit.
//
// Measured, N = 64: 64,800 zones of 20 rows 2.85 ms (9.4 on the FP64 pipe, which its 2 n N^2 flops
// bind at 1.2 TFLOP/s; 1.33 GB and T's 2.1 GB take 0.5 ms), one zone of 324,000 rows 0.27 ms (2.21).
// What bounds it: the staging and the read of the levels, which run one after the other in a CTA.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "oakg_internal.cuh"
#include "oz_slices.cuh"

namespace oakg {

namespace {

constexpr uint32_t kSliceT = 64u * 128u;  // a digit slice of T: 64 members

constexpr int RT = 32;                       // state rows a tile
constexpr int TT = 8 * RT;                   // threads
constexpr int kCtas = 2;                     // an SM
constexpr uint32_t kSliceS = RT * 128u;      // a digit slice of RT state rows
constexpr uint32_t kOffS = 8 * kSliceT;      // T: 7 digit slices and a zero slice
// the exchange of the two halves' sums overlays the rows' slices
constexpr size_t kRows = 7 * (size_t)kSliceS;
static_assert(kRows >= 64 * RT * sizeof(long long), "exchange");
constexpr size_t kSmem = 1024 + kOffS + kRows;
constexpr uint32_t kCols = 8 * RT;           // tensor-memory columns

// Rows with infinities or NaN have no fixed point; they get what the sum of their products is.
__device__ __forceinline__ void mark_infinite(const double (&x)[8], int k0, unsigned long long* pos,
                                              unsigned long long* neg) {
#pragma unroll
  for (int t = 0; t < 8; t++) {
    const unsigned long long bit = 1ull << (k0 + t);
    if (isnan(x[t]) || x[t] == INFINITY) atomicOr(pos, bit);
    if (isnan(x[t]) || x[t] == -INFINITY) atomicOr(neg, bit);
  }
}
__device__ __noinline__ double infinite_row(unsigned long long pos, unsigned long long neg,
                                            const double* Tj, int N) {
  double s = 0.0;
  for (int k = 0; k < N; k++)
    if (((pos | neg) >> k) & 1) {
      const bool p = (pos >> k) & 1, n = (neg >> k) & 1;
      s += (p && n ? NAN : (p ? INFINITY : -INFINITY)) * Tj[(int64_t)k * N];
    }
  return s;
}

template <typename S>
__global__ void __launch_bounds__(TT, kCtas)
    k_zone_update_oz(int N, int32_t z0, int32_t nzc, int nranges,
                     const int64_t* __restrict__ zone_start, const S* xf, const S* Sf, int64_t ldS,
                     const double* __restrict__ T, const double* __restrict__ ampl,
                     const int32_t* __restrict__ nobs, S* xa, S* Sa, int32_t* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char dyn_raw[];
  __shared__ __align__(16) double px[8][RT];
  __shared__ double am[64];
  __shared__ int32_t emT[64], emS[RT];
  __shared__ unsigned long long s_inf[2][RT];  // a row's members at +inf, -inf (NaN: in both)
  __shared__ unsigned long long s_mbar;
  __shared__ uint32_t s_tmem;
  const uint32_t raw_addr = smem_u32(dyn_raw);
  const uint32_t pad = ((raw_addr + 1023u) & ~1023u) - raw_addr;
  unsigned char* sm = dyn_raw + pad;
  const uint32_t sa = raw_addr + pad;
  long long* xch = reinterpret_cast<long long*>(sm + kOffS);  // [RT rows][64 members]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // tensor-memory lane quarter q: members 32 (q & 1) .. + 31, odd digits for q >= 2; the thread
  // owns member j, state rows 8 gi .. 8 gi + 7 of the tile
  const int q = warp & 3, cg = warp >> 2;
  const bool odd = q >= 2;
  const int j = 32 * (q & 1) + lane, gi = 2 * cg + (odd ? 1 : 0), gi_give = 2 * cg + (odd ? 0 : 1);
  const int sr = tid % RT, sc = tid / RT;  // staging: state row, 8-member chunk
  const uint32_t mbar = smem_u32(&s_mbar);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (uint32_t i = tid; i < kSliceT / 16; i += TT)
    reinterpret_cast<uint4*>(sm + 7 * kSliceT)[i] = make_uint4(0, 0, 0, 0);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s_tmem)),
                 "r"(kCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = s_tmem;
  const uint32_t tlane = tmem + ((uint32_t)(32 * q) << 16);
  uint32_t ph = 0;
  bool late = false, timeout = false;

  // tiles [t0, t1) of zone zl, rows i1 .. i2 - 1
  auto zone_tiles = [&](int32_t zl, int64_t i1, int64_t i2, int64_t t0, int64_t t1) {
    if (nobs[zl] == 0) {
      const int64_t r0 = i1 + t0 * RT, r1 = min(i1 + t1 * RT, i2);
      for (int64_t r = r0 + tid; r < r1; r += TT) xa[r] = xf[r];
      if (Sa != Sf)
        for (int k = 0; k < N; k++)
          for (int64_t r = r0 + tid; r < r1; r += TT)
            Sa[r + (int64_t)k * ldS] = Sf[r + (int64_t)k * ldS];
      return;
    }
    // T: unit (member column c, chunk of 8 k), k along the operand row; the first tile's rows beside
    constexpr int NU = 512 / TT;
    double tv[NU][8], sv[8];
    const double* Tz = T + (int64_t)zl * N * N;
#pragma unroll
    for (int u = 0; u < NU; u++) {
      const int c = (tid + u * TT) & 63, ch = (tid + u * TT) >> 6;
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const int k = 8 * ch + t;
        tv[u][t] = (k < N && c < N) ? Tz[(int64_t)k * N + c] : 0.0;
      }
    }
    auto load_rows = [&](int64_t tile) {
      const int64_t r = i1 + tile * RT + sr;
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const int k = 8 * sc + t;
        sv[t] = (r < i2 && k < N) ? (double)Sf[r + (int64_t)k * ldS] : 0.0;
      }
    };
    load_rows(t0);
    __syncthreads();  // the previous item's shared values are consumed
    if (tid < 64) {
      emT[tid] = 0;
      am[tid] = (tid < N) ? ampl[(int64_t)zl * N + tid] : 0.0;
    }
    if (tid < RT) emS[tid] = 0, s_inf[0][tid] = s_inf[1][tid] = 0;
    __syncthreads();
    auto top = [](const double (&x)[8]) {
      int e = 0;
#pragma unroll
      for (int t = 0; t < 8; t++)
        e = max(e, (int)(((unsigned long long)__double_as_longlong(x[t]) >> 52) & 0x7FFu));
      return e;
    };
#pragma unroll
    for (int u = 0; u < NU; u++) atomicMax(&emT[(tid + u * TT) & 63], top(tv[u]));
    for (int64_t tile = t0; tile < t1; tile++) {
      const int es = top(sv);
      atomicMax(&emS[sr], es);
      if (es == 0x7FF) mark_infinite(sv, 8 * sc, &s_inf[0][sr], &s_inf[1][sr]);
      double x = 0.0;
#pragma unroll
      for (int t = 0; t < 8; t++) x = fma(sv[t], am[8 * sc + t], x);
      px[sc][sr] = x;
      __syncthreads();  // exponents and partial sums complete
      if (tile == t0) {
#pragma unroll
        for (int u = 0; u < NU; u++) {
          const int c = (tid + u * TT) & 63, ch = (tid + u * TT) >> 6;
          long long F[8];
#pragma unroll
          for (int t = 0; t < 8; t++) F[t] = fixed_of<54>(tv[u][t], emT[c] - 1022);
          stage_digits<kSliceT>(F, sm, tile_off(c, ch));
        }
      }
      {
        long long F[8];
#pragma unroll
        for (int t = 0; t < 8; t++) F[t] = fixed_of<54>(sv[t], emS[sr] - 1022);
        stage_digits<kSliceS>(F, sm + kOffS, tile_off(sr, sc));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      fence_before();
      if (__syncthreads_or(late)) {
        timeout = true;
        return;
      }
      if (tid == 0) {
        fence_after();
        const uint32_t B = sa + kOffS;
#pragma unroll 1
        for (int kk = 0; kk < 4; kk++) {
          const uint32_t ko = kk * 32, acc = kk > 0 ? 1u : 0u;
          const uint64_t b0 = make_desc(B + ko);
          // D_p D_q, p even (odd in the upper half), in column block p + q
          uint64_t a = make_desc(sa + ko);
          mma_f16(tmem, a, b0, idesc_f16(7 * RT), acc);          // p = 0, q = 0..6
          a = make_desc(sa + 2 * kSliceT + ko);
          mma_f16(tmem + 2 * RT, a, b0, idesc_f16(5 * RT), 1u);  // p = 2, q = 0..4
          mma_f16(tmem + 7 * RT, a, make_desc(B + 5 * kSliceS + ko), idesc_f16(RT), acc);
          mma_f16(tmem + 4 * RT, make_desc(sa + 4 * kSliceT + ko), b0, idesc_f16(4 * RT), 1u);
          mma_f16(tmem + 6 * RT, make_desc(sa + 6 * kSliceT + ko), b0, idesc_f16(2 * RT), 1u);
        }
        mma_commit(mbar);
      }
      // beside the product: the mean, and the next tile's rows
      const int64_t rt = i1 + tile * RT;
      if (tid < RT && rt + tid < i2) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 8; k++) s += px[k][tid];
        xa[rt + tid] = (S)((double)xf[rt + tid] + s);
      }
      if (tile + 1 < t1) load_rows(tile + 1);
      if (!mbar_wait(mbar, ph)) late = true;
      ph ^= 1u;
      fence_after();
      long long v[8];
      read_levels<RT, 3>(tlane + 8 * gi_give, odd, v);
#pragma unroll
      for (int t = 0; t < 8; t++) xch[(8 * gi_give + t) * 64 + j] = v[t];
      read_levels<RT, 3>(tlane + 8 * gi, odd, v);
      fence_before();
      __syncthreads();  // halves exchanged; tensor memory read
      if (j < N) {
        const bool cbad = emT[j] == 0x7FF;
#pragma unroll
        for (int t = 0; t < 8; t++) {
          const int r = 8 * gi + t;
          if (rt + r < i2) {
            double y = scaled_i64(v[t] + xch[r * 64 + j], emT[j] + emS[r] - 2 * 1022 - 57);
            if (cbad) y = __longlong_as_double(0x7FF8000000000000ll);
            else if (emS[r] == 0x7FF) y = infinite_row(s_inf[0][r], s_inf[1][r], Tz + j, N);
            Sa[rt + r + (int64_t)j * ldS] = (S)y;
          }
        }
      }
      __syncthreads();  // the exchange and the exponents are read
      if (tid < RT) emS[tid] = 0, s_inf[0][tid] = s_inf[1][tid] = 0;
      __syncthreads();
    }
  };

  // Work of the zones before zone z: their rows and, a zone, RT more (T's staging and the last
  // tile's padding). A CTA takes equal ranges of it: a long zone's tiles fall into several ranges,
  // short zones follow one another in one.
  const int64_t first = zone_start[z0];
  auto before = [&](int32_t z) { return zone_start[z0 + z] - first + (int64_t)RT * z; };
  const int64_t total = before(nzc);
  for (int range = blockIdx.x; range < nranges && !timeout; range += gridDim.x) {
    const int64_t w0 = total * range / nranges, w1 = total * (range + 1) / nranges;
    // the last zone that starts at or before w0, 32 pivots a step
    int32_t zl = 0;
    for (int32_t end = nzc; end - zl > 1;) {
      const int32_t step = (end - zl + 31) >> 5, p = zl + lane * step;
      const bool le = p < end && before(p) <= w0;
      zl += (__popc(__ballot_sync(0xffffffffu, le)) - 1) * step;  // (lane 0's is)
      end = min(end, zl + step);
    }
    for (; zl < nzc && !timeout; zl++) {
      const int64_t b0 = before(zl), b1 = before(zl + 1);
      if (b0 >= w1) break;
      const int64_t i1 = zone_start[z0 + zl], i2 = zone_start[z0 + zl + 1];
      const int64_t tiles = (i2 - i1 + RT - 1) / RT;
      auto cut = [&](int64_t w) {
        return w <= b0 ? 0 : (w >= b1 ? tiles : ((w - b0) * tiles + (b1 - b0 - 1)) / (b1 - b0));
      };
      const int64_t t0 = cut(w0), t1 = cut(w1);
      if (t0 < t1) zone_tiles(zl, i1, i2, t0, t1);
    }
  }
  // teardown: no MMA may still write tensor memory when it is freed
  if (__syncthreads_or(late) && tid == 0) {
    atomicOr(err, ZST_TIMEOUT);
    mbar_wait(mbar, ph ^ 1u);
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kCols));
}

}  // namespace

int update_oz_max_n() { return 64; }

template <typename S>
cudaError_t zone_update_oz(int N, int32_t z0, int32_t nzc, const int64_t* d_zone_start,
                           int32_t zone_max, const S* xf, const S* Sf, int64_t ldS,
                           const double* d_T, const double* d_ampl, const int32_t* d_nobs, S* xa,
                           S* Sa, int32_t* d_err, cudaStream_t st) {
  if (N < 1 || N > update_oz_max_n() || !Sa) return cudaErrorInvalidValue;
  if (nzc <= 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k_zone_update_oz<S>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_zone_update_oz<S>, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t grid_max = (int64_t)sms * kCtas;
  // Few zones: a range a CTA (no more than tiles). Many: as much work a range as one to four even
  // zones have, so that even zones come in whole ones.
  const int64_t tiles = std::max<int64_t>(1, (zone_max + RT - 1) / RT);
  const int64_t per = std::min<int64_t>(4, std::max<int64_t>(1, nzc / (16 * grid_max)));
  const int64_t nranges = nzc < grid_max ? std::min(nzc * tiles, grid_max) : (nzc + per - 1) / per;
  const int grid = (int)std::min(nranges, grid_max);
  k_zone_update_oz<S><<<grid, TT, kSmem, st>>>(N, z0, nzc, (int)nranges, d_zone_start, xf, Sf, ldS,
                                               d_T, d_ampl, d_nobs, xa, Sa, d_err);
  count_launches(1);
  return cudaGetLastError();
}

template cudaError_t zone_update_oz<double>(int, int32_t, int32_t, const int64_t*, int32_t,
                                            const double*, const double*, int64_t, const double*,
                                            const double*, const int32_t*, double*, double*,
                                            int32_t*, cudaStream_t);
template cudaError_t zone_update_oz<float>(int, int32_t, int32_t, const int64_t*, int32_t,
                                           const float*, const float*, int64_t, const double*,
                                           const double*, const int32_t*, float*, float*, int32_t*,
                                           cudaStream_t);

}  // namespace oakg
