// The plain (FP64) form's square-root transform without eigenvectors, ensembles of 65 to 128
// members: T = (I + G)^(-1/2) Omega and ampl = (I + G)^-1 g (rrsqrt.F90:136-185), from the
// tridiagonal form that E1 of the eigensolve leaves (zone_eig.cu).
//
// G = Q Tri Q^T by Householder reflectors; F = (I + Tri)^(-1/2) by a rational function of the
// tridiagonal matrix; T_sym = Q F Q^T by applying the reflectors to F from both sides, last one
// first, with the rank-two update that the reduction itself uses. Eigenvalues, inverse iteration,
// its re-orthogonalisation and the product U f(L) U^T are not needed.
//
// Rational function. 1/sqrt(x) = (2/pi) int_0^inf dt / (x + t^2); with t = sc(u | 1 - 1/kappa)
// the midpoint rule in u on (0, K) with m points converges like exp(-pi^2 m / log(4 sqrt(kappa)))
// on [1, kappa] (Hale, Higham & Trefethen, SIAM J. Numer. Anal. 46, 2008, method 3):
// x^(-1/2) ~ sum_j w_j / (x + c_j), w_j, c_j > 0. 12 points give the rounding level up to kappa =
// 4^2, 24 up to 4^7, 36 up to 4^11, 48 up to 4^13; a zone takes the first kappa = 4^i
// above its Gershgorin bound. Every Tri + (1 + c) I is positive definite and its inverse
// semiseparable: with L D L^T = I + Tri, the pivots of L D L^T + c from the front (D + s) and
// from the back (p) follow from the differential quotient-difference forms (Dhillon & Parlett,
// Linear Algebra Appl. 387, 2004), which add positive numbers only:
//   s_0 = c, s'_(i+1) = l_i s_i / (D_i + s_i), s = s' + c      (l_i = e_i^2 / D_i)
//   p_(N-1) = D_(N-1) + c, b_(i+1) = l_i + p_(i+1), p_i = p_(i+1) D_i / b_(i+1) + c
//   (L D L^T + c)^-1_ii = 1 / (s'_i + p_i), and a step down column i multiplies by -e_l / b_(l+1).
// A column of F is a running product a pole, all poles' terms of an element have one sign, so
// every element is exact to a few roundings: two FP64 operations an element and pole.
//
// What bounds it: the FP64 pipe (two multiply-adds a cycle and SM), N^3 of which are the
// reflectors (the products F v of all columns, the update of the lower triangle), an eighth the
// poles. The eigenvector path it replaces spent 2 N^3 on U and U f(L) U^T, besides the
// orthogonalisation: 16,200 zones of 100 members 152 ms (eigenvalues 11, inverse iteration 9, U and
// T 132) against 67.4 ms here. Per zone, of about 1.3 million cycles: 29% F v, 27% the update, 19% the
// poles' recurrences (their warp shares its partition's pipe with the other block), 6% columns of F.
// Layout: one zone a block of 256 threads, F's lower triangle in shared memory with an odd row
// stride (rows and columns are read without conflicts), two blocks an SM up to about 100 members, so
// that one block's serial recurrences run under the other's products.
//
// A zone whose Gershgorin bound is above 4^13 (or not finite), or whose I + Tri is not positive
// definite, is left to the eigenvalue stages (ZST_RETRY; Tri and the reflectors are still there).
#include <cuda_runtime.h>
#include <math.h>

#include "oakg_internal.cuh"

namespace oakg {

namespace {

constexpr int kThreads = 256;
constexpr int kMaxN = 128;
constexpr int kCh = 12;       // poles a pass (24 lanes' recurrences)
constexpr int kKappas = 13;   // kappa = 4^1 .. 4^kKappas
constexpr int kMaxPoles = 48;

// poles in use for kappa = 4^ki, a multiple of kCh: within 5e-16 of x^(-1/2) up to ki = 8 (then
// the rounding of the poles themselves, 1e-15 at 4^10, 1e-14 at 4^13)
__host__ __device__ __forceinline__ int pole_count(int ki) {
  return ki <= 2 ? 12 : (ki <= 7 ? 24 : (ki <= 11 ? 36 : 48));
}

struct PoleTable {
  double c[kKappas][kMaxPoles], w[kKappas][kMaxPoles];
};

constexpr int kMaxParts = 5;  // parts of a column's sum in F v

__host__ __device__ __forceinline__ int f_stride(int N) { return N | 1; }

size_t smem_bytes(int N) {
  return ((size_t)N * f_stride(N) + (size_t)2 * N * kCh + (size_t)(8 + kMaxParts) * kMaxN) * sizeof(double);
}

__device__ __forceinline__ double warp_sum(double x) {
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// q / x for x in FP32's normal range: an FP32 reciprocal r and the series of 1 / (1 - e),
// e = 1 - x r (below 2^-21: x's rounding to FP32 and two units of the reciprocal), to the second
// order. e is exact to 2^-53 of itself and the series' remainder is below 2^-63, so the roundings of
// q r and of the last multiply-add are what is left: within 2^-52 of the quotient.
__device__ __forceinline__ double quot(double q, double x) {
  const double r = (double)__fdividef(1.f, (float)x);
  const double e = fma(-x, r, 1.0);
  const double t = q * r;
  return fma(t, fma(e, e, e), t);
}

__global__ void __launch_bounds__(kThreads, 2)
    k_zone_sqrt64(int N, int32_t nzc, double* __restrict__ GT, const double* __restrict__ aux,
                  int aux_stride, const double* __restrict__ gv,
                  const int32_t* __restrict__ nobs, int rotate, double* __restrict__ ampl,
                  int32_t* __restrict__ status, int32_t* __restrict__ work,
                  int32_t* __restrict__ retries, int parts,
                  const __grid_constant__ PoleTable tab) {
  extern __shared__ __align__(16) unsigned char dyn_raw[];
  const int ld = f_stride(N);
  double* ratio = reinterpret_cast<double*>(dyn_raw);  // [N][kCh] -e_l / b_(l+1)
  double* xd = ratio + N * kCh;                        // [N][kCh] s' or p - c, then w / (s' + p)
  double* vec = xd + N * kCh;
  double* F = vec + (8 + kMaxParts) * kMaxN;  // [N][ld]
  double* vv[2] = {vec, vec + kMaxN};
  double* ww = vec + 2 * kMaxN;
  double* D = vec + 3 * kMaxN;
  double* lq = vec + 4 * kMaxN;
  double* es = vec + 5 * kMaxN;
  double* rs = vec + 6 * kMaxN;
  double* e2 = vec + 7 * kMaxN;
  double* part = vec + 8 * kMaxN;  // [kMaxParts][kMaxN]
  __shared__ double red[kThreads / 32];
  __shared__ int32_t s_zone, s_flag;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int col = tid & (kMaxN - 1), half = tid >> 7;

  for (;;) {
    if (tid == 0) {
      s_zone = atomicAdd(work, 1);
      s_flag = 0;
    }
    __syncthreads();
    const int32_t zl = s_zone;
    if (zl >= nzc) break;
    if (nobs[zl] == 0) {
      __syncthreads();
      continue;
    }
    double* Gz = GT + (int64_t)zl * N * N;
    const double* ax = aux + (int64_t)zl * aux_stride;
    const double scale = ax[5 * N];
    // the scaled tridiagonal: D = 1 + d, e
    if (tid < kMaxN) {
      D[tid] = tid < N ? fma(scale, ax[tid], 1.0) : 1.0;
      es[tid] = tid + 1 < N ? scale * ax[N + tid] : 0.0;
      e2[tid] = es[tid] * es[tid];
    }
    __syncthreads();
    // Gershgorin bound, every warp for itself; any NaN stays
    double bound = 0.0;
    bool finite = true;
    for (int i = lane; i < N; i += 32) {
      const double b = D[i] + (i > 0 ? fabs(es[i - 1]) : 0.0) + fabs(es[i]);
      finite = finite && b < 1e30;  // (false for a NaN)
      bound = fmax(bound, b);
    }
    for (int o = 16; o > 0; o >>= 1) bound = fmax(bound, __shfl_xor_sync(0xffffffffu, bound, o));
    finite = __all_sync(0xffffffffu, finite);
    // kappa = 4^ki >= bound
    const int ki = finite ? max(1, ((int)((__double2hiint(bound) >> 20) & 0x7FF) - 1023 + 2) >> 1)
                          : kKappas + 1;
    __syncthreads();  // D read
    if (lane == 0 && warp == (blockIdx.x & 7)) {
      bool ok = ki <= kKappas && D[0] > 0.0;
      if (ok) {
        double d = D[0];
        for (int i = 0; i + 1 < N; i++) {
          const double l = quot(e2[i], d);
          lq[i] = l;
          d = D[i + 1] - l;
          ok = ok && d > 1e-8;  // (1, but for rounding)
          D[i + 1] = d;
        }
      }
      if (!ok) s_flag = 1;
    }
    __syncthreads();
    if (s_flag) {  // uniform
      if (tid == 0) {
        status[zl] |= ZST_RETRY;
        atomicAdd(retries, 1);
      }
      __syncthreads();
      continue;
    }
    // ---- F, kCh poles at a time
    const int np = pole_count(ki);
    for (int j0 = 0; j0 < np; j0 += kCh) {
      // (another warp a pass and block: the SM partitions' FP64 pipes share these chains)
      if (warp == ((blockIdx.x + j0 / kCh) & 7)) {
        // a pole's recurrence from the front (y_(i+1) = s'_(i+1)) on one lane and from the back
        // (y_i = p_i - c) on another: both are x <- y + c, y = B x / (A + x), with (A, B) =
        // (D_i, l_i) and (l_i, D_i). Whichever comes to an element second forms w / (s' + p)
        const bool fwd = lane < kCh;
        const int j = min(fwd ? lane : lane - kCh, kCh - 1);
        const double c = tab.c[ki - 1][j0 + j], w = tab.w[ki - 1][j0 + j];
        const double* pa = fwd ? D : lq;
        const double* pb = fwd ? lq : D;
        double x = fwd ? c : D[N - 1] + c;
        double y = fwd ? 0.0 : D[N - 1];
        for (int n = 0; n < N; n++) {
          const int o = fwd ? n : N - 1 - n;  // y is this element's
          const bool second = 2 * n >= N, mid = 2 * n + 1 == N;
          if (lane < 2 * kCh) {
            double* out = xd + o * kCh + j;
            const double other = second ? *out : 0.0;
            if (second)
              *out = quot(w, y + other + c);
            else if (!mid)
              *out = y;
          }
          if (mid) {  // both at the same element: exchange
            const double other = __shfl_sync(0xffffffffu, y, fwd ? lane + kCh : lane - kCh);
            if (fwd) xd[o * kCh + j] = quot(w, y + other + c);
          }
          __syncwarp();
          if (n + 1 < N && lane < 2 * kCh) {
            const int i = fwd ? o : o - 1;
            const double a = pa[i] + x, q = pb[i] * x;
            const double r = (double)__fdividef(1.f, (float)a);
            const double e = fma(-a, r, 1.0), f = fma(e, e, e), t = q * r;
            y = fma(t, f, t);
            x = y + c;
            if (!fwd) ratio[i * kCh + j] = -es[i] * fma(r, f, r);
          }
        }
      }
      __syncthreads();
      // column i of F: two threads, half of the poles each. Sixteen columns a warp; the warps w
      // and w + 4 of an SM partition get a long and a short group
      {
        constexpr int kQ = kCh / 2;
        const int grp = warp < 4 ? warp : 11 - warp;
        const int i = 16 * grp + (lane >> 1), sub = lane & 1;
        double x[kQ];
#pragma unroll
        for (int q = 0; q < kQ; q++) x[q] = i < N ? xd[i * kCh + kQ * sub + q] : 0.0;
        const double* r = ratio + kQ * sub;
        for (int l = 16 * grp; l < N; l++) {
          if (l > i) {
#pragma unroll
            for (int q = 0; q < kQ; q++) x[q] *= r[(l - 1) * kCh + q];
          }
          double f = ((x[0] + x[1]) + (x[2] + x[3])) + (x[4] + x[5]);
          static_assert(kQ == 6, "the sum above");
          f += __shfl_xor_sync(0xffffffffu, f, 1);
          if (sub == 0 && l >= i) F[l * ld + i] = j0 ? F[l * ld + i] + f : f;
        }
      }
      __syncthreads();
    }
    // ---- T_sym = H_0 .. H_(N-3) F H_(N-3) .. H_0: F -= v w^T + w v^T with p = beta F v,
    // w = p - (beta / 2)(v . p) v; v vanishes on columns <= k
    {
      double vn = 0.0, bn = 0.0;
      if (tid > N - 3 && tid < N && N > 2) vn = Gz[(int64_t)tid * N + N - 3];
      if (N > 2) bn = ax[2 * N + N - 3];
      for (int k = N - 3; k >= 0; k--) {
        const double bk = bn;
        double* v = vv[k & 1];
        if (tid < kMaxN) v[tid] = (tid > k && tid < N) ? vn : 0.0;
        if (k > 0) {  // the next reflector, ahead
          if (tid > k - 1 && tid < N) vn = Gz[(int64_t)tid * N + k - 1];
          bn = ax[2 * N + k - 1];
        }
        __syncthreads();  // v published; the previous update done
        if (bk == 0.0) continue;  // uniform
        // F v, a column's sum in `parts` parts, so that N x parts fills the threads' rounds; v . F v
        const int S = N - 1 - k, len = (S + parts - 1) / parts;
        double pv = 0.0;
        for (int it = tid; it < N * parts; it += kThreads) {
          const int pt = it / N, c = it - pt * N;
          int i = k + 1 + pt * len;
          const int i1 = min(i + len, N);
          double s0 = 0.0, s1 = 0.0;
          for (; i + 1 < i1; i += 2) {
            s0 = fma(v[i], F[i >= c ? i * ld + c : c * ld + i], s0);
            s1 = fma(v[i + 1], F[i + 1 >= c ? (i + 1) * ld + c : c * ld + i + 1], s1);
          }
          if (i < i1) s0 = fma(v[i], F[i >= c ? i * ld + c : c * ld + i], s0);
          s0 += s1;
          part[pt * kMaxN + c] = s0;
          pv = fma(s0, v[c], pv);
        }
        pv = warp_sum(pv);
        if (lane == 0) red[warp] = pv;
        __syncthreads();
        if (32 * warp < N) {  // uniform
          double t = red[lane & 7];
          for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
          pv = t;
        }
        if (tid < N) {
          double p = part[tid];
          for (int q = 1; q < parts; q++) p += part[q * kMaxN + tid];
          ww[tid] = fma(-0.5 * bk * bk * pv, v[tid], bk * p);
        }
        __syncthreads();
        // rows k + 1 .. N - 1: the columns up to k, where v vanishes, and the triangle beyond
        // (flat indices: rows of whole warps would leave a quarter of the pipe's lanes idle)
        const int K1 = k + 1, R = S * K1, E = R + S * (S + 1) / 2;
        const float iK = 1.f / (float)K1;
        for (int it = tid; it < E; it += kThreads) {
          if (it < R) {
            int i = (int)((float)it * iK);  // within one of it / K1
            int j = it - i * K1;
            if (j < 0) i--, j += K1;
            if (j >= K1) i++, j -= K1;
            double* f = F + (K1 + i) * ld + j;
            *f = fma(-v[K1 + i], ww[j], *f);
          } else {
            const int t = it - R;
            int a = (int)((__fsqrt_rn((float)(8 * t + 1)) - 1.f) * 0.5f);
            if ((a + 1) * (a + 2) / 2 <= t) a++;
            if (a * (a + 1) / 2 > t) a--;
            const int i = K1 + a, j = K1 + t - a * (a + 1) / 2;
            double* f = F + i * ld + j;
            *f = fma(-v[i], ww[j], fma(-ww[i], v[j], *f));
          }
        }
      }
    }
    __syncthreads();
    for (int i = warp; i < N; i += kThreads / 32)  // the upper triangle
      for (int j = lane; j < i; j += 32) F[j * ld + i] = F[i * ld + j];
    // ---- amplitudes and rotation
    double* x0 = vv[0];
    double* x1 = vv[1];
    // y = T x for x in shared memory; each of the first N threads gets its row's value
    auto mul_t = [&](const double* x) {
      const int h = (N + 1) >> 1, i0 = half ? h : 0, i1 = half ? N : h;
      double a = 0.0, b = 0.0;
      __syncthreads();  // x published; the last use of part over
      if (col < N) {
        const double* row = F + col * ld;
        int i = i0;
        for (; i + 1 < i1; i += 2) {
          a = fma(row[i], x[i], a);
          b = fma(row[i + 1], x[i + 1], b);
        }
        if (i < i1) a = fma(row[i], x[i], a);
      }
      part[half * kMaxN + col] = a + b;
      __syncthreads();
      return part[col] + part[kMaxN + col];
    };
    // y = (I + G) x: G's diagonal and upper triangle are still in the zone's slot
    auto mul_a = [&](const double* x) {
      const int h = (N + 1) >> 1, i0 = half ? h : 0, i1 = half ? N : h;
      double a = 0.0;
      __syncthreads();
      if (col < N) {
        if (half == 0) a = x[col];
#pragma unroll 8
        for (int i = i0; i < i1; i++) a = fma(i < col ? Gz[i * N + col] : Gz[col * N + i], x[i], a);
      }
      part[half * kMaxN + col] = a;
      __syncthreads();
      return part[col] + part[kMaxN + col];
    };
    const double gt = tid < N ? gv[(int64_t)zl * N + tid] : 0.0;
    if (tid < kMaxN) x0[tid] = gt;
    double y = mul_t(x0);
    if (tid < kMaxN) x1[tid] = tid < N ? y : 0.0;
    y = mul_t(x1);
    // One step of refinement, a + T (T (g - A a)): the reduction's and the poles' errors leave T T g
    // off by a part of |g|, which is up to lambda_max times the amplitudes. Without it the increments at
    // the observations were 0.85 to 222 times as far off as an FP64 eigensolve's (geometric means over
    // 200 zones, 65 to 128 members, one dominant eigenvalue of 10^6 the worst), with it 0.02 to
    // 0.73. 16,200 zones of 100 members: 0.9 ms of 101 (the reduction included).
    {
      const double a0 = tid < N ? y : 0.0;
      if (tid < kMaxN) x0[tid] = a0;
      y = mul_a(x0);
      if (tid < kMaxN) x1[tid] = tid < N ? gt - y : 0.0;
      y = mul_t(x1);
      if (tid < kMaxN) x0[tid] = tid < N ? y : 0.0;
      y = a0 + mul_t(x0);
    }
    int nan_flag = 0;
    if (tid < N) {
      ampl[(int64_t)zl * N + tid] = y;
      nan_flag = !(y == y) || isinf(y);
    }
    nan_flag = __syncthreads_or(nan_flag);
    if (rotate) {
      // v = A^(1/2) 1 / |.| (A = I + G) = A (T 1), with a step of refinement for the T at hand
      // (T v = 1): the product by A amplifies the rounding of T 1
      if (tid < kMaxN) x0[tid] = tid < N ? 1.0 : 0.0;
      const double r1 = mul_t(x0);
      if (tid < kMaxN) rs[tid] = tid < N ? r1 : 0.0;
      const double y0 = mul_a(rs);
      if (tid < kMaxN) x0[tid] = tid < N ? y0 : 0.0;
      y = mul_t(x0);
      if (tid < kMaxN) x1[tid] = tid < N ? 1.0 - y : 0.0;
      y = mul_t(x1);
      if (tid < kMaxN) ww[tid] = tid < N ? y : 0.0;
      y = y0 + mul_a(ww);
      if (tid < kMaxN) x0[tid] = tid < N ? y : 0.0;
      const double ty = mul_t(x0);
      if (warp == 0) {
        double sq = 0.0, sm = 0.0;
        for (int i = lane; i < N; i += 32) {
          sq = fma(x0[i], x0[i], sq);
          sm += x0[i];
        }
        sq = warp_sum(sq);
        sm = warp_sum(sm);
        if (lane == 0) {
          red[0] = 1.0 / sqrt(sq);
          red[1] = sm;
        }
      }
      __syncthreads();
      // Omega = P_v P_w + (1 - s_v) v w^T: T = T_sym - a u_v^T - g u_w^T + b w^T
      const double inv = red[0], vN = x0[N - 1] * inv, sgv = signbit(vN) ? -1.0 : 1.0;
      const double wv = 1.0 / sqrt((double)N);
      if (tid < N) {
        const double tv = ty * inv, te = F[(N - 1) * ld + tid];
        const double uvuw = fma(wv, red[1] * inv, vN) + sgv * (1.0 + wv);
        const double ai = fma(sgv, te, tv) / (1.0 + fabs(vN));
        const double gi = fma(-uvuw, ai, fma(wv, rs[tid], te)) / (1.0 + wv);
        part[tid] = ai;
        part[kMaxN + tid] = gi;
        ww[tid] = fma(1.0 - sgv, tv, -gi) * wv;
        x1[tid] = fma(x0[tid], inv, tid == N - 1 ? sgv : 0.0);  // u_v
      }
      __syncthreads();
      for (int i = warp; i < N; i += kThreads / 32) {
        const double ai = part[i], ci = ww[i], gi = part[kMaxN + i];
        for (int j = lane; j < N; j += 32) {
          double t = fma(-ai, x1[j], F[i * ld + j]) + ci;
          if (j == N - 1) t -= gi;
          Gz[i * N + j] = t;
        }
      }
    } else {
      for (int i = warp; i < N; i += kThreads / 32)
        for (int j = lane; j < N; j += 32) Gz[i * N + j] = F[i * ld + j];
    }
    if (tid == 0 && nan_flag) status[zl] |= ZST_NAN;
    __syncthreads();
  }
}

// poles and weights of 1/sqrt(x) ~ sum_j w_j / (x + c_j) on [1, kappa]: with modulus
// k'^2 = 1 - 1/kappa, c = sc^2(u), w = (2 K / (pi m)) dn(u) / cn^2(u) at the midpoints u of m
// parts of (0, K); the upper half by u -> K - u (sc -> cs / kc), where cn would cancel.
// Amplitudes by the arithmetic-geometric mean (Abramowitz & Stegun 16.4, 16.8).
void poles(double kappa, int m, double* c, double* w) {
  const double kc = 1.0 / sqrt(kappa), k2 = (1.0 - kc) * (1.0 + kc), pi = 3.14159265358979323846;
  double a[32], cc[32], b = kc;
  a[0] = 1.0;
  cc[0] = sqrt(k2);
  int n = 0;
  while (cc[n] > 1e-17 && n < 30) {
    a[n + 1] = 0.5 * (a[n] + b);
    cc[n + 1] = 0.5 * (a[n] - b);
    b = sqrt(a[n] * b);
    n++;
  }
  const double f = 1.0 / (a[n] * m);  // 2 K / (pi m)
  for (int j = 0; j < m / 2; j++) {
    double phi = ldexp(0.5 * pi * (j + 0.5) / m, n);
    for (int i = n; i > 0; i--) phi = 0.5 * (phi + asin(cc[i] / a[i] * sin(phi)));
    const double sn = sin(phi), cn = cos(phi), dn = sqrt(kc * kc + k2 * cn * cn);
    c[j] = (sn / cn) * (sn / cn);
    w[j] = f * dn / (cn * cn);
    c[m - 1 - j] = cn / (kc * sn) * (cn / (kc * sn));
    w[m - 1 - j] = f * dn / (kc * sn * sn);
  }
}

PoleTable make_table() {
  PoleTable t = {};
  for (int k = 0; k < kKappas; k++) poles(ldexp(1.0, 2 * (k + 1)), pole_count(k + 1), t.c[k], t.w[k]);
  return t;
}

}  // namespace

int sqrt64_max_n() { return kMaxN; }

cudaError_t zone_sqrt64(int N, int32_t nzc, double* d_GT, const double* d_aux, int aux_stride,
                        const double* d_g, const int32_t* d_nobs, int rotate, double* d_ampl,
                        int32_t* d_status, int32_t* d_work, int32_t* d_retries, cudaStream_t st) {
  if (N < 3 || N > kMaxN) return cudaErrorInvalidValue;
  if (nzc <= 0) return cudaSuccess;
  static const PoleTable tab = make_table();
  const size_t smem = smem_bytes(N);
  cudaError_t e = cudaFuncSetAttribute(k_zone_sqrt64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0, bps = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_zone_sqrt64, kThreads, smem);
  if (e != cudaSuccess) return e;
  const int grid = min((int)nzc, sms * (bps > 0 ? bps : 1));
  // N x parts items over whole rounds of the block's threads: the fullest
  int parts = 2;
  auto fill = [&](int p) { return (double)N * p / ((N * p + kThreads - 1) / kThreads * kThreads); };
  for (int p = 3; p <= kMaxParts; p++)
    if (fill(p) > fill(parts) + 0.02) parts = p;
  k_zone_sqrt64<<<grid, kThreads, smem, st>>>(N, nzc, d_GT, d_aux, aux_stride, d_g, d_nobs, rotate,
                                              d_ampl, d_status, d_work, d_retries, parts, tab);
  return cudaGetLastError();
}

}  // namespace oakg
