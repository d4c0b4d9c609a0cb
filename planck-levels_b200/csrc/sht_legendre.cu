// Associated-Legendre (spin 0) and Wigner-d (spin s, first derivatives)
// recurrences of the spherical-harmonic transform, FP64, sm_100a.
//
// Reference: libsharp/sharp_core_inc.c:182-293 (seeds, scaled run-up) and
// libsharp/sharp_core_inc2.c:32-619 (synthesis/analysis kernels),
// coefficients libsharp/sharp_ylmgen_c.c:44-198.
//
// Design (not a translation of the SIMD code):
//  * one thread owns R ring pairs, lanes of a warp hold consecutive pairs, so
//    recurrence coefficients and staged a_lm are warp-uniform broadcast loads;
//  * the three-term recurrence is rewritten with a per-l normalisation c_l
//    (lambda_l = c_l mu_l) so that every step is mu_{l+1} = t_l mu_l - mu_{l-1}
//    with t_l = alpha_l x (spin 0) or a_l x -/+ b_l (spin s): 2 FP64 ops per
//    step instead of 3; c_l is folded into the staged a_lm;
//  * seeds sin^m(theta) etc. are formed as (mantissa, exponent) pairs; while
//    the recurrence value is below 2^-kSwitchExp it runs scaled (exponent
//    renormalised once per l-block, nothing accumulated), then switches to
//    plain IEEE values.  Skipped terms are < 2^-88 of the leading ones;
//  * analysis reduces over rings through shared memory within a warp and in a
//    fixed order across warps and tiles: bitwise repeatable results.
//
// What bounds it: the FP64 pipe, and in it the register ports.  A DFMA with
// three distinct register operands issues every 3 cycles per sub-partition, 2/3
// of the rate of one that repeats an operand of its predecessor or of a DADD
// (measured on register-only loops: 42.7, 56.9 and 64 lane operations per cycle
// and SM).  Per l and 32 ring pairs the loops run 4 (spin 0) or 12 (spin s)
// such operations; everything else (staging, reduction, tests on the scaled
// regime) is kept out of them.
#include <cuda_pipeline.h>
#include <cuda_runtime.h>

#include <cmath>
#include <type_traits>
#include <vector>

#include "sht_device.h"
#include "sht_recurrence.cuh"

namespace sht {

namespace {

// Sums v[0..15] over the lanes of the warp through 4 KB of shared memory:
// every lane stores its 16 values as 8 chunks of 16 bytes (chunk c at c ^ (lane
// & 7), so stores and loads touch all banks once per quarter-warp), lane
// (q, c) adds chunk c of rows q, q + 4, ..., and two exchanges add the four
// q.  Lane c < 8 returns the sums of v[2c] and v[2c + 1].
__device__ __forceinline__ double2 warp_reduce16(const double (&v)[16], double2 *buf) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < 8; ++c)
    buf[lane * 8 + (c ^ (lane & 7))] = make_double2(v[2 * c], v[2 * c + 1]);
  __syncwarp();
  const int q = lane >> 3, c = lane & 7;
  double2 w[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int row = q + 4 * t;
    w[t] = buf[row * 8 + (c ^ (row & 7))];
  }
#pragma unroll
  for (int n = 4; n >= 1; n >>= 1)
#pragma unroll
    for (int t = 0; t < n; ++t) w[t] = make_double2(w[t].x + w[t + n].x, w[t].y + w[t + n].y);
  double2 a = w[0];
  __syncwarp();
#pragma unroll
  for (int s = 8; s <= 16; s <<= 1) {
    a.x += __shfl_xor_sync(0xffffffffu, a.x, s);
    a.y += __shfl_xor_sync(0xffffffffu, a.y, s);
  }
  return a;
}

// The same in two steps, so that the next values' loop covers the latency of the
// loads, additions and exchanges: put() stores the values, sums() adds up those
// stored before.
struct WarpSums {
  double2 *buf;        // 256 entries of this warp
  double *dst;         // where the values in buf go, null: none there
  __device__ __forceinline__ double2 sums() const {
    const int lane = threadIdx.x & 31, q = lane >> 3, c = lane & 7;
    double2 a = buf[q * 8 + (c ^ q)];
#pragma unroll
    for (int t = 1; t < 8; ++t) {
      const int row = q + 4 * t;
      const double2 w = buf[row * 8 + (c ^ (row & 7))];
      a.x += w.x;
      a.y += w.y;
    }
#pragma unroll
    for (int s = 8; s <= 16; s <<= 1) {
      a.x += __shfl_xor_sync(0xffffffffu, a.x, s);
      a.y += __shfl_xor_sync(0xffffffffu, a.y, s);
    }
    return a;
  }
  // stores `a` (sums()) for the values in buf, then takes v for d
  __device__ __forceinline__ void put(double2 a, const double (&v)[16], double *d) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    if (dst && lane < 8) *reinterpret_cast<double2 *>(dst + 2 * lane) = a;
#pragma unroll
    for (int c = 0; c < 8; ++c)
      buf[lane * 8 + (c ^ (lane & 7))] = make_double2(v[2 * c], v[2 * c + 1]);
    dst = d;
    __syncwarp();
  }
  __device__ __forceinline__ void drain() {
    if (!dst) return;
    const double2 a = sums();
    const int lane = threadIdx.x & 31;
    if (lane < 8) *reinterpret_cast<double2 *>(dst + 2 * lane) = a;
    dst = nullptr;
    __syncwarp();
  }
};

// ---------------------------------------------------------------------------
// Coefficient tables (one thread per m)
// ---------------------------------------------------------------------------
__global__ void coef_spin0_kernel(int lmax, int mmax, const long long *__restrict__ moff,
                                  double *__restrict__ alpha, double *__restrict__ cfac) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m > mmax) return;
  const long long base = moff[m];
  const int L = lmax - m + 1;
  // f0[l], f1[l] as libsharp/sharp_ylmgen_c.c:160-168 (root/iroot products)
  double c_lm1 = 1.0, c_l = 1.0;  // c_{l-1}, c_l at l=m (c_{m-1} unused)
  for (int i = 0; i < L; ++i) {
    const int l = m + i;
    double f0, f1;
    if (l == m) {
      f0 = sqrt(double(2 * m + 3));
      f1 = 0.0;
    } else {
      const double tmp = sqrt(double(2 * l + 3)) * (1.0 / sqrt(double(l + 1 + m))) *
                         (1.0 / sqrt(double(l + 1 - m)));
      f0 = tmp * sqrt(double(2 * l + 1));
      f1 = tmp * sqrt(double(l + m)) * sqrt(double(l - m)) * (1.0 / sqrt(double(2 * l - 1)));
    }
    // c_{l+1} = f1[l] c_{l-1} (l >= m+1), c_{m+1} = 1
    const double c_lp1 = (l == m) ? 1.0 : f1 * c_lm1;
    cfac[base + i] = c_l;
    alpha[base + i] = (l < lmax) ? f0 * c_l / c_lp1 : 0.0;
    c_lm1 = c_l;
    c_l = c_lp1;
  }
  for (int i = L; i < L + kPad; ++i) {
    cfac[base + i] = 0.0;
    alpha[base + i] = 0.0;
  }
}

__global__ void coef_spin_kernel(int lmax, int mmax, int s, const long long *__restrict__ moff,
                                 double *__restrict__ a, double *__restrict__ b,
                                 double *__restrict__ cfac) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m > mmax) return;
  const long long base = moff[m];
  const int L = lmax - m + 1;
  const int mhi = max(m, s);
  for (int i = 0; i < L + kPad; ++i) {
    a[base + i] = 0.0;
    b[base + i] = 0.0;
    cfac[base + i] = 0.0;
  }
  // fx[l+1] for the step l -> l+1, libsharp/sharp_ylmgen_c.c:172-183
  double c_lm1 = 1.0, c_l = 1.0;
  for (int l = mhi; l <= lmax; ++l) {
    double fx0 = 0.0, fx1 = 0.0, fx2 = 0.0;
    if (l < lmax) {
      const double t = sqrt(1.0 / (l + m + 1.0)) * sqrt(1.0 / (l - m + 1.0)) *
                       sqrt(1.0 / (l + s + 1.0)) * sqrt(1.0 / (l - s + 1.0));
      fx0 = (l + 1.0) * (2 * l + 1.0) * t;
      fx1 = (l == 0) ? 0.0 : double(m) * s * (1.0 / l) * (1.0 / (l + 1.0));
      const double t2 = sqrt((l + m) / (l + m + 1.0)) * sqrt((l - m) / (l - m + 1.0)) *
                        sqrt((l + s) / (l + s + 1.0)) * sqrt((l - s) / (l - s + 1.0));
      fx2 = (l == 0) ? 0.0 : t2 * (l + 1.0) * (1.0 / l);
    }
    const double c_lp1 = (l == mhi) ? 1.0 : fx2 * c_lm1;
    const int i = l - m;
    cfac[base + i] = c_l;
    if (l < lmax) {
      const double al = fx0 * c_l / c_lp1;
      a[base + i] = al;
      b[base + i] = al * fx1;
    }
    c_lm1 = c_l;
    c_l = c_lp1;
  }
}

// ---------------------------------------------------------------------------
// Phase rows: phase[((p * ncm + comp) * 2 + hemisphere) * ms + m], ms = mmax+1
// (ring-major so the ring FFT reads and writes contiguous m runs).
// ---------------------------------------------------------------------------
__device__ __forceinline__ long long phase_row(int p, int ncm, int comp, int h, int ms) {
  return ((long long)(p * ncm + comp) * 2 + h) * ms;
}

// ---------------------------------------------------------------------------
// Coefficient staging.  Recurrence coefficients and staged a_lm are consumed
// in chunks of kChunk l-steps, copied global -> shared with cp.async into one
// of three buffers two chunks ahead of their use.  Synthesis warps stage
// privately (a __syncwarp publishes a chunk, no CTA barrier); analysis CTAs
// share the buffers and merge the publishing barrier with the one of their
// cross-warp reduction.  Inside a chunk all lanes read the same words.
// ---------------------------------------------------------------------------
constexpr int kChunk = 32;
constexpr int kWarps = 4;  // 128-thread CTAs

__device__ __forceinline__ void copy8(double *dst, const double *src) {
  __pipeline_memcpy_async(dst, src, sizeof(double));
}
__device__ __forceinline__ void copy16(double2 *dst, const double2 *src) {
  __pipeline_memcpy_async(dst, src, sizeof(double2));
}

// ---------------------------------------------------------------------------
// State of one warp's rings in the recurrence.  Below 2^-kSwitchExp a ring
// runs scaled and adds nothing (act false).  Rings that are absent or whose
// seed vanished carry zeros and stay out of the test, so a warp is in one of
// three states for each kLBlock steps: every ring scaled (only the recurrence
// runs), every ring active (no test in the loop), or some of each (analysis
// takes zero for the scaled ones; synthesis lets them add and clears their sums
// when they become active).  A warp's rings are consecutive, i.e. neighbours in
// latitude, so the mixed state is short (5% of the steps at Nside 1024 with 128
// rings a warp).
// ---------------------------------------------------------------------------
enum WarpState { kSkip, kMixed, kFull };

template <int R>
__device__ __forceinline__ WarpState warp_state(const bool (&act)[R], const bool (&live)[R]) {
  bool all = true, any = false;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    all = all && (act[r] || !live[r]);
    any = any || act[r];
  }
  if (__all_sync(0xffffffffu, all)) return kFull;
  return __any_sync(0xffffffffu, any) ? kMixed : kSkip;
}

// Spin-0 seed of one ring: (-1)^m mfac sin^m(theta) as mantissa and exponent.
__device__ __forceinline__ void spin0_start(bool valid, double sth, int m, double sgn_mfac,
                                            double &mu0, double &mu1, int &E, bool &live,
                                            bool &act) {
  XD sd = valid ? xd_pow(sth, m) : XD{0.0, 0};
  sd = xd_norm(sd.v * sgn_mfac, sd.e);
  mu0 = 0.0;
  mu1 = sd.v;
  E = sd.e;
  live = valid && sd.v != 0.0;
  act = live && E >= -kSwitchExp;
  if (act) mu1 = ldexp(mu1, E);
}

__device__ __forceinline__ void spin0_renorm(bool &live, bool &act, double &mu0, double &mu1,
                                             int &E) {
  if (!live || act) return;
  live = renorm_pair(mu1, mu0, E);
  if (live && E >= -kSwitchExp) {
    mu1 = ldexp(mu1, E);
    mu0 = ldexp(mu0, E);
    act = true;
  }
}

// ---------------------------------------------------------------------------
// Spin-0 synthesis: phase_m(p) = sum_l lambda_lm(theta_p) a_lm, split into
// even (p1) and odd (p2) l-m; north = p1+p2, south = p1-p2.
// ---------------------------------------------------------------------------
template <int NT, int R>
__global__ void __launch_bounds__(128)
synth_spin0_kernel(const int2 *__restrict__ items, const int *__restrict__ count,
                   const double *__restrict__ cth, const double *__restrict__ sth,
                   const int *__restrict__ nph_ring, const long long *__restrict__ moff,
                   const double *__restrict__ alpha, const double *__restrict__ mfac,
                   const double2 *A, int ncA, int comp0, int lmax,
                   double2 *__restrict__ phase, int ncm, int pcomp0, int ms) {
  grid_wait();
  grid_release_small();
  __shared__ __align__(16) double s_al[kWarps][3][kChunk];
  __shared__ double2 s_A[kWarps][3][kChunk * NT];
  const int2 it = items[blockIdx.x];
  const int m = it.x;
  const int cnt = count[m];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p0 = it.y * (128 * R) + w * (32 * R) + lane;   // this lane's first pair
  if (p0 - lane >= cnt) return;                            // no pair for this warp
  const long long mo = moff[m] - m;  // table index of l is mo + l
  const double *al = alpha + mo;
  const double2 *Am = A + mo * ncA + comp0;
  const int nchunks = (lmax - m + kChunk) / kChunk;
  auto stage = [&](int ch) {
    if (ch < nchunks) {
      const int lc = m + ch * kChunk;
      const int b = ch % 3;
      copy8(&s_al[w][b][lane], al + lc + lane);
#pragma unroll
      for (int t = lane; t < kChunk * NT; t += 32)
        copy16(&s_A[w][b][t], Am + (long long)(lc + t / NT) * ncA + t % NT);
    }
    __pipeline_commit();
  };
  stage(0);
  stage(1);

  double x[R], mu0[R], mu1[R];
  int E[R];
  bool act[R], live[R];
  double2 p1[R][NT], p2[R][NT];
  const double sgn_mfac = (m & 1) ? -mfac[m] : mfac[m];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int p = p0 + r * 32;
    const bool valid = p < cnt;
    x[r] = valid ? cth[p] : 0.0;
    spin0_start(valid, valid ? sth[p] : 0.0, m, sgn_mfac, mu0[r], mu1[r], E[r], live[r], act[r]);
#pragma unroll
    for (int j = 0; j < NT; ++j) p1[r][j] = p2[r][j] = make_double2(0.0, 0.0);
  }
  WarpState state = warp_state(act, live);

  for (int ch = 0; ch < nchunks; ++ch) {
    __pipeline_wait_prior(1);
    __syncwarp();
    stage(ch + 2);
    const double2 *ca = reinterpret_cast<const double2 *>(s_al[w][ch % 3]);
    const double2 *cA = s_A[w][ch % 3];
    const int nb = min(kChunk, lmax + 1 - (m + ch * kChunk));
#pragma unroll 1
    for (int sb = 0; sb < nb; sb += kLBlock) {
      if (state != kSkip) {
#pragma unroll 4
        for (int i = sb; i < sb + kLBlock; i += 2) {
          const double2 a = ca[i >> 1];
          double e[R], o[R];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double nm = fma(a.x * x[r], mu1[r], -mu0[r]);
            const double nn = fma(a.y * x[r], nm, -mu1[r]);
            e[r] = mu1[r];
            o[r] = nm;
            mu0[r] = nm;
            mu1[r] = nn;
          }
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const double2 A0 = cA[i * NT + j], A1 = cA[(i + 1) * NT + j];
#pragma unroll
            for (int r = 0; r < R; ++r) p1[r][j].x = fma(A0.x, e[r], p1[r][j].x);
#pragma unroll
            for (int r = 0; r < R; ++r) p1[r][j].y = fma(A0.y, e[r], p1[r][j].y);
#pragma unroll
            for (int r = 0; r < R; ++r) p2[r][j].x = fma(A1.x, o[r], p2[r][j].x);
#pragma unroll
            for (int r = 0; r < R; ++r) p2[r][j].y = fma(A1.y, o[r], p2[r][j].y);
          }
        }
        if (state == kFull) continue;
      } else {
#pragma unroll 4
        for (int i = sb; i < sb + kLBlock; i += 2) {
          const double2 a = ca[i >> 1];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double nm = fma(a.x * x[r], mu1[r], -mu0[r]);
            mu1[r] = fma(a.y * x[r], nm, -mu1[r]);
            mu0[r] = nm;
          }
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const bool was = act[r];
        spin0_renorm(live[r], act[r], mu0[r], mu1[r], E[r]);
        if (act[r] && !was)   // what the scaled steps added
#pragma unroll
          for (int j = 0; j < NT; ++j) p1[r][j] = p2[r][j] = make_double2(0.0, 0.0);
      }
      state = warp_state(act, live);
    }
  }

#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int p = p0 + r * 32;
    if (p >= cnt) continue;
    const bool has_s = nph_ring[2 * p + 1] > 0;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const long long row = phase_row(p, ncm, pcomp0 + j, 0, ms);
      if (!act[r]) p1[r][j] = p2[r][j] = make_double2(0.0, 0.0);
      phase[row + m] = make_double2(p1[r][j].x + p2[r][j].x, p1[r][j].y + p2[r][j].y);
      if (has_s)
        phase[row + ms + m] = make_double2(p1[r][j].x - p2[r][j].x, p1[r][j].y - p2[r][j].y);
    }
  }
}

// ---------------------------------------------------------------------------
// Spin-s synthesis (DERIV=false: E/B -> Q/U; DERIV=true: a -> d/dtheta,
// d/dphi with spin-1 functions).  Two recurrences mu+ / mu- share a_l, b_l.
//
// In the basis X1 = G - iC, X2 = G + iC (formed when the a_lm are staged) the
// sums over lw = mu+ + mu-, lx = mu- - mu+ of the definition become
//   P = sum mu+ X1,  M = sum mu- X2,  P' = sum (-1)^(l-mhi) mu+ X2,
//   M' = sum (-1)^(l-mhi) mu- X1,
//   Q_north = P + M, U_north = i (P - M), Q_south = P' + M',
//   U_south = -i (P' - M')   (south rows times flip),
// 8 FMAs per l without forming lw and lx.  With C = 0 (DERIV) X1 = X2 = G,
// and P, P' are the sum and difference of the even and odd partial sums: 4
// FMAs per l.
//
// Nside 1024, lmax 2048, one transform: 3.57 ms (FP64 pipe at 61% of its peak,
// 67% being the most with three register operands); in terms of lw and lx, with
// a test per l for the scaled regime, 4.71 ms.  Nside 2048, lmax 4096: 26.2
// against 34.5 ms.  R = 3 or 4 rings per thread: 3.68, 3.94 ms.
// ---------------------------------------------------------------------------
template <int NT, int R, bool DERIV>
__global__ void __launch_bounds__(128)
synth_spin_kernel(const int2 *__restrict__ items, const int *__restrict__ count,
                  const double *__restrict__ cth, const double *__restrict__ sth,
                  const int *__restrict__ nph_ring, const long long *__restrict__ moff,
                  const double *__restrict__ ca, const double *__restrict__ cb,
                  const double *__restrict__ pre_v, const int *__restrict__ pre_e, int s,
                  const double2 *A, int ncA, int comp0, int lmax,
                  double2 *__restrict__ phase, int ncm, int pcomp0, int ms) {
  grid_wait();
  grid_release_small();
  constexpr int NA = DERIV ? 1 : 2;  // staged alm components per transform
  constexpr int NC = NA * NT;        // staged alm entries per l
  __shared__ double2 s_ab[kWarps][3][kChunk];  // (a_l, b_l)
  __shared__ double2 s_A[kWarps][3][kChunk * NC];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int2 it = items[blockIdx.x];
  const int m = it.x;
  const int cnt = count[m];
  const int p0 = it.y * (128 * R) + w * (32 * R) + lane;   // this lane's first pair
  if (p0 - lane >= cnt) return;                            // no pair for this warp
  const int mhi = max(m, s);
  const long long mo = moff[m] - m;
  const double *aa = ca + mo;
  const double *bb = cb + mo;
  const double2 *Am = A + mo * ncA + comp0;
  const int nchunks = (lmax - mhi + kChunk) / kChunk;
  auto stage = [&](int ch) {
    if (ch < nchunks) {
      const int lc = mhi + ch * kChunk;
      const int b = ch % 3;
      copy8(&s_ab[w][b][lane].x, aa + lc + lane);
      copy8(&s_ab[w][b][lane].y, bb + lc + lane);
#pragma unroll
      for (int t = lane; t < kChunk * NC; t += 32)
        copy16(&s_A[w][b][t], Am + (long long)(lc + t / NC) * ncA + t % NC);
    }
    __pipeline_commit();
  };
  stage(0);
  stage(1);

  double x[R], mp0[R], mp1[R], mm0[R], mm1[R];
  int Ep[R], Em[R];
  bool act[R], live[R];
  // SP/SM: P and M, or (DERIV) their even parts; TP/TM: P' and M', or the odd parts
  double2 SP[R][NT], SM[R][NT], TP[R][NT], TM[R][NT];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int p = p0 + r * 32;
    const bool valid = p < cnt;
    x[r] = valid ? cth[p] : 0.0;
    live[r] = spin_start(valid, x[r], valid ? sth[p] : 0.0, m, s, pre_v[m], pre_e[m], mp0[r],
                         mp1[r], mm0[r], mm1[r], Ep[r], Em[r], act[r]);
#pragma unroll
    for (int j = 0; j < NT; ++j)
      SP[r][j] = SM[r][j] = TP[r][j] = TM[r][j] = make_double2(0.0, 0.0);
  }
  WarpState state = warp_state(act, live);

  for (int ch = 0; ch < nchunks; ++ch) {
    __pipeline_wait_prior(1);
    __syncwarp();
    stage(ch + 2);
    const double2 *cab = s_ab[w][ch % 3];
    const double2 *cA = s_A[w][ch % 3];
    const int nb = min(kChunk, lmax + 1 - (mhi + ch * kChunk));
#pragma unroll 1
    for (int sb = 0; sb < nb; sb += kLBlock) {
      if (state != kSkip) {
#pragma unroll 2
        for (int i = sb; i < sb + kLBlock; i += 2) {
#pragma unroll
          for (int odd = 0; odd < 2; ++odd) {
            const double2 ab = cab[i + odd];
            double ep[R], em[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
              ep[r] = mp1[r];
              em[r] = mm1[r];
              const double np = fma(fma(ab.x, x[r], -ab.y), mp1[r], -mp0[r]);
              const double nm = fma(fma(ab.x, x[r], ab.y), mm1[r], -mm0[r]);
              mp0[r] = mp1[r];
              mm0[r] = mm1[r];
              mp1[r] = np;
              mm1[r] = nm;
            }
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              if (DERIV) {
                const double2 G = cA[(i + odd) * NC + j];
                double2(&sp)[R][NT] = odd ? TP : SP;
                double2(&sm)[R][NT] = odd ? TM : SM;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  sp[r][j].x = fma(G.x, ep[r], sp[r][j].x);
                  sm[r][j].x = fma(G.x, em[r], sm[r][j].x);
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  sp[r][j].y = fma(G.y, ep[r], sp[r][j].y);
                  sm[r][j].y = fma(G.y, em[r], sm[r][j].y);
                }
              } else {
                const double2 X1 = cA[(i + odd) * NC + NA * j];
                const double2 X2 = cA[(i + odd) * NC + NA * j + 1];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  SP[r][j].x = fma(X1.x, ep[r], SP[r][j].x);
                  TM[r][j].x = fma(X1.x, odd ? -em[r] : em[r], TM[r][j].x);
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  SP[r][j].y = fma(X1.y, ep[r], SP[r][j].y);
                  TM[r][j].y = fma(X1.y, odd ? -em[r] : em[r], TM[r][j].y);
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  SM[r][j].x = fma(X2.x, em[r], SM[r][j].x);
                  TP[r][j].x = fma(X2.x, odd ? -ep[r] : ep[r], TP[r][j].x);
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                  SM[r][j].y = fma(X2.y, em[r], SM[r][j].y);
                  TP[r][j].y = fma(X2.y, odd ? -ep[r] : ep[r], TP[r][j].y);
                }
              }
            }
          }
        }
        if (state == kFull) continue;
      } else {
#pragma unroll 4
        for (int i = sb; i < sb + kLBlock; ++i) {
          const double2 ab = cab[i];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double np = fma(fma(ab.x, x[r], -ab.y), mp1[r], -mp0[r]);
            const double nm = fma(fma(ab.x, x[r], ab.y), mm1[r], -mm0[r]);
            mp0[r] = mp1[r];
            mm0[r] = mm1[r];
            mp1[r] = np;
            mm1[r] = nm;
          }
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const bool was = act[r];
        spin_renorm(live[r], act[r], mp0[r], mp1[r], mm0[r], mm1[r], Ep[r], Em[r]);
        if (act[r] && !was)   // what the scaled steps added
#pragma unroll
          for (int j = 0; j < NT; ++j)
            SP[r][j] = SM[r][j] = TP[r][j] = TM[r][j] = make_double2(0.0, 0.0);
      }
      state = warp_state(act, live);
    }
  }

  const double flip = ((mhi - m + s) & 1) ? -1.0 : 1.0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int p = p0 + r * 32;
    if (p >= cnt) continue;
    const bool has_s = nph_ring[2 * p + 1] > 0;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const long long rq = phase_row(p, ncm, pcomp0 + 2 * j, 0, ms);
      const long long ru = phase_row(p, ncm, pcomp0 + 2 * j + 1, 0, ms);
      double2 P = SP[r][j], M = SM[r][j], Pd = TP[r][j], Md = TM[r][j];
      if (!act[r]) P = M = Pd = Md = make_double2(0.0, 0.0);
      if (DERIV) {
        const double2 pe = P, po = Pd, me = M, mo_ = Md;
        P = make_double2(pe.x + po.x, pe.y + po.y);
        Pd = make_double2(pe.x - po.x, pe.y - po.y);
        M = make_double2(me.x + mo_.x, me.y + mo_.y);
        Md = make_double2(me.x - mo_.x, me.y - mo_.y);
      }
      phase[rq + m] = make_double2(P.x + M.x, P.y + M.y);
      phase[ru + m] = make_double2(M.y - P.y, P.x - M.x);
      if (has_s) {
        phase[rq + ms + m] = make_double2(flip * (Pd.x + Md.x), flip * (Pd.y + Md.y));
        phase[ru + ms + m] = make_double2(flip * (Pd.y - Md.y), flip * (Md.x - Pd.x));
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Analysis.  One CTA of W warps per m loops over tiles of 32*W*R ring pairs.
// Per l-block (LB steps, LB*VPL == 16 values) every lane accumulates its R
// rings' contributions; the sums over the warp (two each in lanes 0 .. 7) go to
// a per-warp shared array for the whole chunk.  After the next chunk's barrier
// (the same one that publishes staged coefficients) the warps share out the
// sub-blocks, add the warps' sums in a fixed order and store them (first tile)
// or add them (later tiles; the same thread owns an entry in every tile) to
// Aout, which this CTA owns: bitwise repeatable, one barrier per kAChunk l-steps.
// Every row l in [m, lmax] is written.
//
// The reduction through shared memory takes 8 stores, 8 loads, 18 additions and
// 8 shuffles per 16 values (warp_reduce16); recursive halving with shuffles took
// 31 exchanges of a double per 32 values, each with two selects, two shuffles and
// an addition, and left the FP64 pipe at 40%.  With the former and the loops free
// of tests, Nside 1024 / lmax 2048: spin 2 4.72 ms, spin 0 1.70 (before: 6.11 and
// 1.99); Nside 2048 / lmax 4096: 32.9 and 11.8 (44.8 and 14.1).  Overlapping the
// reduction with the next values' loop (WarpSums) is worth 1.5 ms of that at spin
// 2 (R = 3; R = 4 without it 34.4, with it 34.1).  Rings of a thread spread over
// the tile (equal work for the warps between two barriers), with loops compiled
// for each number of active ones: 5.1-5.3 and 1.94 ms, so a warp's rings stay
// consecutive.  The contraction on the FP64 tensor instructions fills 4 (spin s)
// or 2 (spin 0) of the 8 columns of an m8n8k4 with one transform: no gain.
// ---------------------------------------------------------------------------
// l-steps per chunk: as many as keep the CTAs per SM (the warps' sums of two
// chunks lie in shared memory).  Spin 0: 256 (Nside 2048: 11.8 ms, 12.3 with 64),
// spin s: 128 (34.4 ms at R = 4, 34.8 with 64, 40.5 with 256).
template <int VPL, int W>
constexpr int kAChunkOf = VPL * W >= 32 ? 32 : VPL * W > 16 ? 64 : 512 / VPL;
constexpr int kRed = 16;   // values per transpose-reduction

template <int VPL, int W>
__device__ __forceinline__ void flush_chunk(const double *wred, int nwarps, bool first, int l0,
                                            int lmax, long long mo, int ncA, int comp0,
                                            double *__restrict__ Aout) {
  constexpr int ld = kAChunkOf<VPL, W> * VPL;
  const int n = min(kAChunkOf<VPL, W>, lmax + 1 - l0) * VPL;
  for (int t = threadIdx.x; t < n; t += 32 * W) {
    double acc = wred[t];
    for (int w = 1; w < nwarps; ++w) acc += wred[w * ld + t];
    double *out = Aout + ((mo + l0 + t / VPL) * ncA + comp0) * 2 + t % VPL;
    // the same thread owns an entry in every tile, so its additions are in order;
    // as reductions they do not wait for the old value
    if (first) *out = acc;
    else atomicAdd(out, acc);
  }
}

// Dynamic shared memory of an analysis CTA: the warps' transposition buffers and
// their sums of two chunks.
template <int VPL, int W>
constexpr size_t anal_smem() {
  return sizeof(double) * W * (32 * kRed + 2 * kAChunkOf<VPL, W> * VPL);
}
__host__ __device__ constexpr int anal_min_blocks(int spin, int NT, int R, int W) {
  return W == 8 ? (NT * (spin + 1) > 2 ? 1 : 2) : NT > 1 ? 2 : spin == 0 || R <= 2 ? 4 : 3;
}

// Rows [l0, l1) of this CTA's m that no ring reaches.
template <int VPL>
__device__ __forceinline__ void zero_rows(int l0, int l1, long long mo, int ncA, int comp0,
                                          double *__restrict__ Aout) {
  for (int t = threadIdx.x; t < (l1 - l0) * VPL; t += blockDim.x)
    Aout[((mo + l0 + t / VPL) * ncA + comp0) * 2 + t % VPL] = 0.0;
}

// Phase factors of rings that are not active yet are multiplied by zero in the
// mixed state.  Those that are not finite must not enter there: hold() moves
// them to local memory and leaves zeros until release() at the ring's
// activation.
template <int N>
__device__ __forceinline__ bool hold(double *(&f)[N], volatile double *kept) {
  double t = 0.0;
#pragma unroll
  for (int k = 0; k < N; ++k) t += 0.0 * *f[k];
  if (t == 0.0) return false;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    kept[k] = *f[k];
    *f[k] = 0.0;
  }
  return true;
}
template <int N>
__device__ __forceinline__ void release(double *(&f)[N], const volatile double *kept) {
#pragma unroll
  for (int k = 0; k < N; ++k) *f[k] = kept[k];
}

template <int NT, int R, int W>
__global__ void __launch_bounds__(32 * W, anal_min_blocks(0, NT, R, W))
anal_spin0_kernel(const int *__restrict__ count, const double *__restrict__ cth,
                  const double *__restrict__ sth, const int *__restrict__ nph_ring,
                  const long long *__restrict__ moff, const double *__restrict__ alpha,
                  const double *__restrict__ mfac, const double2 *phase, int ncm,
                  int pcomp0, int lmax, int ms, double *__restrict__ Aout, int ncA,
                  int comp0) {
  grid_wait();
  grid_release_small();
  constexpr int VPL = 2 * NT;
  constexpr int LB = kRed / VPL, kAChunk = kAChunkOf<VPL, W>;
  // not with W = 8 (more warps cover the latency) or R = 4 (no registers for it)
  constexpr bool kOverlap = W == 4 && R < 4;
  static_assert(LB % 2 == 0 && kLBlock % LB == 0, "l-block must be even and divide kLBlock");
  extern __shared__ double2 smem[];
  double2(*red)[32 * kRed / 2] = reinterpret_cast<double2(*)[32 * kRed / 2]>(smem);
  double(*wred)[W][kAChunk * VPL] =
      reinterpret_cast<double(*)[W][kAChunk * VPL]>(smem + W * (32 * kRed / 2));
  __shared__ __align__(16) double s_al[3][kAChunk];
  const int m = blockIdx.x;
  const int cnt = count[m];
  const long long mo = moff[m] - m;
  if (cnt == 0) {
    zero_rows<VPL>(m, lmax + 1, mo, ncA, comp0, Aout);
    return;
  }
  const double *al = alpha + mo;
  const double sgn_mfac = (m & 1) ? -mfac[m] : mfac[m];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nchunks = (lmax - m + kAChunk) / kAChunk;
  auto stage = [&](int ch) {
    const int l0 = m + ch * kAChunk;
    // up to the end of the last kLBlock steps (inside the table's padding)
    if (ch < nchunks)
      for (int t = threadIdx.x; t < min(kAChunk, lmax + kLBlock - l0); t += 32 * W)
        copy8(&s_al[ch % 3][t], al + l0 + t);
    __pipeline_commit();
  };

  for (int tb = 0; tb < cnt; tb += 32 * W * R) {
    stage(0);
    stage(1);
    const int nwarps = min(W, (cnt - tb + 32 * R - 1) / (32 * R));
    const int p0 = tb + warp * (32 * R) + lane;
    double x[R], mu0[R], mu1[R];
    int E[R];
    bool act[R], live[R];
    double2 P1[R][NT], P2[R][NT];
    volatile double kept[R][NT][4];
    unsigned held = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int p = p0 + r * 32;
      const bool valid = p < cnt;
      x[r] = valid ? cth[p] : 0.0;
      spin0_start(valid, valid ? sth[p] : 0.0, m, sgn_mfac, mu0[r], mu1[r], E[r], live[r],
                  act[r]);
      const bool has_s = live[r] && nph_ring[2 * p + 1] > 0;   // dead rings stay out of the sums
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const long long row = phase_row(live[r] ? p : 0, ncm, pcomp0 + j, 0, ms);
        const double2 n = live[r] ? phase[row + m] : make_double2(0.0, 0.0);
        const double2 sv = has_s ? phase[row + ms + m] : make_double2(0.0, 0.0);
        P1[r][j] = make_double2(n.x + sv.x, n.y + sv.y);
        P2[r][j] = make_double2(n.x - sv.x, n.y - sv.y);
        double *f[4] = {&P1[r][j].x, &P1[r][j].y, &P2[r][j].x, &P2[r][j].y};
        if (!act[r] && hold(f, kept[r][j])) held |= 1u << (r * NT + j);
      }
    }
    WarpState state = warp_state(act, live);

    for (int ch = 0; ch < nchunks; ++ch) {
      __pipeline_wait_prior(1);
      __syncthreads();
      stage(ch + 2);
      if (ch > 0)
        flush_chunk<VPL, W>(wred[(ch - 1) & 1][0], nwarps, tb == 0, m + (ch - 1) * kAChunk, lmax,
                            mo, ncA, comp0, Aout);
      if (warp >= nwarps) continue;
      WarpSums ws{red[warp], nullptr};
      const double2 *ca = reinterpret_cast<const double2 *>(s_al[ch % 3]);
      const int nb = min(kAChunk, lmax + 1 - (m + ch * kAChunk));
#pragma unroll 1
      for (int b0 = 0; b0 < nb; b0 += kLBlock) {
        auto steps = [&](auto masked) {
          constexpr bool MASK = decltype(masked)::value;
#pragma unroll 1
          for (int sb = b0 / LB; sb < (b0 + kLBlock) / LB; ++sb) {
            double2 sum = make_double2(0.0, 0.0);
            if (kOverlap) sum = ws.sums();   // of the previous values
            double v[kRed];
#pragma unroll
            for (int i = 0; i < LB; i += 2) {
              const double2 a = ca[(sb * LB + i) >> 1];
#pragma unroll
              for (int r = 0; r < R; ++r) {
                const double nm = fma(a.x * x[r], mu1[r], -mu0[r]);
                const double nn = fma(a.y * x[r], nm, -mu1[r]);
                const double e = MASK && !act[r] ? 0.0 : mu1[r];
                const double o = MASK && !act[r] ? 0.0 : nm;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                  double *ve = v + i * VPL + 2 * j, *vo = ve + VPL;
                  ve[0] = r == 0 ? e * P1[r][j].x : fma(e, P1[r][j].x, ve[0]);
                  ve[1] = r == 0 ? e * P1[r][j].y : fma(e, P1[r][j].y, ve[1]);
                  vo[0] = r == 0 ? o * P2[r][j].x : fma(o, P2[r][j].x, vo[0]);
                  vo[1] = r == 0 ? o * P2[r][j].y : fma(o, P2[r][j].y, vo[1]);
                }
                mu0[r] = nm;
                mu1[r] = nn;
              }
            }
            if (kOverlap) {
              ws.put(sum, v, &wred[ch & 1][warp][sb * kRed]);
            } else {
              sum = warp_reduce16(v, red[warp]);
              if (lane < kRed / 2)
                *reinterpret_cast<double2 *>(&wred[ch & 1][warp][sb * kRed + 2 * lane]) = sum;
            }
          }
        };
        if (state == kFull) {
          steps(std::false_type{});
          continue;
        }
        if (state == kMixed) {
          steps(std::true_type{});
        } else {
#pragma unroll 4
          for (int i = b0; i < b0 + kLBlock; i += 2) {
            const double2 a = ca[i >> 1];
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const double nm = fma(a.x * x[r], mu1[r], -mu0[r]);
              mu1[r] = fma(a.y * x[r], nm, -mu1[r]);
              mu0[r] = nm;
            }
          }
          for (int t = lane; t < kLBlock * VPL; t += 32) wred[ch & 1][warp][b0 * VPL + t] = 0.0;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const bool was = act[r];
          spin0_renorm(live[r], act[r], mu0[r], mu1[r], E[r]);
          if (held && act[r] && !was)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              double *f[4] = {&P1[r][j].x, &P1[r][j].y, &P2[r][j].x, &P2[r][j].y};
              if (held >> (r * NT + j) & 1) release(f, kept[r][j]);
            }
        }
        state = warp_state(act, live);
      }
      ws.drain();
    }
    __pipeline_wait_prior(0);
    __syncthreads();
    flush_chunk<VPL, W>(wred[(nchunks - 1) & 1][0], nwarps, tb == 0, m + (nchunks - 1) * kAChunk,
                        lmax, mo, ncA, comp0, Aout);
    __syncthreads();
  }
}

// Spin-s analysis (E/B from Q/U): per l, (G.re, G.im, C.re, C.im) per
// transform (saddstep2, libsharp/sharp_core_inc2.c:338-364), written directly
// in terms of mu+ and mu- (lw = mu+ + mu-, lx = mu- - mu+):
//   lw X - lx Y = mu+ (X+Y) + mu- (X-Y),   lw X + lx Y = mu+ (X-Y) + mu- (X+Y)
// so each output takes 2 FMAs and lw, lx are never formed.  h / g hold the
// combined phase factors of mu+ / mu- for even l-mhi; those of odd l-mhi are
// the same eight numbers in reverse order with alternating signs.
template <int NT, int R, int W>
__global__ void __launch_bounds__(32 * W, anal_min_blocks(1, NT, R, W))
anal_spin_kernel(const int *__restrict__ count, const double *__restrict__ cth,
                 const double *__restrict__ sth, const int *__restrict__ nph_ring,
                 const long long *__restrict__ moff, const double *__restrict__ ca,
                 const double *__restrict__ cb, const double *__restrict__ pre_v,
                 const int *__restrict__ pre_e, int s, const double2 *phase,
                 int ncm, int pcomp0, int lmax, int ms, double *__restrict__ Aout, int ncA,
                 int comp0) {
  grid_wait();
  grid_release_small();
  constexpr int VPL = 4 * NT;
  constexpr int LB = kRed / VPL, kAChunk = kAChunkOf<VPL, W>;
  constexpr bool kOverlap = W == 4;   // as at spin 0
  static_assert(LB % 2 == 0 && kLBlock % LB == 0, "l-block must be even and divide kLBlock");
  extern __shared__ double2 smem[];
  double2(*red)[32 * kRed / 2] = reinterpret_cast<double2(*)[32 * kRed / 2]>(smem);
  double(*wred)[W][kAChunk * VPL] =
      reinterpret_cast<double(*)[W][kAChunk * VPL]>(smem + W * (32 * kRed / 2));
  __shared__ double2 s_ab[3][kAChunk];
  const int m = blockIdx.x;
  const int cnt = count[m];
  const int mhi = max(m, s);
  const long long mo = moff[m] - m;
  zero_rows<VPL>(m, cnt == 0 ? lmax + 1 : mhi, mo, ncA, comp0, Aout);
  if (cnt == 0) return;
  const double *aa = ca + mo;
  const double *bb = cb + mo;
  const double flip = ((mhi - m + s) & 1) ? -1.0 : 1.0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nchunks = (lmax - mhi + kAChunk) / kAChunk;
  auto stage = [&](int ch) {
    const int l0 = mhi + ch * kAChunk;
    // up to the end of the last kLBlock steps (inside the tables' padding)
    if (ch < nchunks)
      for (int t = threadIdx.x; t < 2 * min(kAChunk, lmax + kLBlock - l0); t += 32 * W)
        copy8(reinterpret_cast<double *>(&s_ab[ch % 3][t >> 1]) + (t & 1),
              ((t & 1) ? bb : aa) + l0 + (t >> 1));
    __pipeline_commit();
  };

  for (int tb = 0; tb < cnt; tb += 32 * W * R) {
    stage(0);
    stage(1);
    const int nwarps = min(W, (cnt - tb + 32 * R - 1) / (32 * R));
    const int p0 = tb + warp * (32 * R) + lane;
    double x[R], mp0[R], mp1[R], mm0[R], mm1[R];
    int Ep[R], Em[R];
    bool act[R], live[R];
    double h[R][NT][4], g[R][NT][4];   // G.re, G.im, C.re, C.im
    volatile double kept[R][NT][8];
    unsigned held = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int p = p0 + r * 32;
      const bool valid = p < cnt;
      x[r] = valid ? cth[p] : 0.0;
      live[r] = spin_start(valid, x[r], valid ? sth[p] : 0.0, m, s, pre_v[m], pre_e[m],
                           mp0[r], mp1[r], mm0[r], mm1[r], Ep[r], Em[r], act[r]);
      const bool has_s = live[r] && nph_ring[2 * p + 1] > 0;   // dead rings stay out of the sums
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const long long rq = phase_row(live[r] ? p : 0, ncm, pcomp0 + 2 * j, 0, ms);
        const long long ru = phase_row(live[r] ? p : 0, ncm, pcomp0 + 2 * j + 1, 0, ms);
        const double2 qn = live[r] ? phase[rq + m] : make_double2(0.0, 0.0);
        const double2 un = live[r] ? phase[ru + m] : make_double2(0.0, 0.0);
        double2 qs = has_s ? phase[rq + ms + m] : make_double2(0.0, 0.0);
        double2 us = has_s ? phase[ru + ms + m] : make_double2(0.0, 0.0);
        qs.x *= flip; qs.y *= flip; us.x *= flip; us.y *= flip;
        const double2 P1q = make_double2(qn.x + qs.x, qn.y + qs.y);
        const double2 P2q = make_double2(qn.x - qs.x, qn.y - qs.y);
        const double2 P1u = make_double2(un.x + us.x, un.y + us.y);
        const double2 P2u = make_double2(un.x - us.x, un.y - us.y);
        // even offset: px = p1, py = p2
        //   G.re = lw P1q.re - lx P2u.im   G.im = lw P1q.im + lx P2u.re
        //   C.re = lw P1u.re + lx P2q.im   C.im = lw P1u.im - lx P2q.re
        // odd offset: px = p2, py = p1
        h[r][j][0] = P1q.x + P2u.y; g[r][j][0] = P1q.x - P2u.y;
        h[r][j][1] = P1q.y - P2u.x; g[r][j][1] = P1q.y + P2u.x;
        h[r][j][2] = P1u.x - P2q.y; g[r][j][2] = P1u.x + P2q.y;
        h[r][j][3] = P1u.y + P2q.x; g[r][j][3] = P1u.y - P2q.x;
        double *f[8] = {&h[r][j][0], &h[r][j][1], &h[r][j][2], &h[r][j][3],
                        &g[r][j][0], &g[r][j][1], &g[r][j][2], &g[r][j][3]};
        if (!act[r] && hold(f, kept[r][j])) held |= 1u << (r * NT + j);
      }
    }
    WarpState state = warp_state(act, live);

    for (int ch = 0; ch < nchunks; ++ch) {
      __pipeline_wait_prior(1);
      __syncthreads();
      stage(ch + 2);
      if (ch > 0)
        flush_chunk<VPL, W>(wred[(ch - 1) & 1][0], nwarps, tb == 0, mhi + (ch - 1) * kAChunk, lmax,
                            mo, ncA, comp0, Aout);
      if (warp >= nwarps) continue;
      WarpSums ws{red[warp], nullptr};
      const double2 *cab = s_ab[ch % 3];
      const int nb = min(kAChunk, lmax + 1 - (mhi + ch * kAChunk));
#pragma unroll 1
      for (int b0 = 0; b0 < nb; b0 += kLBlock) {
        auto steps = [&](auto masked) {
          constexpr bool MASK = decltype(masked)::value;
#pragma unroll 1
          for (int sb = b0 / LB; sb < (b0 + kLBlock) / LB; ++sb) {
            double2 sum = make_double2(0.0, 0.0);
            if (kOverlap) sum = ws.sums();   // of the previous values
            double v[kRed];
#pragma unroll
            for (int i = 0; i < LB; ++i) {
              const double2 ab = cab[sb * LB + i];
#pragma unroll
              for (int r = 0; r < R; ++r) {
                const double ep = MASK && !act[r] ? 0.0 : mp1[r];
                const double em = MASK && !act[r] ? 0.0 : mm1[r];
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                  double *o = v + i * VPL + 4 * j;
#pragma unroll
                  for (int k = 0; k < 4; ++k) {
                    // odd: +h3, -h2, -h1, +h0
                    const double f = !(i & 1)             ? h[r][j][k]
                                     : (k == 1 || k == 2) ? -h[r][j][3 - k]
                                                          : h[r][j][3 - k];
                    o[k] = r == 0 ? ep * f : fma(ep, f, o[k]);
                  }
#pragma unroll
                  for (int k = 0; k < 4; ++k) {
                    // odd: -g3, +g2, +g1, -g0
                    const double f = !(i & 1)             ? g[r][j][k]
                                     : (k == 1 || k == 2) ? g[r][j][3 - k]
                                                          : -g[r][j][3 - k];
                    o[k] = fma(em, f, o[k]);
                  }
                }
                const double np = fma(fma(ab.x, x[r], -ab.y), mp1[r], -mp0[r]);
                const double nm = fma(fma(ab.x, x[r], ab.y), mm1[r], -mm0[r]);
                mp0[r] = mp1[r];
                mm0[r] = mm1[r];
                mp1[r] = np;
                mm1[r] = nm;
              }
            }
            if (kOverlap) {
              ws.put(sum, v, &wred[ch & 1][warp][sb * kRed]);
            } else {
              sum = warp_reduce16(v, red[warp]);
              if (lane < kRed / 2)
                *reinterpret_cast<double2 *>(&wred[ch & 1][warp][sb * kRed + 2 * lane]) = sum;
            }
          }
        };
        if (state == kFull) {
          steps(std::false_type{});
          continue;
        }
        if (state == kMixed) {
          steps(std::true_type{});
        } else {
#pragma unroll 4
          for (int i = b0; i < b0 + kLBlock; ++i) {
            const double2 ab = cab[i];
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const double np = fma(fma(ab.x, x[r], -ab.y), mp1[r], -mp0[r]);
              const double nm = fma(fma(ab.x, x[r], ab.y), mm1[r], -mm0[r]);
              mp0[r] = mp1[r];
              mm0[r] = mm1[r];
              mp1[r] = np;
              mm1[r] = nm;
            }
          }
          for (int t = lane; t < kLBlock * VPL; t += 32) wred[ch & 1][warp][b0 * VPL + t] = 0.0;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const bool was = act[r];
          spin_renorm(live[r], act[r], mp0[r], mp1[r], mm0[r], mm1[r], Ep[r], Em[r]);
          if (held && act[r] && !was)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              double *f[8] = {&h[r][j][0], &h[r][j][1], &h[r][j][2], &h[r][j][3],
                              &g[r][j][0], &g[r][j][1], &g[r][j][2], &g[r][j][3]};
              if (held >> (r * NT + j) & 1) release(f, kept[r][j]);
            }
        }
        state = warp_state(act, live);
      }
      ws.drain();
    }
    __pipeline_wait_prior(0);
    __syncthreads();
    flush_chunk<VPL, W>(wred[(nchunks - 1) & 1][0], nwarps, tb == 0, mhi + (nchunks - 1) * kAChunk,
                        lmax, mo, ncA, comp0, Aout);
    __syncthreads();
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
void launch_coef_tables(CoefPlan &cp, cudaStream_t st) {
  ProfScope ps("coef_tables", st);
  const int threads = 128;
  const int blocks = (cp.mmax + 1 + threads - 1) / threads;
  if (cp.spin == 0)
    coef_spin0_kernel<<<blocks, threads, 0, st>>>(cp.lmax, cp.mmax, cp.d_moff, cp.alpha, cp.cfac);
  else
    coef_spin_kernel<<<blocks, threads, 0, st>>>(cp.lmax, cp.mmax, cp.spin, cp.d_moff, cp.alpha,
                                                 cp.beta, cp.cfac);
  SHT_CUDA(cudaGetLastError());
}

void launch_legendre_synth(const JobDesc &job, const GeomPlan &gp, const CoefPlan &cp,
                           const double2 *A, int ncA, int comp0, int nt, double2 *phase,
                           int ncm, int pcomp0, cudaStream_t st) {
  const int nitems = int(gp.synth_items.size());
  if (nitems == 0) return;
  ProfScope ps("legendre_synth", st);
  const bool deriv = job.type == SHARP_ALM2MAP_DERIV1;
  SHT_REQUIRE(gp.synth_tile == 128 || gp.synth_tile == 256, "synthesis tile mismatch");
  auto spin0 = [&](auto kernel) {
    launch_overlapped(kernel, dim3(nitems), 128, 0, st, gp.items, gp.count, gp.cth, gp.sth, gp.nph,
                      cp.d_moff, cp.alpha, cp.seed, A, ncA, comp0, job.lmax, phase, ncm, pcomp0,
                      job.mmax + 1);
  };
  auto spins = [&](auto kernel) {
    launch_overlapped(kernel, dim3(nitems), 128, 0, st, gp.items, gp.count, gp.cth, gp.sth, gp.nph,
                      cp.d_moff, cp.alpha, cp.beta, cp.seed, cp.seed_exp, cp.spin, A, ncA, comp0,
                      job.lmax, phase, ncm, pcomp0, job.mmax + 1);
  };
  auto width = [&](auto r) {
    constexpr int RV = decltype(r)::value;
    if (job.spin == 0 && !deriv) {
      if (nt == 1) spin0(synth_spin0_kernel<1, RV>);
      else if (nt == 2) spin0(synth_spin0_kernel<2, RV>);
      else spin0(synth_spin0_kernel<4, RV>);
    } else if (deriv) {
      if (nt == 1) spins(synth_spin_kernel<1, RV, true>);
      else spins(synth_spin_kernel<2, RV, true>);
    } else {
      if (nt == 1) spins(synth_spin_kernel<1, RV, false>);
      else spins(synth_spin_kernel<2, RV, false>);
    }
  };
  if (gp.synth_tile == 128) width(std::integral_constant<int, 1>{});
  else width(std::integral_constant<int, 2>{});
  SHT_CUDA(cudaGetLastError());
}

void launch_legendre_anal(const JobDesc &job, const GeomPlan &gp, const CoefPlan &cp,
                          const double2 *phase, int ncm, int pcomp0, int nt, double *Aout,
                          int ncA, int comp0, cudaStream_t st) {
  const int nblocks = job.mmax + 1;
  ProfScope ps("legendre_anal", st);
  auto spin0 = [&](auto nt_, auto r_, auto w_) {
    constexpr int NT = decltype(nt_)::value, R = decltype(r_)::value, W = decltype(w_)::value;
    auto kernel = anal_spin0_kernel<NT, R, W>;
    constexpr size_t smem = anal_smem<2 * NT, W>();
    allow_smem(kernel, smem);
    launch_overlapped(kernel, dim3(nblocks), 32 * W, smem, st, gp.count, gp.cth, gp.sth, gp.nph,
                      cp.d_moff, cp.alpha, cp.seed, phase, ncm, pcomp0, job.lmax, job.mmax + 1,
                      Aout, ncA, comp0);
  };
  auto spins = [&](auto nt_, auto r_, auto w_) {
    constexpr int NT = decltype(nt_)::value, R = decltype(r_)::value, W = decltype(w_)::value;
    auto kernel = anal_spin_kernel<NT, R, W>;
    constexpr size_t smem = anal_smem<4 * NT, W>();
    allow_smem(kernel, smem);
    launch_overlapped(kernel, dim3(nblocks), 32 * W, smem, st, gp.count, gp.cth, gp.sth, gp.nph,
                      cp.d_moff, cp.alpha, cp.beta, cp.seed, cp.seed_exp, cp.spin, phase, ncm,
                      pcomp0, job.lmax, job.mmax + 1, Aout, ncA, comp0);
  };
  using std::integral_constant;
  constexpr integral_constant<int, 1> c1{};
  constexpr integral_constant<int, 2> c2{};
  constexpr integral_constant<int, 3> c3{};
  constexpr integral_constant<int, 4> c4{};
  constexpr integral_constant<int, 8> c8{};
  // Shape (R rings per thread, W warps).  More rings per thread share a
  // reduction and more warps a tile; but one warp walks all l of its m alone, so
  // with few ring pairs that chain is the kernel's time and smaller R is faster.
  // Measured with one transform, us, spin 0 / spin 2 (Nside: pairs; lmax = 2 Nside,
  // see anal_eight_warps for other lmax):
  //   Nside 64 (128):    R1 W4 8.8 / 15.0   R2 W4 10.7 / 21.1   R4 W4 15.7 / 33.9
  //   Nside 128 (256):   R1 W4 29.0 / 53.6  R2 W4 19.9 / 38.5   R4 W4 28.5 / 61.7
  //   Nside 256 (512):   R2 W4 79.9 / 177   R2 W8 56.9 / 142    R4 W4 66.3 / 145
  //   Nside 512 (1024):  R2 W8 343 / 801    R3 W4 300 / 769     R4 W4 288 / 778
  //   Nside 1024 (2048): R2 W8 2343 / 5437  R3 W4 1844 / 4719   R4 W4 1701 / 4951
  // The shape fixes the order of the sums over rings, so it does not depend on
  // the number of transforms of the pass: a transform's result is the same bits
  // alone and in any batch.
  auto shape = [&](auto n, auto f) {
    if (gp.npairs <= 128) f(n, c1, c4);
    else if (gp.npairs <= 256) f(n, c2, c4);
    else if (anal_eight_warps(job.spin, gp.npairs, job.lmax)) f(n, c2, c8);
    else if (job.spin == 0) f(n, c4, c4);
    else f(n, c3, c4);
  };
  if (job.spin == 0) {
    if (nt == 1) shape(c1, spin0);
    else if (nt == 2) shape(c2, spin0);
    else shape(c4, spin0);
  } else if (nt == 1) {
    shape(c1, spins);
  } else {
    SHT_REQUIRE(anal_spin_wide(job.spin, gp.npairs, job.lmax), "analysis pass too wide");
    if (gp.npairs <= 128) spins(c2, c1, c4);
    else if (gp.npairs <= 256) spins(c2, c2, c4);
    else spins(c2, c2, c8);
  }
  SHT_CUDA(cudaGetLastError());
}

}  // namespace sht
