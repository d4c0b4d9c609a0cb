// Device-side plan structures and kernel launchers of the transform engine.
//
// Data layout in HBM (one job, FP64 internal arithmetic):
//   * ring pairs are re-ordered by decreasing mlim (sharp_get_mlim), so the
//     pairs that take part at a given m form the prefix [0, count_m[m]);
//   * staged a_lm  A[(moff[m] + l - m) * ncA + comp]   (double2), scaled by the
//     recurrence normalisation c_l (and norm_l for spin > 0); each m segment
//     is followed by kPad zero entries so l-blocks may run past lmax;
//   * phase       P[((p * ncm + comp) * 2 + hemisphere) * (mmax + 1) + m]
//     (double2): ring-major, so the ring FFT reads and writes contiguous rows
//     and the Legendre kernels write one element per (m, pair, comp, ring).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <utility>
#include <vector>

#include "sht_internal.h"

namespace sht {

constexpr int kMaxRadices = 24;

// Factorisation of one complex FFT length.
struct FftDesc {
  int n;        // real ring length
  int N;        // complex FFT length (n/2 for even n, n for odd n)
  int tw;       // offset of exp(-2 pi i j/n), j<n, in the twiddle table
  int nrad;
  int rad[kMaxRadices];
  int blue;     // 1: the size-class kernels run a Bluestein convolution of length M
  int M;       // power-of-two convolution length >= 2N - 1
  long long bhat;   // offset of the transformed chirp in the digit order of the
                    // radix-4 stages (/M), or -1 when no generic-class ring uses it
  long long bhat2;  // the same in the digit order of the radix-16 register passes,
                    // or -1 when no register-Bluestein ring uses it
  long long chirp;  // with bhat2: offset of c_j = exp(-pi i j^2/N), j < N, in natural
                    // order (the register kernels read it coalesced), else -1
};

// Host half of a geometry plan (build_geom_host, no device calls): what the
// cached plans upload and the allocation-free synthesis places in its fixed
// scratch.  Pairs are in internal (decreasing mlim) order; per-ring entries
// are indexed 2*p + hemisphere.
struct GeomHost {
  int npairs = 0, nphmax = 0, nmax_complex = 0;
  int P = 2;                          // largest Bluestein convolution length (>= 2)
  int synth_tile = 256;               // ring pairs per CTA of the FP64 synthesis
  std::vector<int> order, count_m, mlim_sorted;
  std::vector<int2> synth_items, mixed_items;
  std::vector<double> cth, sth, phi0, weight;
  std::vector<int> nph, stride, fft;
  std::vector<long long> ofs;
  std::vector<FftDesc> descs;
  std::vector<int> tw_n, tw_off;      // per distinct length: n and table offset
  std::vector<int> blue_idx;          // descriptors with a radix-4 chirp transform (bhat)
  std::vector<int> blue2_idx;         // descriptors with a register-pass one (bhat2)
  long long tw_total = 0, bhat_total = 0, chirp_total = 0;
  std::vector<int> cls_N, cls_start, cls_count, cls_bufA, cls_bufB, cls_pairs;
  // pairs whose rings run the power-of-two register FFT (pow2_ring_length):
  // complex length pw_N[c], listed at pw_pairs[pw_start[c] .. +pw_count[c])
  std::vector<int> pw_N, pw_start, pw_count, pw_pairs;
  // pairs whose rings run the register Bluestein convolution
  // (blue_ring_length): length pb_M[c], listed at pb_pairs[pb_start[c] ..)
  std::vector<int> pb_M, pb_start, pb_count, pb_pairs;
  // pairs of the short-ring kernels (short_ring_kind), longest first
  std::vector<int> ps_pairs;
  // pairs of odd rings (odd_pair_length): convolution length po_M[c], listed at
  // po_pairs[po_start[c] ..)
  std::vector<int> po_M, po_start, po_count, po_pairs;
  long long map_lo = 0, map_hi = 0;
  bool map_covered = false;
};
// Shared memory of the register ring kernels (pw_entries(N) buffer entries
// of the ring kernels, the phi0 rotation slices and the twiddle slices of
// the power-of-two analysis), in double2 entries.
inline size_t pow2_ring_smem_entries(int N, int mmax) {
  const int n = N - 1;
  return size_t(n + (n >> 4) + (n >> 8) + 1) + 64 + mmax / 64 + 2 + 64 + N / 64 + 1;
}
constexpr size_t kRingSmemLimit = 227 * 1024;
// Complex FFT length N of a ring that the power-of-two ring kernels take
// (n = 2N pixels with N in {1024, 2048, 4096, 8192}, unit stride, no alias
// folding: mm <= N), else 0.
inline int pow2_ring_length(int nph, int stride, int mm) {
  if (nph <= 0 || (nph & 1) || stride != 1) return 0;
  const int N = nph / 2;
  if (N != 1024 && N != 2048 && N != 4096 && N != 8192) return 0;
  return mm <= N ? N : 0;
}
// Convolution length M of a ring that the register Bluestein kernels take,
// else 0: even nph with M in {1024, 2048, 4096, 8192} (any stride, any alias
// folding) whose complex length either calls for a Bluestein convolution by
// the cost model of the size classes or exceeds 1024 (there the size-class
// kernel, one 1024-thread CTA per SM, ran the mixed-radix Stockham passes
// about twice as slowly per ring as the register convolution); with all set
// (every plan but that of the allocation-free synthesis) every ring that has
// such an M, but see smooth_ring_length.
constexpr int kRegBluesteinMinN = 1024;
inline int blue_ring_length(int nph, const FftDesc &d, bool all) {
  if (nph <= 0 || (nph & 1)) return 0;
  if (!all && !d.blue && d.N <= kRegBluesteinMinN) return 0;
  return (d.M == 1024 || d.M == 2048 || d.M == 4096 || d.M == 8192) ? d.M : 0;
}
// Whether an even ring has a complex length N in (512, 1024] without factors
// above 5, whose direct passes in the size classes take less than the
// convolution of length 2048.  Ring FFTs of a Gauss grid of nph pixels per ring,
// 6 components, us, direct and convolution (synthesis / analysis):
//   nph 1000: 58 / 56  50 / 42    1080: 66 / 65  93 / 85    1200: 73 / 72  105 / 95
//       1536: 95 / 93  139 / 123  1800: 134 / 131  179 / 149
//       2000: 144 / 140  203 / 166
// With a factor 7 the convolution takes less (1120: 90 / 88, 97 / 88; 1400: 150
// / 147, 125 / 111) and with larger ones half or a quarter.  In a geometry with
// other rings of that convolution they share its launch, which takes less than one
// of their own (HEALPix, 3 components: Nside 512 145 / 122 us, 165 / 143 with the
// smooth rings in the size classes; Nside 300, whose equatorial rings are smooth,
// 104 / 93 and 113 / 100).
inline bool smooth_ring_length(int nph) {
  if (nph <= 0 || (nph & 1)) return false;
  int N = nph / 2;
  if (N <= 512 || N > 1024) return false;
  for (int p : {2, 3, 5})
    while (N % p == 0) N /= p;
  return N == 1;
}
// How the short-ring kernels run an even ring of complex length N, or kNone:
// directly (N <= 32), by the passes of length L = N (64 .. 512, a power of two),
// or by a Bluestein convolution of length L (N up to 256).
enum class ShortKind { kNone, kDirect, kPasses };
__host__ __device__ inline ShortKind short_ring_kind(int N, int *L, bool *blue) {
  *L = N;
  *blue = (N & (N - 1)) != 0;
  if (N <= 32) return ShortKind::kDirect;
  if (!*blue) return N <= 512 ? ShortKind::kPasses : ShortKind::kNone;
  if (N > 256) return ShortKind::kNone;
  *L = N <= 64 ? 128 : N <= 128 ? 256 : 512;
  return ShortKind::kPasses;
}
// Convolution length M = 256 .. 8192 of the odd-ring kernels for a pair whose
// rings have n0 and n1 pixels (<= 0: absent), else 0: one odd length of at least
// 3.  (Rings of one pixel stay in the size classes, which reproduce the
// reference's fold.)
inline int odd_pair_length(int n0, int n1) {
  const int n = n0 > 0 ? n0 : n1;
  if (n < 3 || !(n & 1) || n > 4096 || (n0 > 0 && n1 > 0 && n0 != n1)) return 0;
  int M = 256;
  while (M < 2 * n - 1) M <<= 1;
  return M;
}
inline size_t odd_ring_smem_entries(int M, int mmax) {
  const int n = M - 1;
  return size_t(n + (n >> 4) + (n >> 8) + 1) + 2 * size_t(64 + mmax / 64 + 1);
}
// registers: every ring that fits goes to the register kernels; false (the
// allocation-free synthesis, whose tables share a fixed scratch) keeps those
// that the size classes can take there.
GeomHost build_geom_host(const sharp_geom_info *g, int lmax, int mmax, int spin,
                         bool registers = true);

// Per-geometry device tables (pairs in internal mlim order).
struct GeomPlan {
  const void *key = nullptr;
  uint64_t hash = 0;
  int lmax = -1, mmax = -1, spin = -1;
  int npairs = 0, nphmax = 0, nmax_complex = 0;
  std::vector<int> count_m;          // host copy, mmax+1 entries
  std::vector<int> order;            // internal index -> reference pair index
  std::vector<int2> synth_items;     // (m, tile) work list for synthesis
  int synth_tile = 0;
  std::vector<int2> mixed_items;     // (m, tile of 256 pairs) for the tensor-core path
  // device arrays
  double *cth = nullptr, *sth = nullptr;
  int *mlim = nullptr, *count = nullptr;
  int2 *items = nullptr;
  int2 *mitems = nullptr;
  // per ring (index 2*p + h)
  double *phi0 = nullptr, *weight = nullptr;
  long long *ofs = nullptr;
  int *nph = nullptr, *stride = nullptr, *fft = nullptr;
  FftDesc *fdesc = nullptr;
  double2 *twiddle = nullptr;
  double2 *bhat = nullptr;           // Bluestein chirp transforms
  double2 *chirp = nullptr;          // chirps of the register Bluestein lengths
  double2 *wpow2 = nullptr;          // exp(-2 pi i j/P), j<P, P = largest M
  int P = 2;
  // ring FFT size classes: pairs whose largest complex FFT length is
  // <= cls_N[c], listed at cls_pairs[cls_start[c] .. +cls_count[c])
  std::vector<int> cls_N, cls_start, cls_count, cls_bufA, cls_bufB;
  int *cls_pairs = nullptr;
  // power-of-two register-FFT classes (see GeomHost)
  std::vector<int> pw_N, pw_start, pw_count;
  int *pw_pairs = nullptr;
  // register-Bluestein classes (see GeomHost)
  std::vector<int> pb_M, pb_start, pb_count;
  int *pb_pairs = nullptr;
  // pairs of the short-ring kernels (see GeomHost)
  int *ps_pairs = nullptr;
  int ps_count = 0;
  // odd-ring classes (see GeomHost)
  std::vector<int> po_M, po_start, po_count;
  int *po_pairs = nullptr;
  // e^{i m phi0} per ring as two slices (see shift_table_kernel), or null
  double2 *shift = nullptr;
  int shift_width = 0;
  // kChainFlags flags of the ring kernels' chains (ChainLink), or null; the epoch
  // of the last chain (changed under the lock of the plans)
  unsigned long long *chain = nullptr;
  mutable unsigned long long chain_epoch = 0;
  long long map_lo = 0, map_hi = 0;  // pixel index extent [lo, hi)
  bool map_covered = false;          // rings tile [lo,hi) exactly
  GeomPlan() = default;
  GeomPlan(const GeomPlan &) = delete;   // owns device memory
  GeomPlan &operator=(const GeomPlan &) = delete;
  ~GeomPlan();
};

// Recurrence coefficient tables for (lmax, mmax, spin).
struct CoefPlan {
  int lmax = -1, mmax = -1, spin = -1;
  long long total = 0;               // table length incl. padding
  std::vector<long long> moff;       // host copy
  long long *d_moff = nullptr;
  double *alpha = nullptr;           // spin 0: alpha; spin>0: a
  double *beta = nullptr;            // spin>0: b = a * fx1
  double *cfac = nullptr;            // c_l
  double *seed = nullptr;            // spin 0: mfac[m]; spin>0: prefac mantissa
  int *seed_exp = nullptr;           // spin>0: prefac exponent (base 2)
  double *norm = nullptr;            // spin>0: norm_l, then (spin 1) that of the derivatives
  double2 *mx_coef = nullptr;        // mixed analysis: (alpha_l, c_l 2^30 / b_l), lazily built
  CoefPlan() = default;
  CoefPlan(const CoefPlan &) = delete;
  CoefPlan &operator=(const CoefPlan &) = delete;
  ~CoefPlan();
};

// a_lm addressing for one alm_info.
struct AlmPlan {
  const void *key = nullptr;
  uint64_t hash = 0;
  int lmax = 0, mmax = 0;
  bool packed = false;
  long long stride = 0;
  long long lo = 0, hi = 0;          // extent in complex (or real if packed) units
  bool covered = false;              // every element in [lo,hi) is an a_lm
  long long *mvstart = nullptr;      // indexed by m
  AlmPlan() = default;
  AlmPlan(const AlmPlan &) = delete;
  AlmPlan &operator=(const AlmPlan &) = delete;
  ~AlmPlan();
};

struct JobDesc {
  int type;        // SHARP_ALM2MAP, SHARP_MAP2ALM, SHARP_ALM2MAP_DERIV1
  int spin;
  int nmaps, nalm;
  int ntrans;
  int flags;
  int lmax, mmax;
  bool dp;
};

// Mixed-precision tensor-core synthesis (sht_mixed.cu)
bool mixed_synth_supported(const JobDesc &job);
void launch_mixed_synth(const JobDesc &job, const GeomPlan &gp, const CoefPlan &cp,
                        const double2 *A, int ncA, double2 *phase, int ncm, int *d_err,
                        cudaStream_t st);
bool mixed_anal_supported(const JobDesc &job);
void launch_mixed_anal(const JobDesc &job, const GeomPlan &gp, CoefPlan &cp,
                       const double2 *phase, int ncm, double2 *Aout, int ncA, int *d_err,
                       cudaStream_t st);

// The device arrays of a job, passed to the kernels by value: no table to
// upload, and a captured launch keeps its arrays.
struct PtrList {
  void *p[2 * kMaxTrans];
};

// Lets a kernel take `bytes` of dynamic shared memory (static and dynamic
// together, 48 KB need no leave).
template <class K>
inline void allow_smem(K kernel, size_t bytes);

// Launch with programmatic stream serialisation: the kernel may become resident
// while its predecessor in the stream runs out (once all its CTAs have called
// grid_release or ended), which hides the launch latency, 1 to 2 us a kernel
// (Nside 64: a synthesis of three kernels takes 19.6 us, 23.8 without; an
// analysis 20.5 and 26.6).  Every kernel launched like this calls grid_wait
// first of all (or is one of a chain, see GridChain): only past it are the writes
// of earlier kernels sure to be visible, and a kernel that ended before its
// predecessor would release its own successors too soon.  What an earlier kernel
// wrote comes through plain pointers: a const __restrict__ one tells the compiler
// that the data stays as it is while the kernel runs, which begins before the
// wait, so that it might be loaded early or through the read-only path.
template <class... P, class... A>
inline void launch_overlapped(void (*kernel)(P...), dim3 grid, int threads, size_t smem,
                              cudaStream_t st, A &&...args);
#ifdef __CUDACC__
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() {
  asm volatile("griddepcontrol.launch_dependents;");
}
constexpr unsigned kSmCount = 148;   // of a B200
// Only a grid of at most two CTAs per SM: the CTAs of the next kernel take
// whatever room there is, and beside a larger grid they end up unevenly spread
// (Gauss grid of 251 pairs, three spin-1 transforms both ways: 559 us with an
// early release of every grid, 477 with this, 495 without overlap).
__device__ __forceinline__ void grid_release_small() {
  if (gridDim.x * gridDim.y <= 2 * kSmCount) grid_release();
}
#endif

// The register ring kernels of one direction read the same phase rows or maps and
// write disjoint ones, so each may run while its predecessor's last CTAs do.  What
// it reads was written before the first of them, which waits (grid_wait) and then
// publishes the call's epoch in a flag of the plan by a release; a later one
// acquires that epoch before it reads or writes anything, or, should the flag
// not hold it yet, waits like every other kernel.  It ends only after its
// predecessor has (grid_wait), so that what follows the last one finds all of
// them done.  The first and the later ones let their successor start as soon as
// all their CTAs have started, the last one as grid_release_small does.  Without a
// flag (a single kernel, a captured stream, whose replays would find the epoch
// of the one before, and the allocation-free synthesis) every kernel waits first.
// T synthesis, Nside 450 / lmax 450: 102 us, 125 if every kernel waits; chi-square
// gradient at Nside 512: 2420 and 2480 us; three Jacobi sweeps at Nside 1024: 11.68
// and 12.06 ms.
struct ChainLink {
  unsigned long long *flag = nullptr;
  unsigned long long epoch = 0;
  bool first = true, last = true;
};
constexpr int kChainFlags = 64;   // calls of a plan in flight that have a flag of their own
#ifdef __CUDACC__
class GridChain {
 public:
  __device__ __forceinline__ explicit GridChain(const ChainLink &l) {
    if (l.flag == nullptr || l.first) {
      grid_wait();
      if (l.flag != nullptr && (threadIdx.x | blockIdx.x | blockIdx.y) == 0)
        asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(l.flag), "l"(l.epoch) : "memory");
    } else {
      // the barrier hands the acquire of thread 0 on to the others
      waited_ = __syncthreads_or(threadIdx.x == 0 && !published(l));
      if (waited_) grid_wait();
      // for the bulk copies of phase rows, which thread 0 issues
      if (threadIdx.x == 0) asm volatile("fence.proxy.async.global;" ::: "memory");
    }
    if (l.flag == nullptr || l.last) grid_release_small();
    else grid_release();
  }
  __device__ __forceinline__ ~GridChain() {
    if (!waited_) grid_wait();
  }

 private:
  // a few tries: usually the epoch is there before the kernel starts
  static __device__ __forceinline__ bool published(const ChainLink &l) {
    for (int i = 0; i < 32; ++i) {
      unsigned long long v;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(l.flag) : "memory");
      if (v == l.epoch) return true;
    }
    return false;
  }
  bool waited_ = true;
};
#endif

// Kernel launchers (sht_legendre.cu)
// Whether the analysis runs CTAs of eight warps with two ring pairs per thread
// (tiles of 512 pairs), 257 .. 512 pairs: one tile, whose sums over rings end early
// for few l.  For many l the sums cost more than the shorter chain gives and four
// warps with more rings per thread take less, at spin s as long as one tile of
// theirs (384 pairs) holds all.  Whole analyses, us, eight warps and four (R4 at
// spin 0, R3 at spin 2), pairs / lmax = mmax:
//   spin 0  257/700: 83, 96   384/500: 62, 71   512/500: 67, 78   512/700: 107, 107
//           320/1000: 158, 139  512/1000: 189, 164  512/2000: 673, 529
//   spin 2  512/500: 146, 201  384/700: 217, 181  512/2000: 1603, 1629
//           257/1000: 340, 290  384/1000: 401, 318  384/2000: 1451, 1117
// (mmax 300, spin 0: 257/1000 112, 128  290/1000 123, 117  512/2000 312, 256.)
inline bool anal_eight_warps(int spin, int npairs, int lmax) {
  if (npairs <= 256 || npairs > 512) return false;
  return lmax <= 750 || (spin == 0 ? npairs <= 288 : npairs > 384);
}
// Whether the spin analysis takes two transforms per pass (three rings per thread
// leave no registers for a second one).
inline bool anal_spin_wide(int spin, int npairs, int lmax) {
  return npairs <= 256 || anal_eight_warps(spin, npairs, lmax);
}
void launch_coef_tables(CoefPlan &cp, cudaStream_t st);
void launch_legendre_synth(const JobDesc &job, const GeomPlan &gp, const CoefPlan &cp,
                           const double2 *A, int ncA, int comp0, int nt,
                           double2 *phase, int ncm, int pcomp0, cudaStream_t st);
void launch_legendre_anal(const JobDesc &job, const GeomPlan &gp, const CoefPlan &cp,
                          const double2 *phase, int ncm, int pcomp0, int nt,
                          double *Aout, int ncA, int comp0, cudaStream_t st);

// Ring FFT and staging launchers (sht_ring.cu)
void launch_twiddles(GeomPlan &gp, int ntw, const std::vector<int> &tw_n,
                     const std::vector<int> &tw_off, cudaStream_t st);
void launch_shift_table(GeomPlan &gp, cudaStream_t st);
void launch_bluestein_setup(GeomPlan &gp, const GeomHost &h, cudaStream_t st);
void launch_twiddles_preplaced(double2 *tw, const int *d_n, const int *d_off, int ntab,
                               cudaStream_t st);
void launch_bluestein_setup_preplaced(const GeomPlan &gp, const int *d_blue_idx, int nblue,
                                      const int *d_blue2_idx, int nblue2, cudaStream_t st);
// map_lo / alm_lo: index (in elements of the user array) that the device
// pointers in maps_dev / alm_dev point at (0 when they are the user's own
// device arrays, the extent start when they are staged copies).
// Ring FFT shared memory.  Entries of the high twiddle slice for ring lengths
// up to 2 nmax_complex, and the double2 entries of one CTA: buffers A and B,
// the phi0 shift slices (64 + mmax/64 + 2), the twiddle slices of the ring
// length and of the Bluestein convolution length P (64 + P/64 + 2).
inline int ring_twiddle_hi_entries(int nmax_complex) { return (2 * nmax_complex) / 64 + 2; }
inline size_t ring_fft_smem_entries(int bufA, int bufB, int mmax, int nmax_complex, int P) {
  return size_t(bufA) + bufB + (64 + mmax / 64 + 2) + (64 + ring_twiddle_hi_entries(nmax_complex)) +
         (64 + P / 64 + 2);
}

void launch_phase2ring(const JobDesc &job, const GeomPlan &gp, long long map_lo,
                       const double2 *phase, int ncm, const PtrList &maps_dev, int nmapptr,
                       cudaStream_t st);
void launch_ring2phase(const JobDesc &job, const GeomPlan &gp, long long map_lo,
                       const PtrList &maps_dev, int nmapptr, double2 *phase, int ncm,
                       cudaStream_t st);
void launch_phase2ring_direct(const JobDesc &job, const GeomPlan &gp, long long map_lo,
                              const double2 *phase, int ncm, const PtrList &maps_dev, int nmapptr,
                              cudaStream_t st);
void launch_ring2phase_direct(const JobDesc &job, const GeomPlan &gp, long long map_lo,
                              const PtrList &maps_dev, int nmapptr, double2 *phase,
                              int ncm, cudaStream_t st);
// pm: pairs of components (G, C) are stored as (G - iC, G + iC), the basis of
// the FP64 spin synthesis.
void launch_stage_alm(const JobDesc &job, const AlmPlan &ap, long long alm_lo,
                      const CoefPlan &cp, const double *norm_l, const PtrList &alm_dev,
                      int nalmptr, double2 *A, int ncA, bool pm, cudaStream_t st);
void launch_scatter_alm(const JobDesc &job, const AlmPlan &ap, long long alm_lo,
                        const CoefPlan &cp, const double *norm_l, const double *Aout, int ncA,
                        const PtrList &alm_dev, int nalmptr, cudaStream_t st);

// Launch accounting: every launcher wraps its kernel in a ProfScope, which
// counts the launch and, when profiling is on, records CUDA events on the
// launching stream around it.
class ProfScope {
 public:
  ProfScope(const char *family, cudaStream_t st);
  ~ProfScope();
  ProfScope(const ProfScope &) = delete;
  ProfScope &operator=(const ProfScope &) = delete;

 private:
  const char *family_;
  cudaStream_t st_;
  cudaEvent_t start_ = nullptr;
};

void check_cuda(cudaError_t e, const char *what, const char *file, int line);
#define SHT_CUDA(call) ::sht::check_cuda((call), #call, __FILE__, __LINE__)

template <class... P, class... A>
inline void launch_overlapped(void (*kernel)(P...), dim3 grid, int threads, size_t smem,
                              cudaStream_t st, A &&...args) {
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  SHT_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
}

template <class K>
inline void allow_smem(K kernel, size_t bytes) {
  if (bytes > 32 * 1024)
    SHT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
}

// Stream-ordered workspace allocation from the library's own memory pool on
// the current device (free with cudaFreeAsync, never cudaFree, which leaves
// the pool's accounting wrong).  The pool keeps freed memory mapped across
// synchronizes (release threshold unlimited), so a transform after a
// synchronize does not map gigabytes of workspace again, and being the
// library's own it leaves the settings of the process's default pool alone.
// Plan-lifetime tables use cudaMalloc.  ws_trim() hands the unused memory
// back (sharp_b200_release_cache); ws_bytes() reports the pool's size.
cudaError_t ws_alloc_bytes(void **p, size_t bytes, cudaStream_t st);
template <typename T>
inline cudaError_t ws_alloc(T **p, size_t bytes, cudaStream_t st) {
  return ws_alloc_bytes(reinterpret_cast<void **>(p), bytes, st);
}
void ws_trim();
bool ws_bytes(unsigned long long *reserved, unsigned long long *used);

}  // namespace sht
