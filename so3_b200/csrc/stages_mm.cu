// DFT stages of the transforms on the FP64 tensor cores (dft_mm.cuh): the
// same stages as stages.cu, any length the planner covers.
//
// Measured against the scalar engines of stages.cu (us, one transform):
//   gamma    L=512 N=64 (127)    769 -> 697 inverse, 800 -> 721 forward
//            L=512 N=16 (31)    1125 -> 113, 1182 -> 107
//            L=256 N=32 real     156 -> 44,   179 -> 44
//   alpha    L=128 N=16 (255)     43 -> 23;  L=256 N=16 (511) 339 -> 78
//            L=300 N=16 (599)    737 -> 190; L=1024 N=8 (2047) 3774 -> 525
//   inv beta L=256 N=16 320 -> 103; L=300 N=16 791 -> 227; L=1024 N=8 3635 -> 758
// What bounds them now: gamma at N = 64 the tensor pipe (0.47 ms of products),
// at small N the memory system; alpha and beta instruction issue and latency
// (ncu at 1023: 43 % of issue slots, 40 % of the FP64 pipe, 21 warps per SM).
#include <algorithm>

#include "dft_mm.cuh"
#include "launch.cuh"
#include "so3gpu_internal.h"

namespace so3g {

namespace {

constexpr int kGT = 128;               // threads of the gamma kernels
constexpr size_t kSmemMax = 200 * 1024;
constexpr int kMaxThr = 256, kMinB = 3;  // alpha / beta kernels: 80 registers a thread, 24 warps per SM
constexpr int kMaxT = 16;              // sequences per CTA

// Signals of a batch (blockIdx.z of the gamma kernels): their samples, and
// their scratch at W + z * wstride.
struct SigIo {
  long long wstride;
  void* f[kMaxBatch];
};
SigIo sig_io(const Batch& bt, const void* f) {
  SigIo io{};
  io.wstride = bt.wstride;
  for (int b = 0; b < bt.n; b++) io.f[b] = bt.io[b];
  if (!bt.n) io.f[0] = const_cast<void*>(f);
  return io;
}
int count(const Batch& bt) { return bt.n ? bt.n : 1; }

// Rows of all signals, plane-major over the nb beta rows of each.
__device__ __forceinline__ long long row_off(const Geometry& g, int row, long long wstride) {
  const int per = g.nplanes * g.nb, sig = row / per;
  row -= sig * per;
  return sig * wstride + (long long)(row / g.nb) * g.PS + (long long)(row % g.nb) * g.RS;
}

// ------------------------------------------------------------------ gamma
// One matrix level over the planes: a CTA holds TA consecutive alpha samples
// of one beta row of every plane, row pitch TA + 2 slots (2 mod 8).
//
struct InvGammaOut {
  double2* dst;
  long long plane_sz;
  int nf;
  __device__ __forceinline__ double2* col(int j) const { return dst + j; }
  __device__ __forceinline__ void put(double2* d, int q, double2 v) const {
    if (q < nf) d[q * plane_sz] = v;
  }
};
struct FwdGammaOut {
  double2* dst;
  long long PS;
  double scale;
  int N, ng, plane0, steer;
  __device__ __forceinline__ double2* col(int j) const { return dst + j; }
  __device__ __forceinline__ void put(double2* d, int k, double2 v) const {
    const int n = k < N ? k : k - ng;
    if (n + plane0 < 0) return;  // k = N of the 2N-point circle: no plane
    const bool keep = !steer || ((n - (N - 1)) & 1) == 0;
    d[(n + plane0) * PS] = keep ? cscale(v, scale) : make_double2(0.0, 0.0);
  }
};

// Complex inverse: circle entry r holds plane n = r (r < N) or r - ng; the
// 2N-point circle of a steerable signal has no plane n = N and keeps N samples.
__global__ void __launch_bounds__(kGT, 6) inv_gamma_mm_kernel(Geometry g, MmLevel lv, const double2* __restrict__ W,
                                                         const __grid_constant__ SigIo io, int tash, int row0) {
  extern __shared__ __align__(16) double2 sm[];
  dep_wait();
  W += blockIdx.z * io.wstride;
  double2* f = static_cast<double2*>(io.f[blockIdx.z]);
  const int TA = 1 << tash, rp = TA + 2;
  const int row = row0 + blockIdx.y, a0 = blockIdx.x << tash, ng = g.ng, nc = min(TA, g.na - a0);
  const double2* src = W + (long long)row * g.RS + a0;
  for (int i = threadIdx.x; i < g.nplanes << tash; i += kGT) {
    const int p = i >> tash, c = i & (TA - 1);
    int r = p - g.plane0;
    if (r < 0) r += ng;
    if (c < nc) mm::cp16(sm + r * rp + c, src + (long long)p * g.PS + c);
  }
  if (g.steer)
    for (int c = threadIdx.x; c < TA; c += kGT) sm[g.N * rp + c] = make_double2(0.0, 0.0);
  mm::cp_wait_all();
  __syncthreads();
  dep_launch();
  const long long plane_sz = (long long)g.nb * g.na;
  double2* dst = f + (long long)row * g.na + a0;
  mm::level<true>(sm, rp, lv, nc, [](int j) { return j; }, InvGammaOut{dst, plane_sz, g.nf});
}

// Complex forward; steerable: samples N..2N-1 of the circle are zero and only
// n = N-1 (mod 2) is analysed (so3_core.c:309-328).
__global__ void __launch_bounds__(kGT, 6) fwd_gamma_mm_kernel(Geometry g, MmLevel lv, const __grid_constant__ SigIo io,
                                                         double2* __restrict__ W, int tash, int row0) {
  extern __shared__ __align__(16) double2 sm[];
  dep_wait();
  W += blockIdx.z * io.wstride;
  const double2* f = static_cast<const double2*>(io.f[blockIdx.z]);
  const int TA = 1 << tash, rp = TA + 2;
  const int row = row0 + blockIdx.y, a0 = blockIdx.x << tash, ng = g.ng, nc = min(TA, g.na - a0);
  const long long plane_sz = (long long)g.nb * g.na;
  const double2* src = f + (long long)row * g.na + a0;
  for (int i = threadIdx.x; i < ng << tash; i += kGT) {
    const int r = i >> tash, c = i & (TA - 1);
    if (r >= g.nf)
      sm[r * rp + c] = make_double2(0.0, 0.0);
    else if (c < nc)
      mm::cp16(sm + r * rp + c, src + (long long)r * plane_sz + c);
  }
  mm::cp_wait_all();
  __syncthreads();
  dep_launch();
  const double scale = 2.0 * 3.141592653589793238462643383279502884 / g.nf;
  double2* dst = W + (long long)row * g.RS + a0;
  mm::level<false>(sm, rp, lv, nc, [](int j) { return j; },
            FwdGammaOut{dst, g.PS, scale, g.N, ng, g.plane0, g.steer});
}

// Real inverse (c2r): y(q) = Re x_0 + sum_r 2 Re x_r cos - 2 Im x_r sin over
// the planes n = r >= 0; 8 real columns (alpha) per tile, so lane (g, c) of an
// accumulator holds output q = g of columns 2c, 2c + 1.
template <int MT>
__device__ __forceinline__ void c2r_task(const double2* __restrict__ src, int rp, const MmLevel& lv, int qt0, int j0,
                                         int nc, double* __restrict__ dst, long long plane_sz) {
  constexpr int NT = 2;
  const int lane = threadIdx.x & 31, kk = lane & 3, gr = lane >> 2, H = lv.H;
  double a[MT][NT][2], b[MT][NT][2];
  const double2* bp[NT];
#pragma unroll
  for (int t = 0; t < NT; t++) {
    bp[t] = src + min(j0 + 8 * t + gr, nc - 1);
    const int c0 = j0 + 8 * t + 2 * kk;
#pragma unroll
    for (int i = 0; i < MT; i++) {
      a[i][t][0] = src[min(c0, nc - 1)].x;
      a[i][t][1] = src[min(c0 + 1, nc - 1)].x;
      b[i][t][0] = b[i][t][1] = 0.0;
    }
  }
  const double2* tab = lv.tab + (size_t)qt0 * lv.KS * 32 + lane;
#pragma unroll 2
  for (int ks = 0; ks < lv.KS; ks++) {
    const int r = min(4 * ks + kk + 1, H);
    double2 x[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) x[t] = cscale(bp[t][r * rp], 2.0);
#pragma unroll
    for (int i = 0; i < MT; i++) {
      const double2 w = __ldg(tab + (i * lv.KS + ks) * 32);
#pragma unroll
      for (int t = 0; t < NT; t++) {
        mm::dmma(a[i][t], w.x, x[t].x);
        mm::dmma(b[i][t], w.y, x[t].y);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < MT; i++) {
    const int q = 8 * (qt0 + i) + gr;
    if (q > H) continue;
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int j = j0 + 8 * t + 2 * kk + e;
        if (j >= nc) continue;
        dst[(long long)q * plane_sz + j] = a[i][t][e] - b[i][t][e];
        if (q) dst[(long long)(lv.p - q) * plane_sz + j] = a[i][t][e] + b[i][t][e];
      }
  }
}

__global__ void __launch_bounds__(kGT, 6) inv_gamma_real_mm_kernel(Geometry g, MmLevel lv,
                                                              const double2* __restrict__ W, const __grid_constant__ SigIo io,
                                                              int tash, int row0) {
  extern __shared__ __align__(16) double2 sm[];
  dep_wait();
  W += blockIdx.z * io.wstride;
  double* f = static_cast<double*>(io.f[blockIdx.z]);
  const int TA = 1 << tash, rp = TA + 2;
  const int row = row0 + blockIdx.y, a0 = blockIdx.x << tash, nc = min(TA, g.na - a0);
  const double2* src = W + (long long)row * g.RS + a0;
  for (int i = threadIdx.x; i < g.nplanes << tash; i += kGT) {
    const int p = i >> tash, c = i & (TA - 1);
    if (c < nc) mm::cp16(sm + p * rp + c, src + (long long)p * g.PS + c);
  }
  mm::cp_wait_all();
  __syncthreads();
  dep_launch();
  const long long plane_sz = (long long)g.nb * g.na;
  double* dst = f + (long long)row * g.na + a0;
  const int ng = (lv.QT + 1) / 2, tasks = (nc + 15) / 16 * ng;
  for (int w = threadIdx.x >> 5; w < tasks; w += kGT / 32) {
    const int qt0 = (w % ng) * 2, j0 = (w / ng) * 16;
    if (lv.QT - qt0 == 1)
      c2r_task<1>(sm, rp, lv, qt0, j0, nc, dst, plane_sz);
    else
      c2r_task<2>(sm, rp, lv, qt0, j0, nc, dst, plane_sz);
  }
}

// Real forward (r2c): planes n = q = 0 .. N-1 of the samples, (a_q, -b_q).
template <int MT>
__device__ __forceinline__ void r2c_task(const double* __restrict__ src, int rp, const MmLevel& lv, int qt0, int j0,
                                         int nc, double2* __restrict__ dst, long long PS, double scale) {
  constexpr int NT = 2;
  const int lane = threadIdx.x & 31, kk = lane & 3, gr = lane >> 2, H = lv.H;
  double a[MT][NT][2], b[MT][NT][2];
  const double* bp[NT];
#pragma unroll
  for (int t = 0; t < NT; t++) {
    bp[t] = src + min(j0 + 8 * t + gr, nc - 1);
    const int c0 = j0 + 8 * t + 2 * kk;
#pragma unroll
    for (int i = 0; i < MT; i++) {
      a[i][t][0] = src[min(c0, nc - 1)];
      a[i][t][1] = src[min(c0 + 1, nc - 1)];
      b[i][t][0] = b[i][t][1] = 0.0;
    }
  }
  const double2* tab = lv.tab + (size_t)qt0 * lv.KS * 32 + lane;
#pragma unroll 2
  for (int ks = 0; ks < lv.KS; ks++) {
    const int r = min(4 * ks + kk + 1, H);
    double s[NT], d[NT];
#pragma unroll
    for (int t = 0; t < NT; t++) {
      const double xp = bp[t][r * rp], xn = bp[t][(lv.p - r) * rp];
      s[t] = xp + xn;
      d[t] = xp - xn;
    }
#pragma unroll
    for (int i = 0; i < MT; i++) {
      const double2 w = __ldg(tab + (i * lv.KS + ks) * 32);
#pragma unroll
      for (int t = 0; t < NT; t++) {
        mm::dmma(a[i][t], w.x, s[t]);
        mm::dmma(b[i][t], w.y, d[t]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < MT; i++) {
    const int q = 8 * (qt0 + i) + gr;
    if (q > H) continue;
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int j = j0 + 8 * t + 2 * kk + e;
        if (j < nc) dst[(long long)q * PS + j] = make_double2(a[i][t][e] * scale, -b[i][t][e] * scale);
      }
  }
}

// Sample rows of TA + 4 doubles (4 mod 16): 4 rows x 4 columns per half warp
// in distinct banks.
__global__ void __launch_bounds__(kGT, 6) fwd_gamma_real_mm_kernel(Geometry g, MmLevel lv,
                                                              const __grid_constant__ SigIo io, double2* __restrict__ W,
                                                              int tash, int row0) {
  extern __shared__ __align__(16) double smd[];
  dep_wait();
  W += blockIdx.z * io.wstride;
  const double* f = static_cast<const double*>(io.f[blockIdx.z]);
  const int TA = 1 << tash, rp = TA + 4;
  const int row = row0 + blockIdx.y, a0 = blockIdx.x << tash, nc = min(TA, g.na - a0);
  const long long plane_sz = (long long)g.nb * g.na;
  const double* src = f + (long long)row * g.na + a0;
  for (int i = threadIdx.x; i < g.ng << tash; i += kGT) {
    const int r = i >> tash, c = i & (TA - 1);
    if (c < nc) mm::cp8(smd + r * rp + c, src + (long long)r * plane_sz + c);
  }
  mm::cp_wait_all();
  __syncthreads();
  dep_launch();
  const double scale = 2.0 * 3.141592653589793238462643383279502884 / g.nf;
  double2* dst = W + (long long)row * g.RS + a0;
  const int ng = (lv.QT + 1) / 2, tasks = (nc + 15) / 16 * ng;
  for (int w = threadIdx.x >> 5; w < tasks; w += kGT / 32) {
    const int qt0 = (w % ng) * 2, j0 = (w / ng) * 16;
    if (lv.QT - qt0 == 1)
      r2c_task<1>(smd, rp, lv, qt0, j0, nc, dst, g.PS, scale);
    else
      r2c_task<2>(smd, rp, lv, qt0, j0, nc, dst, g.PS, scale);
  }
}

// ------------------------------------------------------------------ alpha
// T consecutive rows (plane-major over the beta rows) per CTA, two buffers of
// T sequences.  Inverse: column m + L - 1 of the row is entry m mod P (the
// MWSS Nyquist entry is zero); forward: the other way round, over 1/P.
template <bool INV>
struct AlphaOut {
  double2* const* rows;
  double inv;
  int L, P;
  typedef double2* Seq;
  __device__ __forceinline__ Seq seq(int t) const { return rows[t]; }
  __device__ __forceinline__ void put(Seq d, int k, double2 v) const {
    if (INV) {
      d[k] = v;
    } else {
      const int c = k < L ? k + L - 1 : k - P + L - 1;
      if (c >= 0) d[c] = cscale(v, inv);
    }
  }
};

template <bool INV>
__global__ void __launch_bounds__(kMaxThr, kMinB) alpha_mm_kernel(Geometry g, MmPlan P, double2* __restrict__ W, int T,
                                                              int nrows, long long wstride) {
  extern __shared__ __align__(16) double2 sm[];
  dep_wait();
  __shared__ double2 x0[2 * kMaxT];
  __shared__ double2* rows[kMaxT];
  double2* A = sm;
  double2* Z = sm + (size_t)T * P.ts;
  const int L = g.L, Pn = g.P, r0 = blockIdx.x * T, Ta = min(T, nrows - r0);
  if (threadIdx.x < Ta) rows[threadIdx.x] = W + row_off(g, r0 + threadIdx.x, wstride);
  // column of entry k; -1: the MWSS Nyquist entry k = L, which has no column
  auto col = [&](int k) { return k <= L - 1 ? k + L - 1 : k - Pn + L - 1; };
  for (int t = 0; t < Ta; t++) {
    const double2* src = W + row_off(g, r0 + t, wstride);
    if (P.kind == 3) {
      mm::stage_conv<INV>(P, A + t * P.ts, x0 + 2 * t, [&](int k) {
        const int c = INV ? col(k) : k;
        return c >= 0 ? src[c] : make_double2(0.0, 0.0);
      });
    } else {
      for (int k = threadIdx.x; k < Pn; k += blockDim.x) {
        const int c = INV ? col(k) : k;
        double2* d = A + t * P.ts + mm::pos(P, k);
        if (c >= 0)
          mm::cp16(d, src + c);
        else
          *d = make_double2(0.0, 0.0);
      }
    }
  }
  mm::cp_wait_all();
  __syncthreads();
  dep_launch();
  mm::run<INV>(P, A, Z, Ta, x0, AlphaOut<INV>{rows, 1.0 / Pn, L, Pn});
}

// ------------------------------------------------------------------ inverse beta
// Two columns per DFT as in stages.cu (inv_beta_kernel): T adjacent column
// pairs per CTA; the synthesis of a pair lands in shared memory, where each
// row meets its mirror.
struct SmemOut {
  double2* X;
  int ts;
  typedef double2* Seq;
  __device__ __forceinline__ Seq seq(int t) const { return X + t * ts; }
  __device__ __forceinline__ void put(Seq d, int k, double2 v) const { d[k] = v; }
};

__global__ void __launch_bounds__(kMaxThr, kMinB) inv_beta_mm_kernel(Geometry g, MmPlan P,
                                                                     const double2* __restrict__ half,
                                                                     double2* __restrict__ W, int T, long long wstride) {
  extern __shared__ __align__(16) double2 sm[];
  dep_wait();
  __shared__ double2 x0[2 * kMaxT], b0s[kMaxT];
  double2* A = sm;
  double2* Z = sm + (size_t)T * P.ts;
  const int sig = blockIdx.y / g.nplanes, plane = blockIdx.y - sig * g.nplanes;
  const int n = plane - g.plane0, L = g.L, Pn = g.P, ncols = 2 * L - 1;
  W += sig * wstride;
  const int q0 = blockIdx.x * T, Ta = min(T, L - q0);
  double2* base = W + (long long)plane * g.PS;
  const double2* cbase = W + g.QOFF + (long long)plane * g.QS;
  const bool first_is_a = ((L - 1 + n) & 1) == 0;  // column 2q has m + n even
  // both columns of each pair into Z first (L + L <= ts entries), all copies in flight at once
  for (int t = 0; t < Ta; t++) {
    const int c = 2 * (q0 + t);
    const double2* src = cbase + (long long)c * g.CS;
    double2* z = Z + t * P.ts;
    for (int mp = threadIdx.x; mp < L; mp += blockDim.x) {
      mm::cp16(z + mp, src + mp);
      if (c + 1 < ncols)
        mm::cp16(z + L + mp, src + g.CS + mp);
      else
        z[L + mp] = make_double2(0.0, 0.0);
    }
  }
  mm::cp_wait_all();
  __syncthreads();
  dep_launch();
  // z at +m' and -m'
  auto pair = [&](int t, int mp, double2& zp, double2& zn) {
    const double2 v0 = Z[t * P.ts + mp], v1 = Z[t * P.ts + L + mp];
    const double2 av = first_is_a ? v0 : v1, bv = first_is_a ? v1 : v0;
    zp = cadd(av, bv);
    if (mp == 0) {
      b0s[t] = bv;
      zn = zp;
      return;
    }
    zn = csub(av, bv);
    if (g.mw) {
      const double2 e = __ldg(half + mp);  // e^{-i pi m'/(2L-1)}
      zp = cmul(zp, cconj(e));
      zn = cmul(zn, e);
    }
  };
  for (int t = 0; t < Ta; t++) {
    double2* s = A + t * P.ts;
    if (P.kind == 3) {
      mm::stage_conv<true>(P, s, x0 + 2 * t, [&](int k) {
        double2 zp, zn;
        const int mp = k <= L - 1 ? k : Pn - k;
        if (mp >= L) return make_double2(0.0, 0.0);  // MWSS Nyquist entry
        pair(t, mp, zp, zn);
        return k <= L - 1 ? zp : zn;
      });
    } else {
      for (int mp = threadIdx.x; mp < L; mp += blockDim.x) {
        double2 zp, zn;
        pair(t, mp, zp, zn);
        s[mm::pos(P, mp)] = zp;
        if (mp) s[mm::pos(P, Pn - mp)] = zn;
      }
      if (!g.mw && threadIdx.x == 0) s[mm::pos(P, L)] = make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
  double2* X = P.kind == 1 ? Z : A;
  const int ts = P.ts;
  mm::run<true>(P, A, Z, Ta, x0, SmemOut{X, ts});
  __syncthreads();
  // rows k < nb of both columns
  const int rows = blockDim.x / T, t = threadIdx.x % T;
  if (t >= Ta || threadIdx.x >= rows * T) return;
  for (int row = threadIdx.x / T; row < g.nb; row += rows) {
    const int c = 2 * (q0 + t);
    int mrow = g.mw ? Pn - 1 - row : Pn - row;
    if (mrow >= Pn) mrow -= Pn;
    const double2 y0 = X[t * ts + row], y1 = X[t * ts + mrow], B0 = b0s[t];
    const double2 yA = make_double2(0.5 * (y0.x + y1.x) - B0.x, 0.5 * (y0.y + y1.y) - B0.y);
    const double2 yB = make_double2(0.5 * (y0.x - y1.x) + B0.x, 0.5 * (y0.y - y1.y) + B0.y);
    double2* dst = base + (long long)row * g.RS + c;
    dst[0] = first_is_a ? yA : yB;
    if (c + 1 < ncols) dst[1] = first_is_a ? yB : yA;
  }
}

size_t seq_smem(const MmPlan& P, int T, int bufs) { return bufs * sizeof(double2) * (size_t)T * P.ts; }

// Launch shape of a stage over `nseq` sequences: sequences per CTA, warps, and
// row tiles per warp task of each level (in the returned plan).
//
// About 800 points per CTA at 220 per warp: measured over 1-16 sequences x 2-8
// warps at lengths 31 to 2047, the best shapes hold 150-260 points per warp
// and 600-1000 per CTA (255: 3 x 4 warps, 511: 2 x 5, 1023: 1 x 4, 2047: 1 x
// 8); larger CTAs wait longer at their barriers (1023: 4 sequences on 8 warps
// takes 1.4x the time), smaller ones leave column tiles half empty.  One-level
// plans take 8 columns, a full task.  Fewer sequences where the device would
// not fill; one row tile per task where two would leave warps idle.
struct Shape {
  int T, warps;
  size_t smem;
  MmPlan P;
};
Shape shape_for(const MmPlan& P0, int nseq, int bufs) {
  Shape z{1, 2, 0, P0};
  z.T = P0.kind == 1 ? 8 : std::max(1, std::min(8, (800 + P0.n / 2) / P0.n));
  while (z.T > 1 && (nseq + z.T - 1) / z.T < 148) z.T >>= 1;
  z.warps = std::max(2, std::min(kMaxThr / 32, (z.T * P0.n + 110) / 220));
  if (P0.kind == 1) z.warps = std::max(z.warps, std::min(kMaxThr / 32, (P0.la.QT + 1) / 2));
  for (int l = 0; l < (P0.kind == 1 ? 1 : 2); l++) {
    MmLevel& v = l ? z.P.lb : z.P.la;
    const int cols = P0.kind == 1 ? z.T : z.T * (l ? P0.a : P0.b), nc = (cols + 4 * mm::kNT - 1) / (4 * mm::kNT);
    v.MT = std::min(v.QT, nc * ((v.QT + 1) / 2) < z.warps ? 1 : 2);
    v.QG = (v.QT + v.MT - 1) / v.MT;
  }
  z.smem = seq_smem(P0, z.T, bufs);
  return z;
}

// Gamma kernels: two row tiles per warp task, as level_shape sets them (80 registers,
// 24 warps per SM; four tiles at 128 registers and 16 warps: 766 against 697 us at
// L = 512, N = 64, 277 / 241 at N = 32, 255 / 177 at L = 1024, N = 8).
//
// log2 of the alpha samples per CTA: the planes of six CTAs fit in shared memory
// and a CTA has four tasks or more (L = 1024, N = 2: 16 samples 224 us, 256: 78; N = 8:
// 16: 292, 64: 177; L = 512, N = 32: 16: 241, 32: 253), fewer where the device would not fill.
int gamma_shift(int ng, int na, int rows) {
  int sh = ng <= 7 ? 8 : ng <= 11 ? 7 : ng <= 23 ? 6 : ng <= 47 ? 5 : 4;
  while (sh > 4 && ((na + (1 << sh) - 1) >> sh) * rows < 296) sh--;
  return sh;
}

}  // namespace

// One matrix level costs ng / 4 pairs of products per sample, the scalar engines a
// few passes, so long circles go back to them; how long depends on their radices.
// us a stage, matrix / scalar, inverse at L = 128:
//   complex, radices to 8   135: 76 / 82, 175: 114 / 95, 243: 225 / 181, 399 (L = 64) 239 / 82
//            larger ones    171: 114 / 162, 207: 171 / 179, 231: 214 / 189, 279: 370 / 238
//            Bluestein      265: 279 / 1253, 359: 587 / 1286, 419: 1290 / 1342 (L = 64: 418 / 337;
//                           from 390 on a block's 16 columns leave one block to an SM)
//   real     radices to 8   315: 144 / 158, 343: 173 / 148
//            larger ones    351: 174 / 242, 399: 252 / 236
//            Bluestein      599: 587 / 2565
// Where the device does not fill (L < 49), a warp's chain of products is what takes
// the time: complex, L = 32, 81: 13 / 13, 105: 14 / 13, 175: 23 / 15.  The choice
// depends on the geometry alone, not on the batch: batches equal single calls.
bool mm_gamma_ok(const Geometry& g, const FftPlan& p) {
  if (p.l1.p != g.ng || (size_t)g.ng * 18 * sizeof(double2) > kSmemMax) return false;
  const int blocks = (g.na + 15) / 16 * g.nb;
  if (g.real) return p.blue || g.ng < (p.big() ? 390 : 340);
  if (p.blue) return g.ng < 390;
  return g.ng < (blocks < 2 * 148 ? 100 : p.big() ? 220 : 172);
}
bool mm_ok(const FftPlan& p) { return p.mm.n == p.n && seq_smem(p.mm, 1, 2) <= kSmemMax; }

int launch_mm_inv_gamma(const Geometry& g, const FftPlan& p, const double2* W, void* f, cudaStream_t s, int row_lo,
                        int row_hi, const Batch& bt) {
  int sh = gamma_shift(g.ng, g.na, (row_hi - row_lo) * count(bt));
  const MmLevel& lv = p.l1;
  const int rows = g.real ? g.nplanes : g.ng;
  while (sh > 4 && (size_t)rows * ((1 << sh) + 2) * sizeof(double2) > kSmemMax / 4) sh--;
  const size_t smem = (size_t)rows * ((1 << sh) + 2) * sizeof(double2);
  const dim3 grid((g.na + (1 << sh) - 1) >> sh, row_hi - row_lo, count(bt));
  const SigIo io = sig_io(bt, f);
  if (g.real) {
    return launch_after(inv_gamma_real_mm_kernel, grid, kGT, smem, s, g, lv, W, io, sh, row_lo);
  }
  return launch_after(inv_gamma_mm_kernel, grid, kGT, smem, s, g, lv, W, io, sh, row_lo);
}

int launch_mm_fwd_gamma(const Geometry& g, const FftPlan& p, const void* f, double2* W, cudaStream_t s, int row_lo,
                        int row_hi, const Batch& bt) {
  int sh = gamma_shift(g.ng, g.na, (row_hi - row_lo) * count(bt));
  const MmLevel& lv = p.l1;
  while (sh > 4 && (size_t)g.ng * ((1 << sh) + 4) * (g.real ? 8 : 16) > kSmemMax / 4) sh--;
  const size_t smem = (size_t)g.ng * (g.real ? ((1 << sh) + 4) * 8 : ((1 << sh) + 2) * 16);
  const dim3 grid((g.na + (1 << sh) - 1) >> sh, row_hi - row_lo, count(bt));
  const SigIo io = sig_io(bt, f);
  if (g.real) {
    return launch_after(fwd_gamma_real_mm_kernel, grid, kGT, smem, s, g, lv, io, W, sh, row_lo);
  }
  return launch_after(fwd_gamma_mm_kernel, grid, kGT, smem, s, g, lv, io, W, sh, row_lo);
}

int launch_mm_alpha(const Geometry& g, const FftPlan& p, double2* W, bool inverse, cudaStream_t s, const Batch& bt) {
  const int nrows = g.nplanes * g.nb * count(bt);
  const Shape z = shape_for(p.mm, nrows, p.mm.kind == 1 ? 1 : 2);
  return launch_after(inverse ? alpha_mm_kernel<true> : alpha_mm_kernel<false>, dim3((nrows + z.T - 1) / z.T),
                      32 * z.warps, z.smem, s, g, z.P, W, z.T, nrows, bt.wstride);
}

int launch_mm_inv_beta(const Geometry& g, const FftPlan& p, double2* W, cudaStream_t s, const Batch& bt) {
  const Shape z = shape_for(p.mm, g.L * g.nplanes * count(bt), 2);
  const dim3 grid((g.L + z.T - 1) / z.T, g.nplanes * count(bt));
  return launch_after(inv_beta_mm_kernel, grid, 32 * z.warps, z.smem, s, g, z.P, p.half, W, z.T, bt.wstride);
}

}  // namespace so3g
