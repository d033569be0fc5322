// Resident Wigner Delta(pi/2) table: quarter planes 0 <= m', m <= l for every
// degree l < Lcap, in the blocked layout of so3gpu_internal.h (dl_index).
//
// Replaces the per-call, per-n recomputation inside SSHT (called from the
// reference's src/c/so3_core.c:204, :408) and the in-tree recursions at
// src/c/so3_core.c:1001-1035.  Both recursions the reference offers are built:
//
//  * Trapani & Navaza (2006): the first row of degree l follows from the first
//    row of degree l-1 (eqs. 9-10; one sweep over l), after which every column
//    m of every degree is an independent three-term recursion down m' (eq. 11):
//    one GPU thread per (l, m), no inter-thread dependence.
//  * Risbo (1996): half-step recursion over the eighth m' >= m >= 0 plus the
//    margin its neighbours need; degree l needs all of degree l-1, so one CTA
//    sweeps the degrees with barriers between the half steps.
//
// Upper-triangle entries (m' < m) are filled from Delta_{m'm} =
// (-1)^{m-m'} Delta_{mm'}.
#include "so3gpu_internal.h"

namespace so3g {

__device__ __forceinline__ double sgn(int k) { return (k & 1) ? -1.0 : 1.0; }

// Row m' = l of every plane: Delta^l_{l,0} = -sqrt((2l-1)/(2l)) Delta^{l-1}_{l-1,0},
// Delta^l_{l,m} = sqrt(l(2l-1) / (2(l+m)(l+m-1))) Delta^{l-1}_{l-1,m-1}.
__global__ void dl_trapani_top_rows(double* __restrict__ T, int Lcap) {
  if (threadIdx.x == 0) T[0] = 1.0;
  __syncthreads();
  for (int l = 1; l < Lcap; l++) {
    for (int m = threadIdx.x; m <= l; m += blockDim.x) {
      double v;
      if (m == 0)
        v = -sqrt((2.0 * l - 1.0) / (2.0 * l)) * T[dl_index(l - 1, l - 1, 0)];
      else
        v = sqrt((double)l * (2.0 * l - 1.0) / (2.0 * (l + m) * (l + m - 1.0))) * T[dl_index(l - 1, l - 1, m - 1)];
      T[dl_index(l, l, m)] = v;
    }
    __syncthreads();
  }
}

// Column m of plane l, rows m' = l-1 .. m:
// sqrt((l-m')(l+m'+1)) D_{m'} = 2m D_{m'+1} - sqrt((l-m'-1)(l+m'+2)) D_{m'+2}.
__global__ void dl_trapani_columns(double* __restrict__ T) {
  const int l = blockIdx.x;
  for (int m = threadIdx.x; m <= l; m += blockDim.x) {
    double d1 = T[dl_index(l, l, m)], d2 = 0.0;  // D_{m'+1}, D_{m'+2}
    for (int mp = l - 1; mp >= m; mp--) {
      const double t1 = sqrt((double)(l - mp) * (double)(l + mp + 1));
      const double t2 = (mp + 2 <= l) ? sqrt((double)(l - mp - 1) * (double)(l + mp + 2)) : 0.0;
      const double d0 = (2.0 * m * d1 - t2 * d2) / t1;
      T[dl_index(l, mp, m)] = d0;
      d2 = d1;
      d1 = d0;
    }
  }
}

__global__ void dl_fill_upper(double* __restrict__ T) {
  const int l = blockIdx.x;
  const int ld = l + 1;
  for (int i = threadIdx.x; i < ld * ld; i += blockDim.x) {
    const int m = i / ld, mp = i - m * ld;
    if (mp < m) T[dl_index(l, mp, m)] = sgn(m - mp) * T[dl_index(l, m, mp)];
  }
}

int launch_build_dl_trapani(double* table, int L0cap, int Lcap, cudaStream_t s) {
  (void)L0cap;
  SO3G_CUDA(cudaMemsetAsync(table, 0, (size_t)dl_entries(Lcap) * sizeof(double), s));
  dl_trapani_top_rows<<<1, 1024, 0, s>>>(table, Lcap);
  SO3G_LAUNCHED();
  dl_trapani_columns<<<Lcap, 256, 0, s>>>(table);
  SO3G_LAUNCHED();
  dl_fill_upper<<<Lcap, 256, 0, s>>>(table);
  SO3G_LAUNCHED();
  SO3G_CUDA(cudaGetLastError());
  return kOk;
}

// ---------------------------------------------------------------- Risbo
// Work layout: nine (Lcap+6)^2 layers, index (u+3)*S + (v+3) for u, v >= -3.
// Layer l % 8 holds integer degree l on the eighth plus margin; the last one the
// half degree l+1/2 with H(xp, yp) = d_{xp-1/2, yp-1/2}.  One CTA computes 8
// degrees (from el0, a multiple of 8), then dl_risbo_pack puts them into their
// blocks of the table with the whole device: the sweep's own 8-byte stores 64
// bytes apart took as long as its arithmetic (Lcap = 512: 111 ms in all, 88 into
// row-major planes).
__global__ void __launch_bounds__(1024) dl_risbo_sweep(double* __restrict__ work, int Lcap, int el0) {
  const int S = Lcap + 6;
  double* A = nullptr;
  double* H = work + 8 * (size_t)S * S;
#define RA(u, v) A[((u) + 3) * S + ((v) + 3)]
#define RH(u, v) H[((u) + 3) * S + ((v) + 3)]
  const int tid = threadIdx.x, nt = blockDim.x;
  const double c = 0.70710678118654752440084436210484903928;  // cos(pi/4) = sin(pi/4)
  if (el0 == 0 && tid == 0) work[3 * S + 3] = 1.0;
  __syncthreads();
  for (int el = max(el0, 1); el < el0 + 8; el++) {
    const int l = el - 1;
    A = work + (l & 7) * (size_t)S * S;
    // margin of degree l
    for (int i = tid; i < 2 * (l + 1); i += nt) {
      const int u = i >> 1, v = u + 1 + (i & 1);
      RA(u, v) = v <= l ? sgn(v - u) * RA(v, u) : 0.0;
    }
    __syncthreads();
    for (int u = tid; u <= l; u += nt) RA(u, -1) = sgn(l + u) * RA(u, 1);
    __syncthreads();
    if (tid < 6) {
      // (u, v) pairs: (1,-1),(1,0),(1,1),(2,-1),(2,0),(3,-1)
      const int us[6] = {1, 1, 1, 2, 2, 3}, vs[6] = {-1, 0, 1, -1, 0, -1};
      const int u = us[tid], v = vs[tid];
      RA(-u, v) = (u <= l) ? sgn(l + v) * RA(u, v) : 0.0;
    }
    __syncthreads();
    // half degree J = l + 1/2
    {
      const int tJ = 2 * l + 1;
      const double inv = 1.0 / tJ;
      const int W = l + 3, Hh = l + 2;  // xp in [-1, l+1], yp in [0, l+1]
      for (int i = tid; i < W * Hh; i += nt) {
        const int yp = i / W, xp = i - yp * W - 1;
        const int x0 = yp - 1 > -l ? yp - 1 : -l;
        if (xp < x0) continue;
        const int a = l + xp, b = l + yp;
        const double sa = sqrt((double)a), sb = sqrt((double)b);
        const double sA = sqrt((double)(tJ - a)), sB = sqrt((double)(tJ - b));
        const double v = sa * sb * c * RA(xp - 1, yp - 1) - sa * sB * c * RA(xp - 1, yp) +
                         sA * sb * c * RA(xp, yp - 1) + sA * sB * c * RA(xp, yp);
        RH(xp, yp) = v * inv;
      }
    }
    __syncthreads();
    // integer degree el on the eighth
    A = work + (el & 7) * (size_t)S * S;
    {
      const int tJ = 2 * el;
      const double inv = 1.0 / tJ;
      const int W = el + 1;
      for (int i = tid; i < W * W; i += nt) {
        const int v = i / W, u = i - v * W;
        if (u < v) continue;
        const int a = el + u, b = el + v;
        const double sa = sqrt((double)a), sb = sqrt((double)b);
        const double sA = sqrt((double)(tJ - a)), sB = sqrt((double)(tJ - b));
        const double val = sa * sb * c * RH(u, v) - sa * sB * c * RH(u, v + 1) + sA * sb * c * RH(u + 1, v) +
                           sA * sB * c * RH(u + 1, v + 1);
        RA(u, v) = val * inv;
      }
    }
    __syncthreads();
  }
#undef RA
#undef RH
}

// Degrees 8 lc .. 8 lc + 7 from their layers into the table, one thread per entry.
__global__ void dl_risbo_pack(double* __restrict__ T, const double* __restrict__ work, int Lcap, int lc) {
  const int S = Lcap + 6, cols = 8 * (lc + 1), i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 64 * cols * (lc + 1)) return;
  const int at = i & 63, mu = (i >> 6) % cols, mp = 8 * ((i >> 6) / cols) + (at >> 3);
  const int el = 8 * lc + ((at & 7) ^ (((mp >> 1) & 1) * 4));  // dl_slot
  const double* A = work + (el & 7) * (size_t)S * S;
  double v = 0.0;
  if (mp <= el && mu <= el)
    v = mu <= mp ? A[(mp + 3) * S + mu + 3] : sgn(mu - mp) * A[(mu + 3) * S + mp + 3];
  T[dl_base(lc) + i] = v;
}

size_t risbo_work_bytes(int Lcap) { return 9 * (size_t)(Lcap + 6) * (Lcap + 6) * sizeof(double); }

// Lcap: a multiple of 8; work: risbo_work_bytes(Lcap).
int launch_build_dl_risbo(double* table, int Lcap, double* work, cudaStream_t s) {
  SO3G_CUDA(cudaMemsetAsync(work, 0, risbo_work_bytes(Lcap), s));
  for (int lc = 0; lc < Lcap / 8; lc++) {
    dl_risbo_sweep<<<1, 1024, 0, s>>>(work, Lcap, 8 * lc);
    SO3G_LAUNCHED();
    dl_risbo_pack<<<2 * (lc + 1) * (lc + 1), 256, 0, s>>>(table, work, Lcap, lc);
    SO3G_LAUNCHED();
  }
  SO3G_CUDA(cudaGetLastError());
  return kOk;
}

}  // namespace so3g
