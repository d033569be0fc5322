// FP64 Wigner contractions: the O(N L^3) core of the transform.
//
// Inverse (replaces SSHT's per-spin Fmm accumulation called at the
// reference's src/c/so3_core.c:204 and the in-tree src/c/so3_core.c:1081-1165):
//   F[n][m'][m] = i^{n-m} sum_{l >= max(L0,|n|,|m|,m')} (2l+1)/(8 pi^2)
//                 Delta^l_{m'm} Delta^l_{m'n} f_lmn ,   m' >= 0.
// Forward (replaces SSHT's forward Delta sum, src/c/so3_core.c:408-428 and
// in-tree :1589-1617):
//   f_lmn = i^{m-n} sum_{m'=0}^{l} Delta^l_{m'm} Delta^l_{m'n} G[n][m'][m].
//
// Both are three-operand contractions (every pair of the free indices shares
// an operand), so no plain GEMM exists for one signal.  Negative m, n use
// Delta^l_{m',-k} = (-1)^{l+m'} Delta^l_{m'k}: one product w = Delta_{m'|m|}
// Delta_{m'|n|} feeds the four sign combinations (+m,+n), (-m,+n), (+m,-n),
// (-m,-n), and the (-1)^{l+m'} of combinations with one negative index is split
// between the operand that carries l and the one that carries m'.
//
// contract_mma_kernel (below, on the FP64 tensor cores) runs every transform.
// The two kernels before it, on the FP64 FMA pipe, are an independent
// implementation that the tests compare with (SO3GPU_FP64_MMA=0):
//  * CTA tile: 32 output rows (m' for the inverse, l for the forward) x 32 |m|
//    x 2 |n|.  The reduction index (l, resp. m') is walked in chunks of 4,
//    staged in shared memory with cp.async, double buffered.
//  * Lanes form an 8 (rows) x 4 (|m|) grid, warps step |m| by 4: a warp reads
//    32 distinct Delta_{m'|m|} (2 wavefronts with the 36-double row pitch),
//    8 distinct Delta_{m'|n|} pairs and 4 distinct coefficient quadruples
//    (1 wavefront each), for 72 FP64 instructions per lane (9 per 4 complex MACs).
#include <cstdlib>
#include <type_traits>

#include "dft_mm.cuh"
#include "launch.cuh"
#include "so3gpu_internal.h"
#include "tc_sm100.cuh"

namespace so3g {

namespace {
constexpr int kThreads = 256;
constexpr int kRows = 32;    // output rows per CTA (m' or l)
constexpr int kCols = 32;    // |m| per CTA
constexpr int kNG = 2;       // |n| per CTA
constexpr int kChunk = 4;    // reduction steps per shared-memory stage
constexpr int kPitch = 36;   // doubles per staged Delta row (32 + 4: conflict-free)
constexpr int kPer = kRows / 8;  // rows per lane
constexpr double kInv8Pi2 = 0.012665147955292221430803304553147533;  // 1/(8 pi^2)

struct Slab {
  double B[kChunk][kRows][kPitch];  // Delta^l_{row, |m|}
  double A[kChunk][kRows][kNG];     // Delta^l_{row, |n|}  (times (2l+1)/(8 pi^2) in the inverse)
  double2 H[kChunk][kCols][kNG][4]; // coefficients / spectra, sign-folded
};
constexpr size_t kSmem = 2 * sizeof(Slab);

__device__ __forceinline__ double2 ipow_mul(double2 v, int k) {  // v * i^k
  switch (k & 3) {
    case 0: return v;
    case 1: return make_double2(-v.y, v.x);
    case 2: return make_double2(-v.x, -v.y);
    default: return make_double2(v.y, -v.x);
  }
}
__device__ __forceinline__ double2 sc(double2 v, double s) { return make_double2(v.x * s, v.y * s); }

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(valid ? 8 : 0));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// 4 sign combinations s: bit0 -> m negative, bit1 -> n negative.  scale
// multiplies every product (the (2l+1)/(8 pi^2) of the inverse, 1 in the
// forward); oddneg flips the sign of the combinations with one negative index
// ((-1)^l in the inverse, (-1)^{m'} in the forward); symmu != 0 rebuilds the
// -m coefficient of a real signal with N == 1 from the +m one.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(valid ? 16 : 0));
}

template <int NSIGN, bool SYM>
__device__ __forceinline__ void mac_chunk(const Slab& S, int lc, int warp, int lm, int lu, double scale, bool oddneg,
                                          int mu, double2 (&acc)[kPer][kNG][4]) {
  const int col = 4 * warp + lu;
  double2 h[kNG][4];
#pragma unroll
  for (int j = 0; j < kNG; j++) {
#pragma unroll
    for (int s = 0; s < NSIGN; s++) h[j][s] = S.H[lc][col][j][s];
    if (SYM) h[j][1] = (mu & 1) ? make_double2(-h[j][0].x, h[j][0].y) : make_double2(h[j][0].x, -h[j][0].y);
  }
  const double sneg = oddneg ? -scale : scale;
#pragma unroll
  for (int i = 0; i < kPer; i++) {
    const int row = lm + 8 * i;
    const double b = S.B[lc][row][col];
    const double2 a = *reinterpret_cast<const double2*>(&S.A[lc][row][0]);
    const double p0 = b * a.x, p1 = b * a.y;
    const double w0 = p0 * scale, w1 = p1 * scale, v0 = p0 * sneg, v1 = p1 * sneg;
#pragma unroll
    for (int s = 0; s < NSIGN; s++) {
      const bool one_neg = (s == 1) || (s == 2);
      const double x0 = one_neg ? v0 : w0, x1 = one_neg ? v1 : w1;
      acc[i][0][s].x = fma(x0, h[0][s].x, acc[i][0][s].x);
      acc[i][0][s].y = fma(x0, h[0][s].y, acc[i][0][s].y);
      acc[i][1][s].x = fma(x1, h[1][s].x, acc[i][1][s].x);
      acc[i][1][s].y = fma(x1, h[1][s].y, acc[i][1][s].y);
    }
  }
}
}  // namespace

// FP64 contraction engine: the FP64 tensor cores, unless the environment sets
// SO3GPU_FP64_MMA=0 (the FP64 FMA kernels, an independent implementation that
// the tests compare with).
static bool fp64_tensor_cores() {
  const char* e = getenv("SO3GPU_FP64_MMA");
  return !(e && e[0] == '0');
}

struct InvArgs {
  const double2* flmn;
  const long long* base;  // per plane
  const double* dl;
  double2* W;
  int L, N, L0, plane0, n_mode, real, sym_n0;
  int nu_lo, nu_hi;  // |n| range [nu_lo, nu_hi) of this launch
  long long CS, QS;  // column-major scratch strides
  double wconst;     // > 0: this weight for every l instead of (2l+1)/(8 pi^2) (adjoint forward)
};

// ------------------------------------------------------------------ inverse
template <int NSIGN>
__global__ void __launch_bounds__(kThreads, 1) inverse_contract_kernel(InvArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  Slab* st = reinterpret_cast<Slab*>(smraw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lm = lane & 7, lu = lane >> 3;
  const int nu0 = a.nu_lo + blockIdx.x * kNG, mp0 = blockIdx.y * kRows, mu0 = blockIdx.z * kCols;
  const int L = a.L;
  bool act[kNG];
#pragma unroll
  for (int j = 0; j < kNG; j++) act[j] = (nu0 + j < a.nu_hi) && !plane_skipped(a.n_mode, a.N, nu0 + j);

  double2 acc[kPer][kNG][4];
#pragma unroll
  for (int i = 0; i < kPer; i++)
#pragma unroll
    for (int j = 0; j < kNG; j++)
#pragma unroll
      for (int s = 0; s < 4; s++) acc[i][j][s] = make_double2(0.0, 0.0);

  const int lstart = max(max(a.L0, nu0), max(mp0, mu0));
  const int mu_own = mu0 + 4 * warp + lu;
  long long bsel[kNG][2];  // flmn block bases of +|n| and -|n|
#pragma unroll
  for (int j = 0; j < kNG; j++) {
    const int nu = min(nu0 + j, a.N - 1);
    bsel[j][0] = a.base[a.plane0 + nu];
    bsel[j][1] = NSIGN == 4 ? a.base[a.plane0 - nu] : 0;
  }
  const int nchunk = lstart < L ? (L - lstart + kChunk - 1) / kChunk : 0;

  auto stage = [&](int c, Slab& S) {
    const int lbase = lstart + c * kChunk;
    for (int idx = tid; idx < kChunk * kRows * kCols; idx += kThreads) {
      const int lc = idx / (kRows * kCols), rem = idx - lc * kRows * kCols, r = rem / kCols, col = rem - r * kCols;
      const int l = lbase + lc;
      const bool ok = l < L && mp0 + r <= l && mu0 + col <= l;
      const double* src = ok ? a.dl + dl_index(l, mp0 + r, mu0 + col) : a.dl;
      cp_async8(&S.B[lc][r][col], src, ok);
    }
    for (int idx = tid; idx < kChunk * kRows * kNG; idx += kThreads) {
      const int lc = idx / (kRows * kNG), rem = idx - lc * kRows * kNG, r = rem / kNG, j = rem - r * kNG;
      const int l = lbase + lc, nu = nu0 + j;
      const bool ok = l < L && act[j] && mp0 + r <= l && nu <= l;
      const double* src = ok ? a.dl + dl_index(l, mp0 + r, nu) : a.dl;
      cp_async8(&S.A[lc][r][j], src, ok);
    }
    for (int idx = tid; idx < kChunk * kCols * kNG * NSIGN; idx += kThreads) {
      const int lc = idx / (kCols * kNG * NSIGN), rem = idx - lc * kCols * kNG * NSIGN;
      const int col = rem / (kNG * NSIGN), rem2 = rem - col * kNG * NSIGN, j = rem2 / NSIGN, sg = rem2 - j * NSIGN;
      const int l = lbase + lc, nu = nu0 + j, mu = mu0 + col;
      const bool ok = l < L && act[j] && mu <= l && nu <= l;
      const int m = (sg & 1) ? -mu : mu;
      const double2* src = ok ? a.flmn + bsel[j][sg >> 1] + (long long)l * l + l + m : a.flmn;
      cp_async16(&S.H[lc][col][j][sg], src, ok);
    }
  };

  if (nchunk > 0) {
    stage(0, st[0]);
    cp_commit();
    for (int c = 0; c < nchunk; c++) {
      if (c + 1 < nchunk) {
        stage(c + 1, st[(c + 1) & 1]);
        cp_commit();
        cp_wait<1>();
      } else {
        cp_wait<0>();
      }
      __syncthreads();
      const Slab& S = st[c & 1];
      const int lbase = lstart + c * kChunk;
#pragma unroll
      for (int lc = 0; lc < kChunk; lc++) {
        const int l = lbase + lc;
        const double cl = a.wconst > 0.0 ? a.wconst : (2.0 * l + 1.0) * kInv8Pi2;
        if (a.sym_n0)
          mac_chunk<NSIGN, true>(S, lc, warp, lm, lu, cl, l & 1, mu_own, acc);
        else
          mac_chunk<NSIGN, false>(S, lc, warp, lm, lu, cl, l & 1, mu_own, acc);
      }
      __syncthreads();
    }
  }

  const int mu = mu0 + 4 * warp + lu;
  if (mu >= L) return;
#pragma unroll
  for (int i = 0; i < kPer; i++) {
    const int mp = mp0 + lm + 8 * i;
    if (mp >= L) continue;
    const double odd_mp = (mp & 1) ? -1.0 : 1.0;
#pragma unroll
    for (int j = 0; j < kNG; j++) {
      const int nu = nu0 + j;
      if (nu >= a.nu_hi) continue;
#pragma unroll
      for (int s = 0; s < NSIGN; s++) {
        const int ms = (s & 1) ? -1 : 1, ns = (s & 2) ? -1 : 1;
        if (ms < 0 && mu == 0) continue;
        if (ns < 0 && nu == 0) continue;
        const int m = ms * mu, n = ns * nu;
        double2 v = acc[i][j][s];
        if (ms * ns < 0) v = sc(v, odd_mp);
        v = ipow_mul(v, n - m + 4 * L);
        a.W[(long long)(a.plane0 + n) * a.QS + (long long)(m + L - 1) * a.CS + mp] = v;
      }
    }
  }
}

// ------------------------------------------------------------------ forward
struct FwdArgs {
  const double2* W;
  const long long* base;
  const double* dl;
  double2* flmn;
  int L, N, L0, plane0, n_mode, real, compact;
  int nu_lo, nu_hi;  // |n| range [nu_lo, nu_hi) of this launch
  long long CS, QS;  // column-major scratch strides
  double lw;         // > 0: outputs times lw (2l+1) (adjoint inverse)
};

template <int NSIGN>
__global__ void __launch_bounds__(kThreads, 1) forward_contract_kernel(FwdArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  Slab* st = reinterpret_cast<Slab*>(smraw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lm = lane & 7, lu = lane >> 3;
  const int nu0 = a.nu_lo + blockIdx.x * kNG, l0 = blockIdx.y * kRows, mu0 = blockIdx.z * kCols;
  const int L = a.L;
  bool act[kNG];
#pragma unroll
  for (int j = 0; j < kNG; j++) act[j] = (nu0 + j < a.nu_hi) && !plane_skipped(a.n_mode, a.N, nu0 + j);
  if (!act[0] && !act[1]) return;  // caller-zeroed blocks stay untouched

  double2 acc[kPer][kNG][4];
#pragma unroll
  for (int i = 0; i < kPer; i++)
#pragma unroll
    for (int j = 0; j < kNG; j++)
#pragma unroll
      for (int s = 0; s < 4; s++) acc[i][j][s] = make_double2(0.0, 0.0);

  const int ltop = min(L - 1, l0 + kRows - 1);
  const bool any = ltop >= max(max(a.L0, nu0), mu0);
  const int nchunk = any ? (ltop + 1 + kChunk - 1) / kChunk : 0;

  auto stage = [&](int c, Slab& S) {
    const int mbase = c * kChunk;
    for (int idx = tid; idx < kChunk * kRows * kCols; idx += kThreads) {
      const int mc = idx / (kRows * kCols), rem = idx - mc * kRows * kCols, r = rem / kCols, col = rem - r * kCols;
      const int mp = mbase + mc, l = l0 + r;
      const bool ok = l < L && mp <= l && mu0 + col <= l;
      const double* src = ok ? a.dl + dl_index(l, mp, mu0 + col) : a.dl;
      cp_async8(&S.B[mc][r][col], src, ok);
    }
    for (int idx = tid; idx < kChunk * kRows * kNG; idx += kThreads) {
      const int mc = idx / (kRows * kNG), rem = idx - mc * kRows * kNG, r = rem / kNG, j = rem - r * kNG;
      const int mp = mbase + mc, l = l0 + r, nu = nu0 + j;
      const bool ok = l < L && act[j] && mp <= l && nu <= l;
      const double* src = ok ? a.dl + dl_index(l, mp, nu) : a.dl;
      cp_async8(&S.A[mc][r][j], src, ok);
    }
    for (int idx = tid; idx < kChunk * kCols * kNG * NSIGN; idx += kThreads) {
      // m' fastest: consecutive threads read consecutive entries of a column
      const int mc = idx % kChunk, rem = idx / kChunk;
      const int col = rem / (kNG * NSIGN), rem2 = rem - col * kNG * NSIGN, j = rem2 / NSIGN, sg = rem2 - j * NSIGN;
      const int mp = mbase + mc, nu = nu0 + j, mu = mu0 + col;
      const bool ok = mp < L && act[j] && mu < L;
      const int n = (sg & 2) ? -nu : nu, m = (sg & 1) ? -mu : mu;
      const double2* src =
          ok ? a.W + (long long)(a.plane0 + n) * a.QS + (long long)(L - 1 + m) * a.CS + mp : a.W;
      cp_async16(&S.H[mc][col][j][sg], src, ok);
    }
  };

  if (nchunk > 0) {
    stage(0, st[0]);
    cp_commit();
    for (int c = 0; c < nchunk; c++) {
      if (c + 1 < nchunk) {
        stage(c + 1, st[(c + 1) & 1]);
        cp_commit();
        cp_wait<1>();
      } else {
        cp_wait<0>();
      }
      __syncthreads();
      const Slab& S = st[c & 1];
#pragma unroll
      for (int mc = 0; mc < kChunk; mc++) mac_chunk<NSIGN, false>(S, mc, warp, lm, lu, 1.0, (c * kChunk + mc) & 1, 0, acc);
      __syncthreads();
    }
  }

  const int mu = mu0 + 4 * warp + lu;
  if (mu >= L) return;
#pragma unroll
  for (int i = 0; i < kPer; i++) {
    const int l = l0 + lm + 8 * i;
    if (l >= L || mu > l) continue;
    const double odd_l = (l & 1) ? -1.0 : 1.0;
#pragma unroll
    for (int j = 0; j < kNG; j++) {
      const int nu = nu0 + j;
      if (!act[j]) continue;
      if (a.compact && l < nu) continue;  // not stored
#pragma unroll
      for (int s = 0; s < NSIGN; s++) {
        const int ms = (s & 1) ? -1 : 1, ns = (s & 2) ? -1 : 1;
        if (ms < 0 && mu == 0) continue;
        if (ns < 0 && nu == 0) continue;
        const int m = ms * mu, n = ns * nu;
        double2 v = make_double2(0.0, 0.0);
        if (l >= max(a.L0, nu)) {
          v = acc[i][j][s];
          if (ms * ns < 0) v = sc(v, odd_l);
          v = ipow_mul(v, m - n + 4 * L);
          if (a.lw > 0.0) v = sc(v, a.lw * (2.0 * l + 1.0));
        }
        a.flmn[a.base[a.plane0 + n] + (long long)l * l + l + m] = v;
      }
    }
  }
}

// ------------------------------------------------------------------ FP64 tensor cores
// Both contractions on the FP64 tensor cores (mma.sync m8n8k4 f64).  For a pair
// (mu, nu) = (|m|, |n|) they are products with W = Delta_{m' mu} Delta_{m' nu}:
//   inverse  Y[m', c] = sum_l  W[m', l] X[l, c]
//   forward  Y[l, c]  = sum_m' W[m', l] X[m', c]
// with 8 columns c = 2 s + part: sign combination s (bit 0: m = -mu, bit 1:
// n = -nu) and real / imaginary part.  One MMA: 8 rows x 8 columns x 4
// reduction steps (256 multiply-adds), its row operand formed in registers by
// one multiplication.  (2l+1)/(8 pi^2) rides on the nu factor, the sign
// (-1)^(reduction index) of combinations with one negative index is flipped in
// the column operand, the one of the row index in the result.
//
// CTA tile: 32 rows x 8 mu x 2 nu; 8 reduction entries (two MMA steps) per stage
// of a ring.  Eight warps multiply (16 rows x 4 mu x 1 nu each: 14 fragment reads
// per 8 MMAs), one (forward) or two (inverse, a nu each) more copy and run ahead:
// the Delta blocks as they are stored (dl_index) by bulk copies, 512 bytes per mu
// and row tile, the coefficients from the caller's layout or the spectra from the
// column-major scratch by cp.async, all counted on mbarriers.  Row tiles that a
// degree does not reach (m' > l) are neither copied nor multiplied.
//
// Bound by the latency of the product warps' chains (wait, fragment read, product,
// MMA): MMAs hold the FP64 pipe 49 % of the time and the multiplications that form W
// 10 %, no other unit above 50 %.  Hence as many warps as fit: forward three CTAs
// per SM at 72 registers and two ring slots, inverse (whose copies scatter and whose
// weight takes registers) two at 96 and three slots; forward as inverse 2.48 ms at
// L = 512, N = 64, inverse as forward 2.77.  Measured at L = 512, N = 64 (ms, inverse
// / forward): 2.54 / 2.36 (2.50 / 2.33 were no warp to look whether its wait gave up),
// against 2.61 / 2.48 with one copying warp and two CTAs in both; 4.97 / 5.92 for staging by all warps with 8-byte copies from row-major
// planes; 3.09 / 2.89 without copying warps (a barrier per chunk aligned the warps'
// bursts).  64 rows x 4 nu (one CTA of 16 warps) gives 2.57 / 2.42 there but 39 / 37
// us against 23 / 30 at L = 128, N = 16.  Two signals per CTA share the Delta reads:
// forward 2.02 ms a signal, inverse 2.51, and 12 % slower below L = 256.  X by
// 128-byte bulk copies: 6.4 / 6.7 ms (64 per stage are too many).  m16n8k8 MMAs
// change nothing.
namespace {
constexpr int kCRt = 4, kCMu = 8, kCNu = 2;  // row tiles, mu, nu of a CTA
constexpr int kCMt = 2;                      // row tiles of a warp (4 mu, 1 nu)
constexpr int contract_slots(int ctas) { return ctas == 3 ? 2 : 3; }  // of the ring, by CTAs per SM
constexpr int kCCopy[2] = {2, 1};    // copying warps
constexpr int kCWarps = (kCRt / kCMt) * 2 * kCNu;  // product warps
constexpr int contract_threads(bool fwd) { return 32 * (kCWarps + kCCopy[fwd]); }
constexpr int kXB = 33;  // slots of an X block of one (mu, nu): 8 entries x 4 combinations, and one of padding

struct ContractArgs {
  void* flmn[kMaxBatch];   // coefficients of each signal (blockIdx.z = mu tile + tiles * signal)
  long long wstride;       // scratch of signal b at W + b * wstride
  const long long* base;   // per plane
  const double* dl;
  double2* W;              // column-major scratch part
  int L, N, L0, plane0, n_mode, nsign, sym_n0, compact;
  int nu_lo, nu_hi, nu0;   // |n| range of this launch; first nu of the grid (a multiple of the tile)
  long long CS, QS;
  double wconst;           // inverse, > 0: this weight for every l
  double lw;               // forward, > 0: outputs times lw (2l+1)
  int* fault;              // the caller's word (Workspace::fault) or null
};

// Bit 2: a wait for a copy gave up (see tc::mbar_wait).  The results that lacked
// the copy are NaN, and so is every sample that depends on them.
__device__ int g_contract_error;

__device__ __forceinline__ void cp16_to(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0));
}

// The end of a copying warp: no copy into the block's shared memory is in flight
// any more, also where a product warp that would have waited for it gave up.  Bulk
// copies by each slot's latest use: st is the slot that comes next, phase the parity
// of its latest use.
__device__ __forceinline__ void drain_copies(uint32_t full0, int slots, int st, uint32_t phase) {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  for (int i = 0; i < slots; i++) tc::mbar_wait(full0 + 8 * i, i < st ? phase ^ 1 : phase, &g_contract_error, 4);
}

constexpr int kCStage = kCRt * kCMu * 64 + kCRt * kCNu * 64 + 2 * kCMu * kCNu * kXB;  // doubles
}  // namespace

template <bool FWD, int CTAS>
__global__ void __launch_bounds__(contract_threads(FWD), CTAS) contract_mma_kernel(const __grid_constant__ ContractArgs a) {
  constexpr int RT = kCRt, NU = kCNu, MT = kCMt, ST = contract_slots(CTAS);
  constexpr int WR = RT / MT, NWARP = kCWarps, CW = kCCopy[FWD];
  constexpr int BSZ = RT * kCMu * 64, ASZ = RT * NU * 64, STAGE = kCStage;
  extern __shared__ __align__(16) double smc[];
  __shared__ long long bsel[NU][2];
  __shared__ __align__(8) unsigned long long full[ST], empty[ST];
  __shared__ volatile int gave_up;  // a wait of this block did: its results are void
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int wr = warp % WR, wm = warp / WR % 2, wn = warp / (2 * WR);
  const int nu0 = a.nu0 + blockIdx.x * NU, rt0 = blockIdx.y * RT;
  const int mts = (a.L + kCMu - 1) / kCMu, sig = blockIdx.z / mts, mu0 = (blockIdx.z - sig * mts) * kCMu;
  double2* const W = a.W + sig * a.wstride;
  const int L = a.L, LC = (L + 7) >> 3;
  unsigned act = 0;  // bit j: nu0 + j is computed by this launch
#pragma unroll
  for (int j = 0; j < NU; j++)
    if (nu0 + j >= a.nu_lo && nu0 + j < a.nu_hi && !plane_skipped(a.n_mode, a.N, nu0 + j)) act |= 1u << j;
  if (FWD && !act) {  // caller-zeroed blocks stay untouched
    dep_wait();  // a launch of such blocks alone must not finish before the stage that the next launch reads
    return;
  }
  if (tid < NU) {
    const int nu = min(nu0 + tid, a.N - 1);
    bsel[tid][0] = a.base[a.plane0 + nu];
    bsel[tid][1] = a.nsign == 4 ? a.base[a.plane0 - nu] : 0;
  }
  __syncthreads();

  // chunks of 8 reduction entries: inverse l >= max(L0, mu, nu, m'), forward m' <= l
  const int lmin = max(max(a.L0, nu0), mu0);
  int ch0, ch1;
  if (FWD) {
    ch0 = 0;
    ch1 = 8 * (rt0 + RT) > lmin ? min(rt0 + RT, LC) : 0;
  } else {
    ch0 = max(lmin >> 3, rt0);
    ch1 = act ? LC : 0;
  }

  const uint32_t full0 = tc::smem_u32(full), empty0 = tc::smem_u32(empty);
  if (tid == 0) {
    gave_up = 0;
    for (int st = 0; st < ST; st++) {
      tc::mbar_init(full0 + 8 * st, 32 * CW + 1);  // the copying lanes' loads of X and the expected bytes
      tc::mbar_init(empty0 + 8 * st, NWARP);
    }
    tc::mbar_fence_init();
  }
  __syncthreads();

  if (warp >= NWARP) {
    // ------------------------------------------------ copies
    // The Delta blocks of a row tile are one run per operand (8 mu, NU nu): 2 RT
    // lanes bring them with one bulk copy each.  X by 16-byte copies, forward
    // with m' fastest (128 bytes of a column), inverse with mu fastest (runs of
    // a coefficient row).
    static_assert(2 * RT <= 32, "one lane per bulk copy");
    const uint32_t sm0 = tc::smem_u32(smc), xs0 = sm0 + (BSZ + ASZ) * 8;
    const int trt = rt0 + lane % RT;
    const bool tmu = lane < RT;
    const uint32_t tdst = sm0 + (tmu ? (trt - rt0) * (kCMu * 512) : BSZ * 8 + (trt - rt0) * (NU * 512));
    const long long toff = (tmu ? mu0 : nu0) * 64;
    // forward: lane = (entry, combination); inverse: lane = (mu, entry & 3)
    const int xe = FWD ? lane & 7 : lane >> 3, xm = lane & 7, xc = lane >> 3;
    constexpr int NJ = NU / CW;  // nu of a copying warp
    const int j0 = (warp - NWARP) * NJ;
    const double2* const flmn = static_cast<const double2*>(a.flmn[sig]);
    const double2* px[FWD ? NJ : 1];
    int poff[FWD ? 1 : 4 * NJ], xlo[NJ];  // coefficient counts fit an int (the C interface)
#pragma unroll
    for (int j = 0; j < NJ; j++) {
      const int nu = nu0 + j0 + j, mu = mu0 + xm;
      if (FWD) {
        px[j] = W + (long long)(a.plane0 + ((xc & 2) ? -nu : nu)) * a.QS + (long long)(L - 1 + ((xc & 1) ? -mu0 : mu0)) * a.CS;
        xlo[j] = xc < a.nsign && (act >> (j0 + j) & 1) ? 0 : L;
      } else {
#pragma unroll
        for (int c = 0; c < 4; c++) poff[4 * j + c] = (int)bsel[j0 + j][c >> 1] + ((c & 1) ? -mu : mu);
        xlo[j] = mu < L && (act >> (j0 + j) & 1) ? max(max(a.L0, mu), nu) : L;
      }
    }
    const long long cstep = (xc & 1) ? -a.CS : a.CS;
    auto blocks = [&](int ch, int st) {
      const int lc = FWD ? trt : ch, mt = FWD ? ch : trt;
      const bool v = lane < 2 * RT && mt <= lc && lc < LC && (tmu ? mu0 <= 8 * lc : nu0 < 8 * (lc + 1));
      const unsigned got = __ballot_sync(0xffffffffu, v);
      if (lane == 0)
        tc::mbar_arrive_expect_tx(full0 + 8 * st, __popc(got & ((1u << RT) - 1)) * (kCMu * 512) +
                                                      __popc(got >> RT) * (NU * 512));
      __syncwarp();
      if (v)
        tc::bulk_g2s(tdst + (uint32_t)(st * STAGE * 8), a.dl + dl_base(lc) + (long long)mt * (512 * (lc + 1)) + toff,
                     (tmu ? kCMu : NU) * 512, full0 + 8 * st);
    };
    // the first Delta blocks come while the kernel before finishes; X is its output
    if (j0 == 0 && ch0 < ch1) blocks(ch0, 0);
    dep_wait();
    int st = 0;
    uint32_t phase = 1;  // of the ring slot's previous use
    for (int ch = ch0; ch < ch1; ch++) {
      if (ch - ch0 >= ST) {
        if (!tc::mbar_wait(empty0 + 8 * st, phase, &g_contract_error, 4, &gave_up)) {
          drain_copies(full0, ST, st, phase);  // the lanes that are left do not wait for one that has gone
          return;
        }
      }
      if (j0 == 0 && ch > ch0) blocks(ch, st);
      const uint32_t at = (uint32_t)(st * STAGE * 8), bar = full0 + 8 * st;
#pragma unroll
      for (int j = 0; j < NJ; j++) {
        if (FWD) {
          const int e = 8 * ch + xe;
          const double2* src = px[j] + e;
#pragma unroll
          for (int m = 0; m < kCMu; m++, src += cstep) {
            const bool ok = e >= xlo[j] && e < L && mu0 + m < L;
            cp16_to(xs0 + at + 16 * (((j0 + j) * kCMu + m) * kXB + xc * 8 + (xe ^ (4 * (xc & 1)))), ok ? src : W, ok);
          }
        } else {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int e = 8 * ch + 4 * h + xe, off = e * e + e;
            const bool in = e >= xlo[j] && e < L;
#pragma unroll
            for (int c = 0; c < 4; c++) {
              const bool ok = in && c < a.nsign;
              cp16_to(xs0 + at + 16 * (((j0 + j) * kCMu + xm) * kXB + 4 * (4 * h + xe) + (c ^ (xe & 2))),
                      ok ? flmn + (poff[4 * j + c] + off) : flmn, ok);
            }
          }
        }
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
      if (++st == ST) st = 0;
      if (st == 0) phase ^= 1;
    }
    drain_copies(full0, ST, st, phase);
    return;
  }

  // -------------------------------------------------- products
  dep_wait();
  double acc[MT][4][2];
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int m = 0; m < 4; m++) acc[i][m][0] = acc[i][m][1] = 0.0;

  const int s = g >> 1, part = g & 1;
  // real signals with N = 1: the -m coefficient is (-1)^m conj of the +m one
  const bool sym = !FWD && a.sym_n0 && s == 1;
  const int xs = sym ? 0 : s;
  // sign of this lane's column entries, for even and odd mu: the parity of the
  // reduction index (entry 4 ks + q) of combinations with one negative index
  const int flip = (s == 1 || s == 2) && (q & 1) ? 0x80000000 : 0;
  const int flip0 = flip ^ (sym && part ? 0x80000000 : 0), flip1 = flip ^ (sym && !part ? 0x80000000 : 0);
  const int slot0 = FWD ? q * 8 + (g ^ ((q >> 1) * 4)) : g * 8 + (q ^ (((g >> 1) & 1) * 4));
  const int x0 = FWD ? 2 * (s * 8 + (q ^ (4 * (s & 1)))) + part : 2 * (4 * q + (xs ^ (q & 2))) + part;
  // weight (2l+1)/(8 pi^2), or the constant one: fma(2l+1, wmul, wadd) is exact in its product
  const double wmul = a.wconst > 0.0 ? 0.0 : kInv8Pi2, wadd = a.wconst > 0.0 ? a.wconst : 0.0;
  double l21 = 2.0 * (8 * ch0 + q) + 1.0;
  const int rt_lo = rt0 + wr * MT;
  // one chunk; ALL: every row tile of the warp has entries with m' <= l
  auto products = [&](int ch, int st, auto all) {
    constexpr bool ALL = decltype(all)::value;
    const double* Bs = smc + st * STAGE + (wr * MT * kCMu + wm * 4) * 64;
    const double* As = smc + st * STAGE + BSZ + (wr * MT * NU + wn) * 64;
    const double* Xs = smc + st * STAGE + BSZ + ASZ + 2 * (wn * kCMu + wm * 4) * kXB + x0;
#pragma unroll
    for (int ks = 0; ks < 2; ks++) {
      // entry 4 + q: forward the lower half block (its row pairs swap alike), inverse the other l half
      const int slot = FWD ? slot0 + 32 * ks : slot0 ^ (4 * ks);
      const int dx = FWD ? 8 * ks * (1 - 2 * (s & 1)) : 32 * ks;
      const double w = fma(l21 + 8.0 * ks, wmul, wadd);
      double an[MT];
#pragma unroll
      for (int i = 0; i < MT; i++) {
        an[i] = As[i * NU * 64 + slot];
        if (!FWD) an[i] *= w;
      }
#pragma unroll
      for (int m = 0; m < 4; m++) {
        double x = Xs[2 * m * kXB + dx], wp[MT];
        x = __hiloint2double(__double2hiint(x) ^ ((m & 1) ? flip1 : flip0), __double2loint(x));
#pragma unroll
        for (int i = 0; i < MT; i++) wp[i] = Bs[(i * kCMu + m) * 64 + slot] * an[i];
#pragma unroll
        for (int i = 0; i < MT; i++) {
          if (!ALL && (FWD ? ch > rt_lo + i || rt_lo + i >= LC : rt_lo + i > ch)) continue;  // m' > l throughout
          mm::dmma(acc[i][m], wp[i], x);
        }
      }
    }
  };
  const int rt_hi = rt_lo + MT - 1;
  int st = 0;
  uint32_t phase = 0;
  for (int ch = ch0; ch < ch1; ch++) {
    if (!__all_sync(0xffffffffu, tc::mbar_wait(full0 + 8 * st, phase, &g_contract_error, 4, &gave_up))) break;
    if (FWD ? (ch <= rt_lo && rt_hi < LC) : rt_hi <= ch)
      products(ch, st, std::true_type{});
    else
      products(ch, st, std::false_type{});
    l21 += 16.0;
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(empty0 + 8 * st);
    if (++st == ST) st = 0, phase ^= 1;
  }
  if (gave_up) {
    if (a.fault) *static_cast<volatile int*>(a.fault) = 4;
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int m = 0; m < 4; m++) acc[i][m][0] = acc[i][m][1] = __longlong_as_double(0x7ff8000000000000ll);
  }

  dep_launch();
  // accumulator (row g, columns 2q, 2q+1) = combination q, real / imaginary part
  const int ms = (q & 1) ? -1 : 1, ns = (q & 2) ? -1 : 1;
  if (q >= a.nsign) return;
#pragma unroll
  for (int i = 0; i < MT; i++) {
    const int row = 8 * (rt0 + wr * MT + i) + g;
    if (row >= L) break;
    const double odd_row = (row & 1) ? -1.0 : 1.0;
    const int nu = nu0 + wn;
    if (nu < a.nu_lo || nu >= a.nu_hi || (ns < 0 && nu == 0)) break;
    const bool on = act >> wn & 1;
    if (FWD && (!on || (a.compact && row < nu))) continue;  // untouched, or not stored
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int mu = mu0 + wm * 4 + m;
      if (mu >= L || (ms < 0 && mu == 0) || (FWD && mu > row)) continue;
      double2 v = make_double2(acc[i][m][0], acc[i][m][1]);
      if (ms * ns < 0) v = sc(v, odd_row);
      if (FWD) {
        if (row >= max(a.L0, nu)) {
          v = ipow_mul(v, ms * mu - ns * nu + 4 * L);
          if (a.lw > 0.0) v = sc(v, a.lw * (2.0 * row + 1.0));
        } else {
          v = make_double2(0.0, 0.0);
        }
        static_cast<double2*>(a.flmn[sig])[bsel[wn][q >> 1] + (long long)row * row + row + ms * mu] = v;
      } else {
        v = ipow_mul(v, ns * nu - ms * mu + 4 * L);
        W[(long long)(a.plane0 + ns * nu) * a.QS + (long long)(ms * mu + L - 1) * a.CS + row] = v;
      }
    }
  }
}

namespace {
template <bool FWD>
int contract(ContractArgs a, const void* flmn, const Batch& bt, cudaStream_t s) {
  for (int b = 0; b < bt.n; b++) a.flmn[b] = bt.io[b];
  if (!bt.n) a.flmn[0] = const_cast<void*>(flmn);
  a.wstride = bt.wstride;
  a.nu0 = a.nu_lo / kCNu * kCNu;  // tiles stay aligned: a block of 8 degrees holds whole groups of nu
  const dim3 grid((a.nu_hi - a.nu0 + kCNu - 1) / kCNu, (a.L + 8 * kCRt - 1) / (8 * kCRt), (a.L + kCMu - 1) / kCMu * (bt.n ? bt.n : 1));
  // Forward, three CTAs per SM where the grid fills them.  A grid that two per SM
  // hold anyway keeps the registers: 9.4 against 10.5 us at L = 16, N = 4 and 10.7
  // against 11.4 us at L = 32, N = 8 (8 signals each).
  const bool three = FWD && (long long)grid.x * grid.y * grid.z > 2 * 148;
  auto* const kernel = three ? contract_mma_kernel<FWD, FWD ? 3 : 2> : contract_mma_kernel<FWD, 2>;
  return launch_after(kernel, grid, contract_threads(FWD), contract_slots(three ? 3 : 2) * kCStage * sizeof(double), s, a);
}
}  // namespace

int contract_take_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_contract_error, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_contract_error, &zero, sizeof(int));
  return v;
}

int launch_inverse_contract(const Geometry& g, int n_mode, const double2* flmn, const long long* bases,
                            const double* dl, double2* W, int sym_n0, cudaStream_t s, int nu_lo, int nu_hi,
                            double wconst, const Batch& bt) {
  if (nu_hi < 0 || nu_hi > g.N) nu_hi = g.N;
  if (nu_lo >= nu_hi) return kOk;
  if (fp64_tensor_cores()) {
    ContractArgs c{};
    c.base = bases, c.dl = dl, c.W = W + g.QOFF;
    c.L = g.L, c.N = g.N, c.L0 = g.L0, c.plane0 = g.plane0, c.n_mode = n_mode, c.nsign = g.real ? 2 : 4;
    c.sym_n0 = sym_n0, c.nu_lo = nu_lo, c.nu_hi = nu_hi, c.CS = g.CS, c.QS = g.QS, c.wconst = wconst;
    c.fault = g.fault;
    return contract<false>(c, flmn, bt, s);
  }
  if (bt.n) {  // the FMA engine runs signal by signal
    for (int b = 0; b < bt.n; b++)
      if (int rc = launch_inverse_contract(g, n_mode, static_cast<const double2*>(bt.io[b]), bases, dl,
                                           W + b * bt.wstride, sym_n0, s, nu_lo, nu_hi, wconst))
        return rc;
    return kOk;
  }
  InvArgs a{flmn, bases, dl, W + g.QOFF, g.L, g.N, g.L0, g.plane0, n_mode, g.real, sym_n0, nu_lo, nu_hi, g.CS, g.QS,
            wconst};
  dim3 grid((nu_hi - nu_lo + kNG - 1) / kNG, (g.L + kRows - 1) / kRows, (g.L + kCols - 1) / kCols);
  if (g.real) {
    SO3G_CUDA(cudaFuncSetAttribute(inverse_contract_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    inverse_contract_kernel<2><<<grid, kThreads, kSmem, s>>>(a);
  } else {
    SO3G_CUDA(cudaFuncSetAttribute(inverse_contract_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    inverse_contract_kernel<4><<<grid, kThreads, kSmem, s>>>(a);
  }
  SO3G_LAUNCHED();
  SO3G_CUDA(cudaGetLastError());
  return kOk;
}

int launch_forward_contract(const Geometry& g, int n_mode, const double2* W, const long long* bases,
                            const double* dl, double2* flmn, int storage_compact, cudaStream_t s, int nu_lo,
                            int nu_hi, double lw, const Batch& bt) {
  if (nu_hi < 0 || nu_hi > g.N) nu_hi = g.N;
  if (nu_lo >= nu_hi) return kOk;
  if (fp64_tensor_cores()) {
    ContractArgs c{};
    c.base = bases, c.dl = dl, c.W = const_cast<double2*>(W) + g.QOFF;
    c.L = g.L, c.N = g.N, c.L0 = g.L0, c.plane0 = g.plane0, c.n_mode = n_mode, c.nsign = g.real ? 2 : 4;
    c.compact = storage_compact, c.nu_lo = nu_lo, c.nu_hi = nu_hi, c.CS = g.CS, c.QS = g.QS, c.lw = lw;
    c.fault = g.fault;
    return contract<true>(c, flmn, bt, s);
  }
  if (bt.n) {
    for (int b = 0; b < bt.n; b++)
      if (int rc = launch_forward_contract(g, n_mode, W + b * bt.wstride, bases, dl, static_cast<double2*>(bt.io[b]),
                                           storage_compact, s, nu_lo, nu_hi, lw))
        return rc;
    return kOk;
  }
  FwdArgs a{W + g.QOFF, bases, dl, flmn, g.L, g.N, g.L0, g.plane0, n_mode, g.real, storage_compact, nu_lo, nu_hi,
            g.CS, g.QS, lw};
  dim3 grid((nu_hi - nu_lo + kNG - 1) / kNG, (g.L + kRows - 1) / kRows, (g.L + kCols - 1) / kCols);
  if (g.real) {
    SO3G_CUDA(cudaFuncSetAttribute(forward_contract_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    forward_contract_kernel<2><<<grid, kThreads, kSmem, s>>>(a);
  } else {
    SO3G_CUDA(cudaFuncSetAttribute(forward_contract_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    forward_contract_kernel<4><<<grid, kThreads, kSmem, s>>>(a);
  }
  SO3G_LAUNCHED();
  SO3G_CUDA(cudaGetLastError());
  return kOk;
}

}  // namespace so3g
