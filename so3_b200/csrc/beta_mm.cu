// Beta stages as matrix products on the FP64 tensor cores.
//
// Every beta stage maps a column (plane n, order m, s = (-1)^{m+n}) of nb
// samples to the L spectrum entries m' >= 0 or back by one real matrix per
// parity s, times i for s = -1:
//   inverse          y(k) = sum_{m'} C_s(k, m') F(m'),  C_+ = 2 cos(m' beta_k) (1 at m' = 0),
//                                                       C_- = 2 sin(m' beta_k)
//   forward          G(m') + s G(-m') = sum_b R_s(m', b) x(b): extension onto the circle, its
//                    DFT, the MW phase, the quadrature-weight convolution and the fold at once
//   adjoint inverse  C_s^T, times -i for s = -1
//   adjoint forward  2 pi R_s^T, times -i for s = -1
// (stages.cu has the same stages through DFTs.)  The entry m' = 0 of s = -1
// columns is left out: the contractions meet it with Delta^l_{0m} Delta^l_{0n},
// which is zero unless l+m and l+n are both even.
//
// The product costs 2 L multiply-adds per point and reads and writes the
// planes once; the DFT chain of the forward stage is three to four transforms
// of 2L or 4L points, so the matrix wins wherever those have no compile-time plan
// (see beta_matrix_pays).  A CTA takes 8 MT WR rows x 8 NP WC columns: a warp holds
// MT row tiles of NP column tiles of either parity (4 complex columns each),
// so the two 16-byte values that a lane holds of columns 2c, 2c+1 complete
// each other's sectors.  Matrix fragments are stored in MMA lane order; both
// operands go through a three-stage cp.async ring of 16 reduction entries.
#include <algorithm>

#include "dft_mm.cuh"
#include "launch.cuh"
#include "so3gpu_internal.h"

namespace so3g {

namespace {

constexpr int kK = 16;        // reduction entries per stage (4 MMA steps)
constexpr int kStages = 3;

__device__ __forceinline__ void cp16z(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(valid ? 16 : 0));
}

struct BetaMmArgs {
  const double* tab;       // [parity][row tile][step][lane]
  double2* W;              // scratch of the transform
  int M, K, RT, KS;        // rows, reduction entries; row tiles and steps of the table (zero padded)
  double isign;            // s = -1: times isign * i
  long long wstride;       // blockIdx.z = plane + nplanes * signal
};

// SPEC_IN: reduction over the spectra m' (column-major part -> row-major
// part), else over the beta rows (row-major -> column-major).
template <bool SPEC_IN, int MT, int WR, int NP, int WC>
__global__ void __launch_bounds__(32 * WR * WC, WR * WC == 8 ? 2 : 4) beta_mm_kernel(Geometry g, BetaMmArgs a) {
  constexpr int NTHR = 32 * WR * WC, RT = MT * WR, COLS = 8 * NP * WC, HC = COLS / 2;
  // smem: A[2][RT][4][32] doubles, then B: rows of entries k, parity halves of
  // HC columns (SPEC_IN false) or columns of kK entries (true)
  constexpr int ASZ = 2 * RT * 4 * 32;                      // doubles
  constexpr int KP = 2 * HC + 2, CP = kK + 4;               // pitches: 2 and 4 mod 8 slots
  constexpr int BSZ = SPEC_IN ? COLS * CP : kK * KP;        // double2
  constexpr int STAGE = ASZ + 2 * BSZ;                      // doubles
  extern __shared__ __align__(16) double smd[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wr = warp % WR, wc = warp / WR;
  const int kk = lane & 3, gr = lane >> 2;
  const int ncols = 2 * g.L - 1, c0 = blockIdx.x * COLS, rt0 = blockIdx.y * RT;
  const int sig = blockIdx.z / g.nplanes, plane = blockIdx.z - sig * g.nplanes;
  double2* const W = a.W + sig * a.wstride;
  const int first_is_a = ((g.L - 1 + plane - g.plane0) & 1) == 0;  // even columns have s = +1
  const double2* in = SPEC_IN ? W + g.QOFF + (long long)plane * g.QS + (long long)c0 * g.CS
                              : W + (long long)plane * g.PS + c0;
  const int nch = (a.K + kK - 1) / kK;

  auto stage_matrix = [&](int ch) {
    double* As = smd + (ch % kStages) * STAGE;
    for (int i = tid; i < ASZ / 2; i += NTHR) {  // 16-byte pieces: [parity][row tile][64 of 4 steps]
      const int p = i / (RT * 64), rt = i / 64 % RT, o = i % 64;
      const int par = first_is_a ? p : 1 - p;
      mm::cp16(As + 2 * i, a.tab + (((size_t)par * a.RT + rt0 + rt) * a.KS + 4 * ch) * 32 + 2 * o);
    }
  };
  auto stage_columns = [&](int ch) {
    double2* Bs = reinterpret_cast<double2*>(smd + (ch % kStages) * STAGE + ASZ);
    for (int i = tid; i < COLS * kK; i += NTHR) {
      const int k = SPEC_IN ? i % kK : i / COLS, c = SPEC_IN ? i / kK : i % COLS;
      const bool ok = ch * kK + k < a.K && c0 + c < ncols;
      const double2* src = SPEC_IN ? in + (long long)c * g.CS + ch * kK + k : in + (long long)(ch * kK + k) * g.RS + c;
      const int h = (c & 1) * HC + (c >> 1);
      cp16z(Bs + (SPEC_IN ? h * CP + k : k * KP + h), ok ? src : W, ok);
    }
  };

  double acc[2][MT][NP][2];
#pragma unroll
  for (int p = 0; p < 2; p++)
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int t = 0; t < NP; t++) acc[p][i][t][0] = acc[p][i][t][1] = 0.0;

#pragma unroll
  for (int s = 0; s < kStages - 1; s++)
    if (s < nch) stage_matrix(s);
  dep_wait();  // the columns are the stage before's
#pragma unroll
  for (int s = 0; s < kStages - 1; s++) {
    if (s < nch) stage_columns(s);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  for (int ch = 0; ch < nch; ch++) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2) : "memory");
    __syncthreads();
    if (ch + kStages - 1 < nch) {
      stage_matrix(ch + kStages - 1);
      stage_columns(ch + kStages - 1);
    }
    asm volatile("cp.async.commit_group;\n" ::);
    const double* As = smd + (ch % kStages) * STAGE + wr * MT * 128 + lane;
    const double* Bs = smd + (ch % kStages) * STAGE + ASZ + (gr & 1);
#pragma unroll
    for (int ks = 0; ks < 4; ks++) {
#pragma unroll
      for (int p = 0; p < 2; p++) {
        double b[NP];
#pragma unroll
        for (int t = 0; t < NP; t++) {
          const int h = p * HC + 4 * (wc * NP + t) + (gr >> 1), k = 4 * ks + kk;
          b[t] = Bs[2 * (SPEC_IN ? h * CP + k : k * KP + h)];
        }
#pragma unroll
        for (int i = 0; i < MT; i++) {
          const double w = As[p * RT * 128 + i * 128 + ks * 32];
#pragma unroll
          for (int t = 0; t < NP; t++) mm::dmma(acc[p][i][t], w, b[t]);
        }
      }
    }
  }

  dep_launch();
  // lane (gr, kk): row gr of a tile, columns 2c and 2c + 1 (c = 4 (wc NP + t) + kk)
#pragma unroll
  for (int i = 0; i < MT; i++) {
    const int row = 8 * (rt0 + wr * MT + i) + gr;
    if (row >= a.M) break;
#pragma unroll
    for (int t = 0; t < NP; t++)
#pragma unroll
      for (int p = 0; p < 2; p++) {
        const int c = c0 + 2 * (4 * (wc * NP + t) + kk) + p;
        if (c >= ncols) continue;
        const double* v = acc[p][i][t];
        const double2 y = p == 1 - first_is_a ? make_double2(v[0], v[1])
                                              : make_double2(-a.isign * v[1], a.isign * v[0]);
        if (SPEC_IN)
          W[(long long)plane * g.PS + (long long)row * g.RS + c] = y;
        else
          W[g.QOFF + (long long)plane * g.QS + (long long)c * g.CS + row] = y;
      }
  }
}

// Matrix entries.  half: e^{-i pi k / P}, k < P.
struct Angles {
  const double2* half;
  int P;
  __device__ __forceinline__ double2 at(long long j) const {  // (cos, sin)(pi j / P)
    j %= 2 * P;
    return on_circle((int)(j < 0 ? j + 2 * P : j));
  }
  __device__ __forceinline__ double2 on_circle(int j) const {  // 0 <= j < 2 P
    const double2 e = half[j < P ? j : j - P];
    return j < P ? make_double2(e.x, -e.y) : make_double2(-e.x, e.y);
  }
};
__device__ double synthesis_entry(const Angles& t, int mw, int sc, int k, int mp) {
  const double2 e = t.at((long long)mp * (2 * k + mw));
  return mp == 0 ? (sc ? 0.0 : 1.0) : 2.0 * (sc ? e.y : e.x);
}
// R_s(m', b): the circle's spectrum of the extended unit sample b is
// c(m'') = kappa cos(m'' beta) / P (s = +1) or -2 i sin(m'' beta) / P, kappa =
// 1 at the samples that mirror onto themselves, else 2; against the even
// weights w(p) = 2 / (1 - p^2) (even p), folded.  The odd weights w(+-1)
// cancel in the fold but for the self-mirrored samples of s = -1 columns at
// m' = L - 1.
__device__ double analysis_entry(const Angles& t, int L, int mw, int sc, int mp, int b) {
  const double pi = 3.141592653589793238462643383279502884;
  const bool self = mw ? b == L - 1 : (b == 0 || b == L);
  if (sc) {
    if (mp == 0) return 0.0;
    if (self) return mp == L - 1 ? -2.0 * pi * pi * t.at((long long)(L - 2) * (2 * b + mw)).x / t.P : 0.0;
  }
  double acc = 0.0, low = 0.0;  // compensated: the terms cancel
  const int first = -(L - 1) + ((L - 1 + mp) & 1), turn = 2 * t.P, step = 2 * (2 * b + mw) % turn;
  int j = (int)((long long)first * (2 * b + mw) % turn);
  if (j < 0) j += turn;
  for (int m = first; m <= L - 1; m += 2, j = j + step < turn ? j + step : j + step - turn) {
    const double2 e = t.on_circle(j);
    const double p = mp - m;
    const double term = (sc ? -2.0 * e.y : (self ? e.x : 2.0 * e.x)) * (2.0 / (1.0 - p * p));
    const double sum = acc + term, z = sum - acc;
    low += (acc - (sum - z)) + (term - z);
    acc = sum;
  }
  return (mp ? 4.0 : 2.0) * pi / t.P * (acc + low);
}

__global__ void beta_matrix_tab_kernel(int kind, int L, int mw, Angles t, int M, int K, int RT, int KS, double* tab) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2LL * RT * KS * 32) return;
  const int lane = (int)(i & 31), ks = (int)(i / 32 % KS), rt = (int)(i / 32 / KS % RT), sc = (int)(i / 32 / KS / RT);
  const int row = 8 * rt + lane / 4, k = 4 * ks + lane % 4;
  double v = 0.0;
  if (row < M && k < K) {
    if (kind == kBetaInverse) v = synthesis_entry(t, mw, sc, row, k);
    if (kind == kBetaForward) v = analysis_entry(t, L, mw, sc, row, k);
    if (kind == kBetaAdjInverse) v = synthesis_entry(t, mw, sc, k, row);
    if (kind == kBetaAdjForward) v = 6.283185307179586476925286766559005768 * analysis_entry(t, L, mw, sc, k, row);
  }
  tab[i] = v;
}

void table_shape(const Geometry& g, int kind, int* M, int* K, int* RT, int* KS) {
  const bool to_rows = kind == kBetaInverse || kind == kBetaAdjForward;
  *M = to_rows ? g.nb : g.L;
  *K = to_rows ? g.L : g.nb;
  *RT = (*M + 63) / 64 * 8;  // row tiles of the largest CTA
  *KS = (*K + kK - 1) / kK * (kK / 4);
}

template <bool SPEC_IN, int MT, int WR, int NP, int WC>
int go(const Geometry& g, const BetaMmArgs& a, int nsig, cudaStream_t s) {
  constexpr int COLS = 8 * NP * WC, ROWS = 8 * MT * WR;
  constexpr int BSZ = SPEC_IN ? COLS * (kK + 4) : kK * (COLS + 2);
  constexpr size_t smem = kStages * (2 * MT * WR * 128 + 2 * BSZ) * sizeof(double);
  const dim3 grid((2 * g.L - 1 + COLS - 1) / COLS, (a.M + ROWS - 1) / ROWS, g.nplanes * nsig);
  return launch_after(beta_mm_kernel<SPEC_IN, MT, WR, NP, WC>, grid, 32 * WR * WC, smem, s, g, a);
}

}  // namespace

// Where the matrix replaces the DFTs (us per 31-plane transform, matrix / DFT):
//   inverse  L=64 (8 kernels N=8) 8.8 / 12.6, 80: 16 / 23, 100: 27 / 27, 128: 31 / 27,
//            200: 104 / 56 -- one paired DFT per two columns, so the matrix only while small;
//   forward  L=64 23 / 123 (N=64), 128: 33 / 112, 256: 181 / 580, 300: 317 / 1400,
//            400: 690 / 1900; 15 planes: 600: 1100 / 3350, 1024: 4770 / 6000.  The DFT chain
//            of the 1023-point compile-time plan (L = 512, MW) is faster: 1270 / 976.
// The adjoints have no other path.
bool beta_matrix_pays(const Geometry& g, int kind) {
  if (kind == kBetaInverse) return g.L <= 96;
  if (kind == kBetaForward) return !conv_chain(g);
  return true;
}

size_t beta_matrix_bytes(const Geometry& g, int kind) {
  int M, K, RT, KS;
  table_shape(g, kind, &M, &K, &RT, &KS);
  return 2 * sizeof(double) * (size_t)RT * KS * 32;
}

int launch_beta_matrix_table(const Geometry& g, int kind, const FftPlan& pP, double* tab, cudaStream_t s) {
  int M, K, RT, KS;
  table_shape(g, kind, &M, &K, &RT, &KS);
  const long long n = 2LL * RT * KS * 32;
  beta_matrix_tab_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(kind, g.L, g.mw, Angles{pP.half, g.P}, M, K, RT, KS,
                                                                 tab);
  SO3G_LAUNCHED();
  SO3G_CUDA(cudaGetLastError());
  return kOk;
}

int launch_beta_matrix(const Geometry& g, int kind, const double* tab, double2* W, cudaStream_t s, const Batch& bt) {
  const int nsig = bt.n ? bt.n : 1;
  BetaMmArgs a{};
  a.tab = tab;
  a.W = W;
  a.wstride = bt.wstride;
  table_shape(g, kind, &a.M, &a.K, &a.RT, &a.KS);
  a.isign = kind == kBetaInverse || kind == kBetaForward ? 1.0 : -1.0;
  const bool spec_in = kind == kBetaInverse || kind == kBetaAdjForward;
  // 64 x 64 tiles (two CTAs per SM), 32 x 32 (four per SM; 5-7 % slower per
  // product) where their waves over 148 SMs and the padding of the rows cost
  // less, 16 x 32 where those would not fill half the device.
  const long long big = (long long)((2 * g.L + 62) / 64) * ((a.M + 63) / 64) * g.nplanes * nsig;
  const long long mid = (long long)((2 * g.L + 30) / 32) * ((a.M + 31) / 32) * g.nplanes * nsig;
  if (mid >= 296 && 1.9 * ((big + 295) / 296) <= (mid + 591) / 592)
    return spec_in ? go<true, 4, 2, 2, 4>(g, a, nsig, s) : go<false, 4, 2, 2, 4>(g, a, nsig, s);
  if (mid >= 296) return spec_in ? go<true, 4, 1, 1, 4>(g, a, nsig, s) : go<false, 4, 1, 1, 4>(g, a, nsig, s);
  return spec_in ? go<true, 2, 1, 1, 4>(g, a, nsig, s) : go<false, 2, 1, 1, 4>(g, a, nsig, s);
}

}  // namespace so3g
