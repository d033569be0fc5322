// DFTs on the FP64 tensor cores (mma.sync m8n8k4 f64).
//
// A DFT of prime or small length p over many columns is a matrix product.
// With the pairs s_r = x_r + x_{p-r}, d_r = x_r - x_{p-r} (1 <= r <= p/2)
//   X_q     = x_0 + sum_r cos(2 pi q r / p) s_r - i sum_r sin(2 pi q r / p) d_r
//   X_{p-q} = the same with + i,
// so two real (p/2+1) x (p/2) matrices act on the real and imaginary parts of
// every column: about p multiply-adds per complex point, all on the tensor
// pipe, against the four real products of a plain complex matrix.  For even p
// the unpaired r = p/2 is stored with half its cosine (x_r meets itself).
// A length n = a b runs as two such levels through shared memory with one
// twiddle sweep on the way (n = b n1 + n2, k = k1 + a k2); a length without a
// good split runs as a cyclic convolution (Rader for primes, Bluestein
// otherwise) whose two transforms are themselves two-level.
//
// Why matrices: at 64 FP64 multiply-adds per clock and SM a point that is
// read from and written to HBM once leaves time for about 88 of them, and
// p + P/p (32 + 33 at 1023, 15 + 17 at 255) is below or near that for most
// lengths, while a scalar mixed-radix pass is bound by its shared-memory and
// twiddle loads and by the few warps its registers leave.  One kernel serves
// every length; only loop counts differ.
//
// One MMA: 8 rows q x 8 columns x 4 steps r.  The 8 columns are 4 complex
// columns (real, imaginary interleaved), so lane (g, c) of an accumulator
// holds one complex value: output q = g of column c.  A warp task is MT row
// tiles x NT column tiles; per step it reads 2 MT table fragments (one 16-byte
// (cos, sin) load each, L1 resident) and 2 NT column values, and issues
// 2 MT NT MMAs.
#pragma once
#include "fft_core.cuh"

namespace so3g {
namespace mm {

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// floor(n / d) for n < 65536, magic = ceil(2^32 / d) (d >= 2; magic 0: d = 1)
__device__ __forceinline__ int fastdiv(int n, unsigned magic) { return magic ? (int)__umulhi((unsigned)n, magic) : n; }

__device__ __forceinline__ void cp16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp8(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

constexpr int kNT = 2;  // column tiles of a warp task (8 complex columns)

// One task: row tiles qt0 .. qt0+MT-1 of columns j0 .. j0+7.  Reduction entry
// r of column j is src[off(j) + r * rp].  out.col(j) prepares a column (its
// addresses), out.put(c, q, X_q) takes every output of it.
// INV: conjugate transform (e^{+2 pi i q r / p}).
template <int MT, bool INV, class Off, class Out>
__device__ __forceinline__ void task(const double2* __restrict__ src, int rp, const MmLevel& lv, int qt0, int j0,
                                     int ncols, const Off& off, const Out& out) {
  const int lane = threadIdx.x & 31, kk = lane & 3, g = lane >> 2;
  const double* bp[kNT];
  double a[MT][kNT][2], b[MT][kNT][2], dc[kNT];
  const int p = lv.p, H = lv.H, KS = lv.KS;
#pragma unroll
  for (int t = 0; t < kNT; t++) {
    const int jb = min(j0 + 4 * t + (lane >> 3), ncols - 1);
    bp[t] = reinterpret_cast<const double*>(src + off(jb)) + (g & 1);
    const double2 x0 = src[off(min(j0 + 4 * t + kk, ncols - 1))];
    dc[t] = bp[t][0];
    if (kk) dc[t] = 0.0;
#pragma unroll
    for (int i = 0; i < MT; i++) {
      a[i][t][0] = x0.x;
      a[i][t][1] = x0.y;
      b[i][t][0] = b[i][t][1] = 0.0;
    }
  }
  const double2* tab = lv.tab + (size_t)qt0 * KS * 32 + lane;
  const int tstep = KS * 32;
  const int rp2 = 2 * rp, rpp = rp2 * p;
#pragma unroll 2
  for (int ks = 0; ks < KS; ks++) {
    const int r = min(4 * ks + kk + 1, H) * rp2;  // entries above H meet zero table entries
    double s[kNT], d[kNT];
#pragma unroll
    for (int t = 0; t < kNT; t++) {
      const double xp = bp[t][r], xn = bp[t][rpp - r];
      s[t] = xp + xn;
      d[t] = INV ? xn - xp : xp - xn;
      dc[t] += s[t];
    }
#pragma unroll
    for (int i = 0; i < MT; i++) {
      const double2 w = __ldg(tab + i * tstep + ks * 32);
#pragma unroll
      for (int t = 0; t < kNT; t++) {
        dmma(a[i][t], w.x, s[t]);
        dmma(b[i][t], w.y, d[t]);
      }
    }
  }
#pragma unroll
  for (int t = 0; t < kNT; t++) {
    const int j = j0 + 4 * t + kk;
    if (j >= ncols) break;
    const auto c = out.col(j);
#pragma unroll
    for (int i = 0; i < MT; i++) {
      const int q = 8 * (qt0 + i) + g + lv.q0;
      if (q > H) break;
      out.put(c, q, make_double2(a[i][t][0] + b[i][t][1], a[i][t][1] - b[i][t][0]));
      if (q != 0 && 2 * q != p)
        out.put(c, p - q, make_double2(a[i][t][0] - b[i][t][1], a[i][t][1] + b[i][t][0]));
    }
  }
  if (lv.q0 && qt0 == 0) {
    // X_0 = sum of the column, left out of the row tiles (q0 = 1: H is a
    // multiple of 8, a row tile for q = 0 alone would be seven eighths empty).
    // Each lane has the terms r = 4 ks + kk + 1 of real column g; for even p
    // the last one is x_r + x_r.
#pragma unroll
    for (int t = 0; t < kNT; t++) {
      if (2 * H == p && kk == 3) dc[t] -= bp[t][H * rp2];
      dc[t] += __shfl_xor_sync(0xffffffffu, dc[t], 1);
      dc[t] += __shfl_xor_sync(0xffffffffu, dc[t], 2);
      const double im = __shfl_xor_sync(0xffffffffu, dc[t], 4);
      const int j = j0 + 4 * t + (lane >> 3);
      if ((lane & 7) == 0 && j < ncols) out.put(out.col(j), 0, make_double2(dc[t], im));
    }
  }
}

// One level over ncols columns, tasks (up to two row tiles) dealt to the
// warps of the CTA.
template <bool INV, class Off, class Out>
__device__ __forceinline__ void level(const double2* __restrict__ src, int rp, const MmLevel& lv, int ncols,
                                      const Off& off, const Out& out) {
  const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int ng = lv.QG, nc = (ncols + 4 * kNT - 1) / (4 * kNT);
  int jc = warp, gi = 0;
  while (jc >= nc) jc -= nc, gi++;
  while (gi < ng) {
    const int qt0 = gi * lv.MT, j0 = jc * 4 * kNT;
    const int mt = min(lv.MT, lv.QT - qt0);
    if (mt == 1)
      task<1, INV>(src, rp, lv, qt0, j0, ncols, off, out);
    else
      task<2, INV>(src, rp, lv, qt0, j0, ncols, off, out);
    jc += nwarps;
    while (jc >= nc) jc -= nc, gi++;
  }
}

// Position of entry n of a staged sequence (two-level layouts: row n1 = n / b
// of pitch ldb; pitches are 2 or 6 mod 8 slots, so the 4 rows x 32 bytes that
// half a warp reads, and the stores of the twiddled transpose, fall into
// distinct banks; the one-level layout is dense with sequence pitch 4 mod 8).
__device__ __forceinline__ int pos(const MmPlan& P, int n) {
  if (P.kind == 1) return n;
  const int r = fastdiv(n, P.mdiv_b);
  return r * P.ldb + (n - r * P.b);
}

// First level's outputs: times w_m^{n2 k1}, transposed into Z[n2][k1].
template <bool INV>
struct TwiddleOut {
  double2* Z;
  const double2* tw;
  int b, lda, ts, twc, twk;  // twiddle of (n2, k1) at n2 * twc + k1 * twk
  unsigned db;
  struct Col {
    double2* z;
    const double2* w;
  };
  __device__ __forceinline__ Col col(int j) const {
    const int t = fastdiv(j, db), n2 = j - t * b;
    return {Z + t * ts + n2 * lda, tw + n2 * twc};
  }
  __device__ __forceinline__ void put(const Col& c, int k1, double2 v) const {
    double2 w = __ldg(c.w + k1 * twk);
    c.z[k1] = INV ? make_double2(fma(v.x, w.x, v.y * w.y), fma(v.y, w.x, -v.x * w.y)) : cmul(v, w);
  }
};
// Second level's outputs: X(k1 + a k2) of sequence t to the caller.
template <class Out>
struct SplitOut {
  const Out& out;
  int a;
  unsigned da;
  struct Col {
    typename Out::Seq s;
    int k1;
  };
  __device__ __forceinline__ Col col(int j) const {
    const int t = fastdiv(j, da);
    return {out.seq(t), j - t * a};
  }
  __device__ __forceinline__ void put(const Col& c, int k2, double2 v) const { out.put(c.s, c.k1 + a * k2, v); }
};
// One level: column j is sequence j.
template <class Out>
struct PlainOut {
  const Out& out;
  __device__ __forceinline__ typename Out::Seq col(int j) const { return out.seq(j); }
  __device__ __forceinline__ void put(const typename Out::Seq& s, int q, double2 v) const { out.put(s, q, v); }
};

// The two levels of T sequences staged in A (sequence pitch ts), A -> Z and
// Z -> out, a barrier between them.  FLIP: the split b x a instead of a x b
// (entry n at (n / a) * lda + n % a).  out.seq(t) prepares a sequence,
// out.put(s, k, X_k) takes its outputs.
template <bool INV, bool FLIP>
__device__ __forceinline__ void first_level(const MmPlan& P, const double2* A, double2* Z, int T) {
  const int a = FLIP ? P.b : P.a, b = FLIP ? P.a : P.b;
  const int lda = FLIP ? P.ldb : P.lda, ldb = FLIP ? P.lda : P.ldb, ts = P.ts;
  const unsigned db = FLIP ? P.mdiv_a : P.mdiv_b;
  auto off = [&](int j) {
    const int t = fastdiv(j, db);
    return t * ts + (j - t * b);
  };
  level<INV>(A, ldb, FLIP ? P.lb : P.la, T * b, off,
                TwiddleOut<INV>{Z, P.tw, b, lda, ts, FLIP ? 1 : a, FLIP ? b : 1, db});
}
template <bool INV, bool FLIP, class Out>
__device__ __forceinline__ void second_level(const MmPlan& P, const double2* Z, int T, const Out& out) {
  const int a = FLIP ? P.b : P.a, lda = FLIP ? P.ldb : P.lda, ts = P.ts;
  const unsigned da = FLIP ? P.mdiv_b : P.mdiv_a;
  auto off = [&](int j) {
    const int t = fastdiv(j, da);
    return t * ts + (j - t * a);
  };
  level<INV>(Z, lda, FLIP ? P.la : P.lb, T * a, off, SplitOut<Out>{out, a, da});
}

// Stages entry n (0 <= n < P.n) of a sequence: x(n) returns it.  Convolution
// plans: Bluestein stages x(n) chirp(n) and zero padding up to m, Rader the
// entries in the order of powers of a primitive root and x(0) in x0[0]
// (x0[1] later holds X(0)).
template <bool INV, class X>
__device__ __forceinline__ void stage_conv(const MmPlan& P, double2* A, double2* x0, const X& x) {
  for (int i = threadIdx.x; i < P.m; i += blockDim.x) {
    double2 v = make_double2(0.0, 0.0);
    if (P.rader) {
      v = x(__ldg(P.perm + i));
      if (INV) v.y = -v.y;
    } else if (i < P.n) {
      v = x(i);
      if (INV) v.y = -v.y;
      v = cmul(v, __ldg(P.chirp + i));
    }
    A[pos(P, i)] = v;
  }
  if (P.rader && threadIdx.x == 0) {
    double2 v = x(0);
    if (INV) v.y = -v.y;
    x0[0] = v;
  }
}

// The spectrum of the first transform of a convolution: conj(U V) staged for
// the second one.
struct ConvMid {
  const MmPlan& P;
  double2 *A, *x0;
  struct Seq {
    double2 *a, *x0;
  };
  __device__ __forceinline__ Seq seq(int t) const { return {A + t * P.ts, x0 + 2 * t}; }
  __device__ __forceinline__ void put(const Seq& s, int k, double2 v) const {
    if (P.rader && k == 0) s.x0[1] = cadd(s.x0[0], v);  // X(0), the sum of all entries
    const int r = fastdiv(k, P.mdiv_a);
    s.a[r * P.lda + (k - r * P.a)] = cconj(cmul(v, __ldg(P.kern + k)));
  }
};
// The outputs of the second one.
template <bool INV, class Out>
struct ConvEnd {
  const MmPlan& P;
  const double2* x0;
  const Out& out;
  struct Seq {
    typename Out::Seq s;
    const double2* x0;
  };
  __device__ __forceinline__ Seq seq(int t) const { return {out.seq(t), x0 + 2 * t}; }
  __device__ __forceinline__ void put(const Seq& s, int k, double2 v) const {
    if (P.rader) {
      const double2 y = cadd(s.x0[0], cconj(v));
      out.put(s.s, __ldg(P.perm + P.m + k), INV ? cconj(y) : y);
      if (k == 0) out.put(s.s, 0, INV ? cconj(s.x0[1]) : s.x0[1]);
    } else if (k < P.n) {
      const double2 y = cmul(__ldg(P.chirp + k), cconj(v));
      out.put(s.s, k, INV ? cconj(y) : y);
    }
  }
};

// DFT of T staged sequences (after the caller's barrier).  Convolution plans
// (staged by stage_conv): conj(F(conj(F(u) V))), V = F(v) / m, conjugated again
// for INV; x0: two entries per sequence (Rader).  out may write A for two-level
// and convolution plans, Z for one-level plans.
template <bool INV, class Out>
__device__ __forceinline__ void run(const MmPlan& P, double2* A, double2* Z, int T, double2* x0, const Out& out) {
  if (P.kind == 1) {
    const int ts = P.ts;
    level<INV>(A, 1, P.la, T, [&](int j) { return j * ts; }, PlainOut<Out>{out});
  } else if (P.kind == 2) {
    first_level<INV, false>(P, A, Z, T);
    __syncthreads();
    second_level<INV, false>(P, Z, T, out);
  } else {
    first_level<false, false>(P, A, Z, T);
    __syncthreads();
    second_level<false, false>(P, Z, T, ConvMid{P, A, x0});
    __syncthreads();
    first_level<false, true>(P, A, Z, T);
    __syncthreads();
    second_level<false, true>(P, Z, T, ConvEnd<INV, Out>{P, x0, out});
  }
}

}  // namespace mm
}  // namespace so3g
