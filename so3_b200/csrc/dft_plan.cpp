// Plans of the tensor-core DFTs (dft_mm.cuh): the choice of the split for a
// length, and its tables in device memory.  Host code only.
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>

#include "so3gpu_internal.h"

namespace so3g {

namespace {

typedef std::complex<long double> cld;
const long double kPiL = 3.141592653589793238462643383279502884L;

cld root_l(long long num, long long den) {  // e^{-2 pi i num/den}
  num %= den;
  const long double a = 2.0L * kPiL * (long double)num / (long double)den;
  return cld(cosl(a), -sinl(a));
}

// Longest matrix level: its table has p^2 / 4 entries (1.4 MB at 600) and is
// read from L2 by then; the two-level costs below never prefer a longer one.
constexpr int kMaxLevel = 600;
// Slots of a sequence buffer: two buffers of one sequence in shared memory.
constexpr int kMaxSlots = 6400;

// Tensor-pipe multiply-adds per complex point of one level, padding included.
double level_cost(int p) {
  const int h = p / 2, rows = h > 0 && h % 8 == 0 ? h : (h + 8) / 8 * 8;
  return 4.0 * rows * ((h + 3) / 4 * 4) / p;
}
// What the second level costs beside its products (twiddles, a shared-memory
// round trip and a barrier), in multiply-adds per point.
constexpr double kLevelOverhead = 60.0;

int pitch(int n) {  // smallest pitch >= n that is 2 or 6 mod 8
  while (n % 4 != 2) n++;
  return n;
}

double two_level_cost(int n, int* a, int* b) {
  double best = 1e30;
  for (int p = 2; p * p <= n; p++) {
    if (n % p) continue;
    const int q = n / p;
    if (q > kMaxLevel) continue;
    const double c = level_cost(p) + level_cost(q) + kLevelOverhead;
    // the longer factor first: the last level's stores run along its outputs k1
    if (c < best && (long)q * pitch(p) <= kMaxSlots && (long)p * pitch(q) <= kMaxSlots) best = c, *a = q, *b = p;
  }
  return best;
}

bool is_prime(int n) {
  if (n < 2) return false;
  for (int p = 2; p * p <= n; p++)
    if (n % p == 0) return false;
  return true;
}

int primitive_root(int n) {
  std::vector<int> f;
  int r = n - 1;
  for (int p = 2; p * p <= r; p++)
    if (r % p == 0) {
      f.push_back(p);
      while (r % p == 0) r /= p;
    }
  if (r > 1) f.push_back(r);
  auto power = [&](long long b, int e) {
    long long v = 1;
    for (b %= n; e; e >>= 1, b = b * b % n)
      if (e & 1) v = v * b % n;
    return v;
  };
  for (int g = 2;; g++) {
    bool ok = true;
    for (int p : f) ok = ok && power(g, (n - 1) / p) != 1;
    if (ok) return g;
  }
}

void level_shape(int p, bool sum_apart, MmLevel* v) {
  v->p = p;
  v->H = p / 2;
  v->KS = (v->H + 3) / 4;
  v->q0 = sum_apart && v->H > 0 && v->H % 8 == 0;
  v->QT = v->q0 ? v->H / 8 : v->H / 8 + 1;
  v->MT = v->QT < 2 ? v->QT : 2;
  v->QG = (v->QT + v->MT - 1) / v->MT;
}

void level_table(const MmLevel& v, std::vector<double2>* host) {
  std::vector<cld> w(v.p);
  for (int k = 0; k < v.p; k++) w[k] = root_l(k, v.p);
  for (int t = 0; t < v.QT; t++)
    for (int s = 0; s < v.KS; s++)
      for (int lane = 0; lane < 32; lane++) {
        const int q = 8 * t + lane / 4 + v.q0, r = 4 * s + lane % 4 + 1;
        double2 e = make_double2(0.0, 0.0);
        if (q <= v.H && r <= v.H) {
          const cld x = w[(long long)q * r % v.p];
          const bool self = 2 * r == v.p;  // x_r paired with itself
          e = make_double2((double)(self ? 0.5L * x.real() : x.real()), self ? 0.0 : (double)-x.imag());
        }
        host->push_back(e);
      }
}

// DFT of x (length a * b) in long double, two-level.
std::vector<cld> dft_host(const std::vector<cld>& x, int a, int b) {
  const int n = a * b;
  std::vector<cld> wn(n), y(n), z(n);
  for (int k = 0; k < n; k++) wn[k] = root_l(k, n);
  for (int n2 = 0; n2 < b; n2++)
    for (int k1 = 0; k1 < a; k1++) {
      cld s(0, 0);
      for (int n1 = 0; n1 < a; n1++) s += x[b * n1 + n2] * wn[(long long)n1 * k1 % a * b];
      y[n2 * a + k1] = s * wn[(long long)n2 * k1 % n];
    }
  for (int k1 = 0; k1 < a; k1++)
    for (int k2 = 0; k2 < b; k2++) {
      cld s(0, 0);
      for (int n2 = 0; n2 < b; n2++) s += y[n2 * a + k1] * wn[(long long)n2 * k2 % b * a];
      z[k1 + a * k2] = s;
    }
  return z;
}

double2 to_d2(cld v) { return make_double2((double)v.real(), (double)v.imag()); }
unsigned magic(int d) { return d < 2 ? 0u : (unsigned)((0x100000000ULL + d - 1) / d); }

}  // namespace

// Cheapest of one level, two levels and a cyclic convolution (Rader's for
// primes; Bluestein's over the cheapest m in [2n-1, 2.3n]).  A convolution
// runs two transforms of length m and touches its points about five more
// times; measured against one level, primes change over near 320.
void mm_plan_host(int n, bool with_mm, bool with_l1, FftPlan* F, MmTables* T) {
  MmPlan P{};
  MmLevel one{};
  std::vector<double2>& host = T->host;
  std::vector<int>& perm = T->perm;
  if (with_l1 && n <= kMaxLevel) level_shape(n, false, &one);  // the real gamma kernels take q = 0 from the tiles
  if (one.p) level_table(one, &host);
  int a = n, b = 1;
  if (with_mm) {
    double best = n <= kMaxLevel ? level_cost(n) : 1e30;
    P.kind = n <= kMaxLevel ? 1 : 0;
    int ta = 0, tb = 0;
    const double c = two_level_cost(n, &ta, &tb);
    if (c < best) best = c, P.kind = 2, a = ta, b = tb;
    if (n > 64) {
      int m = 0, ca = 0, cb = 0;
      bool rader = false;
      double conv = 1e30;
      auto consider = [&](int len, bool r) {
        int ta = 0, tb = 0;
        const double c = (2.0 * two_level_cost(len, &ta, &tb) + 40.0) * len / n;
        if (c < conv) conv = c, m = len, ca = ta, cb = tb, rader = r;
      };
      if (is_prime(n)) consider(n - 1, true);
      for (int len = 2 * n - 1; len <= 2 * n + 3 * n / 10; len++) consider(len, false);
      if (conv < best) best = conv, P.kind = 3, P.rader = rader, P.m = m, a = ca, b = cb;
    }
  }
  if (P.kind) {
    P.n = n;
    P.a = a;
    P.b = b;
    if (P.kind != 3) P.m = n;
    level_shape(a, true, &P.la);
    P.mdiv_a = magic(a);
    P.mdiv_b = magic(b);
    if (P.kind == 1) {
      T->at_a = host.size();
      level_table(P.la, &host);
      P.ts = n;
      while (P.ts % 8 != 4) P.ts++;
    } else {
      level_shape(b, true, &P.lb);
      P.lda = pitch(a);
      P.ldb = pitch(b);
      P.ts = a * P.ldb > b * P.lda ? a * P.ldb : b * P.lda;
      // a sequence buffer also holds the n outputs, and the two columns (n + 1 entries) of
      // an inverse beta pair; a Rader plan transforms only n - 1
      if (P.ts < n + 1) P.ts = n + 1;
      T->at_a = host.size();
      level_table(P.la, &host);
      T->at_b = host.size();
      level_table(P.lb, &host);
      T->at_tw = host.size();
      std::vector<cld> w(P.m);
      for (int k = 0; k < P.m; k++) w[k] = root_l(k, P.m);
      for (int n2 = 0; n2 < b; n2++)
        for (int k1 = 0; k1 < a; k1++) host.push_back(to_d2(w[n2 * k1]));
    }
    if (P.kind == 3) {
      std::vector<cld> v(P.m, cld(0, 0));
      if (P.rader) {
        const int g = primitive_root(n);
        std::vector<int> pw(P.m);
        long long e = 1;
        for (int j = 0; j < P.m; j++, e = e * g % n) pw[j] = (int)e;
        for (int j = 0; j < P.m; j++) perm.push_back(pw[j]);
        for (int j = 0; j < P.m; j++) perm.push_back(pw[(P.m - j) % P.m]);
        for (int j = 0; j < P.m; j++) v[j] = root_l(perm[P.m + j], n);
      } else {
        T->at_chirp = host.size();
        for (int k = 0; k < n; k++) {
          const cld c = root_l((long long)k * k % (2LL * n), 2LL * n);
          host.push_back(to_d2(c));
          v[k] = std::conj(c);
          if (k) v[P.m - k] = std::conj(c);
        }
      }
      T->at_kern = host.size();
      for (const cld& x : dft_host(v, a, b)) host.push_back(to_d2(x / (long double)P.m));
    }
  }
  F->mm = P;
  F->l1 = one;
}

void mm_plan_device(const MmTables& T, const double2* mem, const int* imem, FftPlan* F) {
  F->l1.tab = mem;
  F->mm.la.tab = mem + T.at_a;
  F->mm.lb.tab = mem + T.at_b;
  F->mm.tw = mem + T.at_tw;
  F->mm.chirp = mem + T.at_chirp;
  F->mm.kern = mem + T.at_kern;
  F->mm.perm = imem;
}

int build_mm_plan(int n, FftPlan* F, double2** mem, int** imem, size_t* bytes) {
  MmTables T;
  mm_plan_host(n, true, true, F, &T);
  *mem = nullptr;
  *imem = nullptr;
  *bytes = T.host.size() * sizeof(double2) + T.perm.size() * sizeof(int);
  if (T.host.empty()) return kOk;  // length 1: no entries to multiply
  cudaError_t e = cudaMalloc(mem, T.host.size() * sizeof(double2));
  if (e == cudaSuccess && !T.perm.empty()) e = cudaMalloc(imem, T.perm.size() * sizeof(int));
  if (e != cudaSuccess) {
    cudaFree(*mem);
    *mem = nullptr;
    return fail(kOutOfMemory, "DFT table allocation failed");
  }
  e = upload(*mem, T.host.data(), T.host.size() * sizeof(double2));
  if (e == cudaSuccess && !T.perm.empty()) e = upload(*imem, T.perm.data(), T.perm.size() * sizeof(int));
  if (e != cudaSuccess) {
    cudaFree(*mem);
    cudaFree(*imem);
    *mem = nullptr;
    *imem = nullptr;
    return fail(kCudaError, std::string("DFT table upload: ") + cudaGetErrorString(e));
  }
  mm_plan_device(T, *mem, *imem, F);
  return kOk;
}

}  // namespace so3g
