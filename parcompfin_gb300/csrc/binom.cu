// Closed binomial sum (the reference's binom_embar) as a parallel reduction.
//
// Reference: binom() of src/binom_embar.cpp:5-50 (OpenMP src/binom_embar_omp.cpp:5-53,
// MPI k-range split src/binom_embar_mpi.cpp:38-57) with comb() of
// include/common.h:63-72:
//   price = e^{-rT} sum_{i < ceil(N/2)} [ e^{comb(N,i) + i lp + (N-i) lq} payoff(S0 u^i d^{N-i})
//                                       + e^{comb(N,i) + (N-i) lp + i lq} payoff(S0 u^{N-i} d^i) ]
//           (+ the middle term for even N), lp = log p, lq = log q.
// comb(N,i) is one FP64 accumulator: + log n for n = N..i+1, then - log j for
// j = 2..N-i. Its rounding drift (~1e-9 relative at N = 5e4) is part of the
// reference's result, so the default mode reproduces that chain exactly.
//
// mode 0 (reference order): every term inside the window is bit-identical
//   to the reference's, up to the last-ulp differences of the GPU's
//   exp/pow. The O(N) chain per term is replaced by an exact shortcut. While
//   the accumulator stays inside one binade [2^e, 2^{e+1}), every step
//   fl(acc +- log n) is an integer operation in units of that binade's ulp
//   u_e = 2^{e-52}: acc/u_e +- D_e[n], with D_e[n] = log n / u_e rounded to
//   nearest, ties excepted. A table of prefix sums of D_e per binade turns a
//   whole stretch of steps into one difference, found by binary search. The
//   steps that cross a binade or hit an exact tie (fraction exactly 1/2,
//   where round-to-even depends on the accumulator) are replayed as real
//   __dadd_rn / __dsub_rn. The integer stretches are exact by construction,
//   so the result equals the sequential chain bit for bit.
// mode 1 (accurate): log C(N,k) p^k q^{N-k} by Loader's saddle-point
//   formula (C. Loader, "Fast and Accurate Computation of Binomial
//   Probabilities", 2000: Stirling-series remainders plus bd0 deviance
//   terms), accurate to some 1e-15 + |k - N p| 2^-53 relative per term (N p
//   is rounded): prices of N = 2001 .. 50,001 with p = 0.36 .. 0.64 are within
//   4e-14 of 60-digit sums.
//
// Two kernels a batch (GB300, 1024 contracts of N = 1e3 .. 2e5, 2.6 million
// terms: 3.67 ms before, 0.28 ms now; accurate mode 4.6 -> 0.5 ms):
//   binom_prep_kernel  walks the additions of the contract's accumulator once
//            (they are the same for every term up to where it subtracts; a walk
//            per term was 85 % of the integer work) and takes the logarithms of
//            u, d and S0 (in the accurate mode p and 1 - p too) to 96 bits
//            after the point. Bound by the latency of its chain of loads, 48 us.
//   binom_kernel       one thread a pair of terms. The FP64 pipe is the scarce
//            unit of GB300 (19 cycles a warp instruction and SM against 0.25 for
//            the other pipes), so only the reference's own additions and
//            products run there, 20 a term; pow and exp are 64-bit fixed-point
//            powers of two (they were 650 of 700 FP64 operations), and tests
//            are made on the bits. 233 us, of which FP64 107 and issue 128.
//
// Only terms with k within 8 sqrt(N) of N p or N p' (p' = p u / R, the
// share-measure probability) are evaluated. By Chernoff's bound the weight
// outside is below 2 e^{-128} of S0 R^N + E.
//
// This translation unit is compiled with -fmad=false and the explicit
// __dadd_rn/__dmul_rn intrinsics, so no a*b+c is contracted into an FMA that
// the reference's x86-64 build does not perform.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <climits>
#include <vector>

#include "pcf_api_internal.h"
#include "pcf_device.cuh"

namespace pcf {

// The reference's lattice parameters, src/binom_embar.cpp:19-27 and
// src/binom_vanilla_eur.cpp:14-22 (this unit's host code is compiled with
// -ffp-contract=off, like the reference on x86-64).
void lattice(double r, double sigma, double T, int N, double& u, double& d, double& p,
             double& q, double& R) {
  const double dt = (double)T / (double)N;
  const double beta = 0.5 * (exp(-r * dt) + exp((r + pow(sigma, 2)) * dt));
  u = beta + sqrt(pow(beta, 2) - 1);
  d = beta - sqrt(pow(beta, 2) - 1);
  R = exp(r * dt);
  p = (R - d) / (u - d);
  q = 1 - p;
}

namespace {

constexpr int kEmin = -1;  // binades of the comb() accumulator with integer tables
constexpr int kEmax = 23;  // 2^24 > log(N!) for N <= 1e6
constexpr int kNbin = kEmax - kEmin + 1;
constexpr int kTieShift = 10;  // the tie index has an entry per 1024 places
constexpr int kBinomBlock = 256;
constexpr int kMaxN = 1000000;
constexpr double kWindow = 8.0;  // half-width of the term window, in sqrt(N)

struct BinomTables {
  const double* logt;               // logt[n] = log((double)n), n = 0..nmax
  const unsigned long long* pref;   // [kNbin][nmax+1] prefix sums of D_e (mod 2^64)
  const int* tie_idx;               // [kNbin][(nmax >> kTieShift) + 2]: see first_tie_ge
  const int* tie_pos;               // sorted tie positions of binade 0, 1, ..
  int nmax, tie_pitch;
};

struct BinomContract {
  double S0, E, u, d, lp, lq;
  double p, q;   // accurate mode
  double stirl_n, twopi_n;  // accurate mode: stirlerr(N), 2 pi / N
  int N, pf, i_lo, i_hi;  // pair indices i_lo..i_hi (inclusive)
  int has_mid, items, terms;
  int wide;      // a power of u or d may leave the FP64 range: binom_wide_kernel prices it
};

constexpr int kSegs = 20;  // stretches of the accumulator's first half kept per contract

// What binom_prep_kernel leaves for a contract's terms.
struct BinomPrep {
  // log2 of the share price at pair index i, S0 u^i d^(N-i), is y1 + i dy, and
  // of its mirror S0 u^(N-i) d^i is y2 - i dy: signed 128-bit numbers (high,
  // low word) with 96 bits after the point.
  unsigned long long y1[2], y2[2], dy[2];
  // Accurate mode: -|log(p / (1 - p))|, high and low part.
  double ratio[2];
  // The accumulator of comb() after + log N .. + log(n + 1) at the stretch
  // starts n = seg_n[0] (the largest index of the window) > seg_n[1] > ...
  int segs, cut;           // cut: more stretches than kSegs, the last one goes on
  double seg_acc[kSegs];
  int seg_n[kSegs];
};

struct BinomLaunch {
  const BinomContract* cs;
  const int* item_start;
  int ncontracts;
  double* partial;
  unsigned* tickets;
  double* out;
  int mode;
  const double* stirl;  // stirlerr(n), n = 0..15 (accurate mode)
  const unsigned long long* exp2t;  // 2^(-j/256) in units of 2^-63, j = 0..255
  BinomPrep* prep;
  int* item_contract;  // contract of each item, filled by binom_prep_kernel
  BinomTables t;
};

__device__ __forceinline__ int binade(double a) {
  return (int)((__double_as_longlong(a) >> 52) & 0x7ff) - 1023;
}
__device__ __forceinline__ long long to_units(double a) {
  return (__double_as_longlong(a) & 0xfffffffffffffLL) | (1LL << 52);
}
__device__ __forceinline__ double from_units(long long A, int e) {
  return __longlong_as_double(((long long)(e + 1023) << 52) | (A & 0xfffffffffffffLL));
}
// Most steps a stretch inside binade e can hold: every log n >= log 2.
__device__ __forceinline__ int stretch_cap(int e) {  // 1.4427 2^e + 2, in integers
  return (int)(0x5C550000u >> (30 - e)) + 3;
}

// The ties of binade b are tie_pos[idx[0] .. idx[last]), idx[k] being the first
// at or above k << kTieShift, so a search covers the ties among 1024 places:
// none or one from binade 13 on. (A binary search over the binade's whole list
// was half of the walk's instructions.)
__device__ __forceinline__ int last_tie_le(const BinomTables& T, int b, int n) {
  const int* idx = T.tie_idx + b * T.tie_pitch + (n >> kTieShift);
  const int first = T.tie_idx[b * T.tie_pitch];
  int lo = idx[0], hi = idx[1];  // first tie > n is in [lo, hi]
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (T.tie_pos[mid] <= n) lo = mid + 1; else hi = mid;
  }
  return lo > first ? T.tie_pos[lo - 1] : -1;
}
__device__ __forceinline__ int first_tie_ge(const BinomTables& T, int b, int j) {
  const int* idx = T.tie_idx + b * T.tie_pitch + (j >> kTieShift);
  const int end = T.tie_idx[(b + 1) * T.tie_pitch - 1];
  int lo = idx[0], hi = idx[1];  // first tie >= j is in [lo, hi]
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (T.tie_pos[mid] < j) lo = mid + 1; else hi = mid;
  }
  return lo < end ? T.tie_pos[lo] : INT_MAX;
}

__device__ __forceinline__ float lnf(float x) { return 0.693147181f * lg2_approx(x); }
// ln(m!) by Stirling's formula, in FP32.
__device__ __forceinline__ float ln_factorial(float m) {
  return m * lnf(m) - m + 0.5f * lnf(6.28318531f * m);
}
// The m with ln(m!) = g, in FP32 (Newton's method): within a place or two for
// m up to 10^6. It only picks where a search starts.
__device__ __forceinline__ float inverse_ln_factorial(float g) {
  g = fmaxf(g, 1.f);
  const float l = lnf(g + 3.f);
  float m = g / fmaxf(l - lnf(l), 0.5f) + 1.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) m = fmaxf(m - (ln_factorial(m) - g) / lnf(m + 1.f), 2.f);
  return m;
}
// A positive double's leading 24 bits as a float, on the integer pipe.
__device__ __forceinline__ float lead_float(double v) {
  const uint32_t h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
  return __uint_as_float((h << 3) - (896u << 23) + (l >> 29));
}
// An integer below 2^20 as a double, on the integer pipe.
__device__ __forceinline__ double small_to_double(int i) {
  if (i == 0) return 0.0;
  const int e = 31 - __clz(i);
  return __hiloint2double(((1023 + e) << 20) + ((i << (20 - e)) & 0xfffff), 0);
}

// acc + log(hi) + log(hi-1) + ... + log(lo+1), each step rounded, in that order.
__device__ double add_chain_desc(const BinomTables& T, double acc, int hi, int lo) {
  int n = hi;
  const long long LIM = (1LL << 53) - 1;
  while (n > lo) {
    if (acc == 0.0) { acc = T.logt[n]; --n; continue; }
    const int e = binade(acc);
    if (e >= kEmin && e <= kEmax) {
      const int b = e - kEmin;
      const unsigned long long* P = T.pref + (size_t)b * (T.nmax + 1);
      long long A = to_units(acc);
      int mlo = max(lo + 1, n - stretch_cap(e) + 1);
      const int t = last_tie_le(T, b, n);
      if (t >= mlo) mlo = t + 1;
      if (mlo <= n && A + (long long)(P[n] - P[n - 1]) <= LIM) {
        int a = mlo, z = n;  // smallest m in [a, z] with A + sum(m..n) <= LIM
        while (a < z) {
          const int mid = (a + z) >> 1;
          if (A + (long long)(P[n] - P[mid - 1]) <= LIM) z = mid; else a = mid + 1;
        }
        A += (long long)(P[n] - P[a - 1]);
        acc = from_units(A, e);
        n = a - 1;
      }
    }
    if (n > lo) { acc = __dadd_rn(acc, T.logt[n]); --n; }
  }
  return acc;
}

// acc - log(2) - log(3) - ... - log(hi), each step rounded, in that order. The
// end of a stretch is looked for around the place where ln(m!) has brought the
// accumulator down to its binade's floor: three to five loads of one line
// instead of a binary search's 16 spread ones.
__device__ double sub_chain_asc(const BinomTables& T, double acc, int hi) {
  int j = 2;
  const long long FLOOR = (1LL << 52) + 1;
  const float top = lead_float(acc);
  while (j <= hi) {
    if (__double_as_longlong(acc) > 0) {  // acc > 0, off the FP64 pipe
      const int e = binade(acc);
      if (e >= kEmin && e <= kEmax) {
        const int b = e - kEmin;
        const unsigned long long* P = T.pref + (size_t)b * (T.nmax + 1);
        int mhi = (int)min((long long)hi, (long long)j + stretch_cap(e) - 1);
        const int t = first_tie_ge(T, b, j);
        if (t <= mhi) mhi = t - 1;
        const long long A = to_units(acc);
        const unsigned long long before = P[j - 1];
        // A - sum(j..m) >= FLOOR
        const unsigned long long room = (unsigned long long)(A - FLOOR) + before;
        if (mhi >= j && (long long)(room - P[j]) >= 0) {
          int a = mhi;  // largest m in [j, mhi] that fits
          if ((long long)(room - P[mhi]) < 0) {
            a = j;
            int z = mhi - 1;
            const int m0 = (int)inverse_ln_factorial(
                top - __uint_as_float((uint32_t)(127 + e) << 23));  // top - 2^e
            const int lo = min(max(m0 - 1, j), z), up = min(max(m0 + 2, j), z);
            if ((long long)(room - P[lo]) >= 0) {
              a = lo;
              if ((long long)(room - P[up + 1]) >= 0) a = up + 1;
              else z = up;
            } else {
              z = lo - 1;
            }
            while (a < z) {
              const int mid = (a + z + 1) >> 1;
              if ((long long)(room - P[mid]) >= 0) a = mid; else z = mid - 1;
            }
          }
          acc = from_units(A - (long long)(P[a] - before), e);
          j = a + 1;
        }
      }
    }
    if (j <= hi) { acc = __dsub_rn(acc, T.logt[j]); ++j; }
  }
  return acc;
}

// include/common.h:63-72, evaluated exactly.
__device__ double comb_ref(const BinomTables& T, int N, int i) {
  if (i == 0 || i == N) return 0.0;
  if (i == 1 || i == N - 1) return T.logt[N];
  const double acc = add_chain_desc(T, 0.0, N, i);
  return sub_chain_asc(T, acc, N - i);
}

__device__ __forceinline__ double payoff_d(double S, double E, int pf) {
  return fmax(__dmul_rn((double)pf, __dsub_rn(S, E)), 0.0);
}

// ---- Loader's saddle-point terms (accurate mode) ----
__host__ __device__ inline double stirlerr_series(double n) {  // n > 15
  const double S0 = 1.0 / 12, S1 = 1.0 / 360, S2 = 1.0 / 1260, S3 = 1.0 / 1680, S4 = 1.0 / 1188;
  const double nn = n * n;
  if (n > 500) return (S0 - S1 / nn) / n;
  if (n > 80) return (S0 - (S1 - S2 / nn) / nn) / n;
  if (n > 35) return (S0 - (S1 - (S2 - S3 / nn) / nn) / nn) / n;
  return (S0 - (S1 - (S2 - (S3 - S4 / nn) / nn) / nn) / nn) / n;
}

__device__ double stirlerr(double n, const double* tab) {
  return n <= 15.0 ? tab[(int)n] : stirlerr_series(n);
}

// bd0(x, np) = x log(x / np) + np - x, with the series for x near np.
__device__ double bd0(double x, double np) {
  if (fabs(x - np) < 0.1 * (x + np)) {
    const double v = (x - np) / (x + np);
    double s = (x - np) * v;
    double ej = 2 * x * v;
    const double v2 = v * v;
    for (int j = 1; j < 1000; ++j) {
      ej *= v2;
      const double s1 = s + ej / (2 * j + 1);
      if (s1 == s) return s1;
      s = s1;
    }
    return s;
  }
  return x * log(x / np) + np - x;
}

__device__ double log_dbinom(int k, int N, double p, double q, const double* stirl) {
  if (k == 0) return N * log1p(-p);
  if (k == N) return N * log(p);
  const double lc = stirlerr((double)N, stirl) - stirlerr((double)k, stirl) -
                    stirlerr((double)(N - k), stirl) - bd0((double)k, N * p) -
                    bd0((double)(N - k), N * q);
  const double lf = 1.8378770664093454836 + log((double)k) + log1p(-(double)k / N);  // log(2 pi k (N-k)/N)
  return lc - 0.5 * lf;
}

// src/binom_embar.cpp:35-40: the terms of pair index i in the reference's order.
__device__ double pair_terms(const BinomLaunch& L, const BinomContract& C, int i) {
  const int N = C.N;
  double t1, t2;
  if (L.mode == 0) {
    const double cv = comb_ref(L.t, N, i);
    const double b1 = __dadd_rn(__dadd_rn(cv, __dmul_rn((double)i, C.lp)),
                                __dmul_rn((double)(N - i), C.lq));
    const double b2 = __dadd_rn(__dadd_rn(cv, __dmul_rn((double)(N - i), C.lp)),
                                __dmul_rn((double)i, C.lq));
    t1 = exp(b1);
    t2 = exp(b2);
  } else {
    t1 = exp(log_dbinom(i, N, C.p, C.q, L.stirl));
    t2 = exp(log_dbinom(N - i, N, C.p, C.q, L.stirl));
  }
  const double s1 = __dmul_rn(__dmul_rn(C.S0, pow(C.u, (double)i)), pow(C.d, (double)(N - i)));
  const double s2 = __dmul_rn(__dmul_rn(C.S0, pow(C.u, (double)(N - i))), pow(C.d, (double)i));
  return __dadd_rn(__dmul_rn(t1, payoff_d(s1, C.E, C.pf)), __dmul_rn(t2, payoff_d(s2, C.E, C.pf)));
}

// src/binom_embar.cpp:42-45: the middle term of an even N.
__device__ double mid_term(const BinomLaunch& L, const BinomContract& C) {
  const int N = C.N, h = N / 2;
  double w;
  if (L.mode == 0) {
    const double cv = comb_ref(L.t, N, h);
    w = exp(__dadd_rn(__dadd_rn(cv, __dmul_rn((double)h, C.lp)), __dmul_rn((double)h, C.lq)));
  } else {
    w = exp(log_dbinom(h, N, C.p, C.q, L.stirl));
  }
  const double s = __dmul_rn(__dmul_rn(C.S0, pow(C.u, (double)h)), pow(C.d, (double)h));
  return __dmul_rn(w, payoff_d(s, C.E, C.pf));
}

// log_dbinom(k, N, p, q) for the fixed-point kernel, with stirlerr(N) given and
// the divisions shared: an IEEE division costs nine FP64 operations. The two
// deviance divisions stay, as their error is the weight's.
__device__ __forceinline__ double stirlerr_inv(int n, double r, const double* tab) {
  if (n <= 15) return tab[n];
  const double S0 = 1.0 / 12, S1 = 1.0 / 360, S2 = 1.0 / 1260, S3 = 1.0 / 1680, S4 = 1.0 / 1188;
  const double rr = r * r;
  if (n > 500) return __fma_rn(-S1, rr, S0) * r;
  double h = __fma_rn(-S4, rr, S3);
  h = __fma_rn(-h, rr, S2);
  h = __fma_rn(-h, rr, S1);
  return __fma_rn(-h, rr, S0) * r;
}

// bd0(x, np) where x is near np: (x - np) v + 2 x v sum_{j>=1} v^{2j}/(2j+1)
// with v = (x - np)/(x + np), |v| < 0.1; 5 terms reach 2^-60 for v^2 < 1/1024.
__device__ __forceinline__ double bd0_near(double x, double np) {
  const double d = __dsub_rn(x, np), v = __ddiv_rn(d, __dadd_rn(x, np));
  const double vv = v * v;
  double h = 0.0;
  if (__double2hiint(vv) >= 0x3F500000) {  // v^2 >= 2^-10
    h = 1.0 / 23;
    h = __fma_rn(h, vv, 1.0 / 21);
    h = __fma_rn(h, vv, 1.0 / 19);
    h = __fma_rn(h, vv, 1.0 / 17);
    h = __fma_rn(h, vv, 1.0 / 15);
    h = __fma_rn(h, vv, 1.0 / 13);
    h = h * vv;
  }
  h = h + 1.0 / 11;
  h = __fma_rn(h, vv, 1.0 / 9);
  h = __fma_rn(h, vv, 1.0 / 7);
  h = __fma_rn(h, vv, 1.0 / 5);
  h = __fma_rn(h, vv, 1.0 / 3);
  return __fma_rn(d, v, (2.0 * x * v) * (vv * h));
}

__device__ double log_dbinom_shared(int k, const BinomContract& C, double stirl_N,
                                    const double* stirl) {
  const int N = C.N;
  const double x = small_to_double(k), y = small_to_double(N - k), n = small_to_double(N);
  const double np = n * C.p, nq = n * C.q;
  // |x - np| < 0.1 (x + np) for both, tested in FP32 with room to spare
  const float fx = (float)k, fp = lead_float(np), fy = (float)(N - k), fq = lead_float(nq);
  if (k == 0 || k == N || fabsf(fx - fp) > 0.099f * (fx + fp) ||
      fabsf(fy - fq) > 0.099f * (fy + fq))
    return log_dbinom(k, N, C.p, C.q, stirl);
  const double xy = x * y, inv = __ddiv_rn(1.0, xy);
  const double lc = stirl_N - stirlerr_inv(k, y * inv, stirl) - stirlerr_inv(N - k, x * inv, stirl) -
                    bd0_near(x, np) - bd0_near(y, nq);
  return __fma_rn(-0.5, log(xy * C.twopi_n), lc);  // 2 pi k (N-k)/N
}

// One block's contract and its first term; false if it is not this kernel's.
__device__ __forceinline__ bool binom_item(const BinomLaunch& L, bool wide, int& c, int& j) {
  c = L.item_contract[blockIdx.x];
  j = blockIdx.x - L.item_start[c];
  return (L.cs[c].wide != 0) == wide;
}

// Terms whose powers may leave the FP64 range, as the reference evaluates
// them (pow and exp in FP64).
__global__ void __launch_bounds__(kBinomBlock) binom_wide_kernel(BinomLaunch L) {
  __shared__ double sh[32];
  int c, j;
  if (!binom_item(L, true, c, j)) return;
  const BinomContract C = L.cs[c];
  const int ti = j * kBinomBlock + threadIdx.x;
  double v = 0.0;
  if (ti < C.terms) {
    const int i = C.i_lo + ti;
    if (i <= C.i_hi) v = pair_terms(L, C, i);
    else if (C.has_mid) v = mid_term(L, C);
  }
  double vv[1] = {v}, tot[1];
  block_sum<1>(vv, sh, tot);
  grid_finalize<1>(tot, L.partial + L.item_start[c], L.tickets + c, L.out + c, C.items, j);
}

// ---- powers and exponentials in 64-bit fixed point ----
//
// GB300's FP64 pipe takes 19 cycles per warp instruction and SM; a 64-bit
// high product on the integer pipe takes 4.8. pow and exp in FP64 were about
// 650 of a term's 700 FP64 operations and the kernel's bound, so both are
// evaluated as powers of two in fixed point, to 2^-57 relative, and only the
// reference's own additions and products remain in FP64. (A power's exponent has
// 64 bits after the point; an exponential's, |b| log2(e), has 62 - e for |b| in
// [2^e, 2^(e+1)): 2^-57 relative up to |b| = 64, 2^-53 at the smallest weights
// that are not 0, |b| = 690.)

// 2^-f for a fraction f in units of 2^-64, in units of 2^-63. With f = j/256 + r
// and x = r ln 2 < 2^-8.5: 2^-f = T[j] (1 - c), c = 1 - e^-x = x (1 - h),
// h = x/2 - x^2 (1/6 - x/24 + x^2/120); x^6/720 < 2^-60 is dropped.
__device__ __forceinline__ unsigned long long exp2_neg(unsigned long long f,
                                                       const unsigned long long* T) {
  const unsigned long long t = T[f >> 56];
  const unsigned long long x = __umul64hi(f << 8, 0xB17217F7D1CF79ACULL);  // x 2^72 (ln 2 2^64)
  const uint32_t x40 = (uint32_t)(x >> 32);                                // x 2^40
  const uint32_t xx = __umulhi(x40, x40);                                  // x^2 2^48
  const uint32_t w = 715827883u - __umulhi(x40, 699051u) + __umulhi(xx, 546u);  // (1/6 - ..) 2^32
  const unsigned long long h = (x >> 1) - (((unsigned long long)xx * w) >> 8);  // h 2^72
  const unsigned long long c = x - __umul64hi(x, h >> 8);                       // c 2^72
  return t - (__umul64hi(t, c) >> 8);
}

// m 2^(-63 + k) as a double, rounded to nearest (m in [2^62, 2^63]; the
// exponent stays in the normal range).
__device__ __forceinline__ double fixed_to_double(unsigned long long m, int k) {
  const int lz = (int)((m >> 63) ^ 1);  // 1, or 0 for m = 2^63
  const unsigned long long r = ((m << lz) + 1024u) >> 11;  // 53 bits (2^53 carries over)
  return __longlong_as_double((long long)(((unsigned long long)(1023 + k - lz - 1) << 52) + r));
}

// e^b for b <= 0 (a logarithm of a weight; e^b < 1e-300 is 0).
__device__ __forceinline__ double exp_weight(double b, const unsigned long long* T) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(b);
  if (bits <= 1ULL << 63) return exp(b);  // b >= 0: a weight of nearly 1
  const int e = (int)((bits >> 52) & 0x7ff) - 1023;
  if (e < -55) return 1.0;
  if (bits >= 0xC085900000000000ULL) return 0.0;  // b <= -690 (and NaN)
  // |b| log2(e) = hi 2^(e - 62)
  const unsigned long long hi = __umul64hi((bits << 11) | (1ULL << 63), 0xB8AA3B295C17F0BCULL);
  const int k = e >= -1 ? (int)(hi >> (62 - e)) : 0;
  const unsigned long long f = e >= -2 ? hi << (2 + e) : hi >> (-2 - e);
  return fixed_to_double(exp2_neg(f, T), -k);
}

__device__ __forceinline__ unsigned __int128 u128(const unsigned long long (&w)[2]) {
  return ((unsigned __int128)w[0] << 64) | w[1];
}

// 2^y for y in units of 2^-96.
__device__ __forceinline__ double exp2_q96(unsigned __int128 y, const unsigned long long* T) {
  const unsigned long long f = (unsigned long long)(y >> 32);
  const int k = (int)(y >> 96);
  // 2^(k + f) = 2^(k + 1) 2^-(1 - f)
  return fixed_to_double(exp2_neg(0ULL - f, T), f ? k + 1 : k);
}

// log2 x in units of 2^-96, to about 2^-100: x = 2^k m, ln m = 2 atanh z with
// z = (m - 1)/(m + 1) in double-double arithmetic; the series beyond z^3/3 in
// FP64, which its weight z^4 allows.
__device__ __int128 log2_q96(double x) {
  long long bits = __double_as_longlong(x);
  int k = (int)(bits >> 52) - 1023;
  double m = __longlong_as_double((bits & 0xfffffffffffffLL) | (1023LL << 52));
  if (m > 1.4142135623730951) {
    m *= 0.5;
    k += 1;
  }
  const double a = m - 1.0;  // exact
  const double bh = m + 1.0, bl = m - (bh - 1.0);
  const double zh = __ddiv_rn(a, bh);
  const double zl = __ddiv_rn(__fma_rn(-zh, bl, __fma_rn(-zh, bh, a)), bh);
  const double wh = zh * zh, wl = __fma_rn(zh, zh, -wh) + 2.0 * zh * zl;
  double q = 1.0 / 29;
#pragma unroll 1
  for (int d = 27; d >= 5; d -= 2) q = __fma_rn(q, wh, __ddiv_rn(1.0, (double)d));
  // p = 1/3 + w q
  const double t = wh * q, tl = __fma_rn(wh, q, -t) + wl * q;
  const double third = 0.33333333333333331, third_l = 1.850371707708594e-17;
  const double ph = third + t, pl = (third - ph) + t + (tl + third_l);
  // u = z w p
  const double ah = wh * ph, al = __fma_rn(wh, ph, -ah) + (wh * pl + wl * ph);
  const double uh = zh * ah, ul = __fma_rn(zh, ah, -uh) + (zh * al + zl * ah);
  const double sh = zh + uh, sl = (zh - sh) + uh + (zl + ul);
  // times 2 log2(e)
  const double ch = 2.8853900817779268, cl = 4.0710547481862066e-17;
  const double gh = sh * ch, gl = __fma_rn(sh, ch, -gh) + (sh * cl + sl * ch);
  auto q96 = [](double v) -> __int128 {
    const long long vb = __double_as_longlong(v);
    const int e = (int)((vb >> 52) & 0x7ff) - 1023;
    if (e < -150) return 0;
    const __int128 mant = (vb & 0xfffffffffffffLL) | (1LL << 52);
    const int sft = e + 44;  // mantissa 2^(e - 52), times 2^96
    const __int128 r = sft >= 0 ? mant << sft : mant >> -sft;
    return vb < 0 ? -r : r;
  };
  return ((__int128)k << 96) + q96(gh) + q96(gl);
}

// add_chain_desc by a warp, whose lanes all hold the same state: adds log(n), log(n-1), ..., log(lo+1) to acc; if rec is not NULL, records the
// state (n, acc) at the start of every stretch there. `total` is ln(N!) in
// FP32, N being where the chain began with acc = 0.
__device__ void add_chain_warp(const BinomTables& T, double& acc, int& n, int lo, float total,
                               BinomPrep* rec) {
  const int lane = threadIdx.x & 31;
  const long long LIM = (1LL << 53) - 1;
  int segs = 0;
  if (!rec && n - 32 >= lo) {  // the first 32 steps fill the low binades one by one
    const double lg = T.logt[n - lane];
    for (int k = 0; k < 32; ++k) {
      const double x = __shfl_sync(0xffffffffu, lg, k);
      acc = k == 0 ? x : __dadd_rn(acc, x);
    }
    n -= 32;
  }
  for (;;) {
    if (rec) {
      if (segs == kSegs) {
        if (lane == 0) rec->cut = 1;
        break;
      }
      if (lane == 0) {
        rec->seg_n[segs] = n;
        rec->seg_acc[segs] = acc;
      }
      ++segs;
    }
    if (n <= lo) break;
    if (acc != 0.0) {
      const int e = binade(acc);
      if (e >= kEmin && e <= kEmax) {
        const int b = e - kEmin;
        const unsigned long long* P = T.pref + (size_t)b * (T.nmax + 1);
        const unsigned long long Pn = P[n], Pn1 = P[n - 1];
        const long long A = to_units(acc);
        // ln((m-1)!) = ln(N!) - 2^(e+1) at the end of the stretch. The 32
        // places around it are loaded with everything else the iteration
        // needs, so that it waits for memory twice (the ties need two).
        const int m0 = (int)inverse_ln_factorial(
            total - __uint_as_float((uint32_t)(128 + e) << 23)) + 1;
        const int base = min(max(m0 - 16, lo + 1), n), wm = min(base + lane, n);
        const unsigned long long Pw = P[wm - 1];
        const double lw = T.logt[wm - 1];
        int mlo = max(lo + 1, n - stretch_cap(e) + 1);
        const int t = last_tie_le(T, b, n);
        if (t >= mlo) mlo = t + 1;
        if (mlo <= n && A + (long long)(Pn - Pn1) <= LIM) {
          int a = mlo, z = n;  // smallest m in [a, z] with A + sum(m..n) <= LIM
          unsigned ok = __ballot_sync(0xffffffffu,
                                      base + lane >= z || A + (long long)(Pn - Pw) <= LIM);
          int f = ok ? __ffs(ok) - 1 : 32;  // lanes below f do not fit
          if (f < 32) z = max(min(z, base + f), a);
          if (f > 0) a = max(a, min(base + f, z));
          while (a < z) {
            const int step = (z - a + 31) >> 5, m = a + lane * step;
            ok = __ballot_sync(0xffffffffu,
                               m >= z || A + (long long)(Pn - P[m - 1]) <= LIM);
            f = ok ? __ffs(ok) - 1 : 32;
            const int a0 = a;
            if (f < 32) z = min(z, a0 + f * step);
            if (f > 0) a = min(a0 + (f - 1) * step + 1, z);
          }
          const int in = a - base;  // place a in the window
          const double lg = __shfl_sync(0xffffffffu, lw, in & 31);
          const unsigned long long Pi = __shfl_sync(0xffffffffu, Pw, in & 31);
          const bool inside = in >= 0 && in < 32;
          acc = from_units(A + (long long)(Pn - (inside ? Pi : P[a - 1])), e);
          n = a - 1;
          if (n <= lo) break;
          acc = __dadd_rn(acc, inside ? lg : T.logt[n]);
          --n;
          continue;
        }
      }
    }
    acc = acc == 0.0 ? T.logt[n] : __dadd_rn(acc, T.logt[n]);
    --n;
  }
  if (rec && lane == 0) rec->segs = segs;
}

// Two warps a contract. The first takes the logarithms of u, d and S0, names the
// contract of its items and clears its ticket; the second walks the comb() accumulator's
// additions from N down through the window. The additions are the same for
// every term up to where it starts to subtract, so they are walked once; a
// term then needs one difference.
constexpr int kPrepBlock = 128;
__global__ void __launch_bounds__(kPrepBlock) binom_prep_kernel(BinomLaunch L) {
  const int c = blockIdx.x * (kPrepBlock / 64) + (threadIdx.x >> 6), lane = threadIdx.x & 31;
  if (c >= L.ncontracts) return;
  const BinomContract& C = L.cs[c];
  BinomPrep* R = L.prep + c;
  if (threadIdx.x & 32) {
    if (C.wide || L.mode != 0) return;
    if (lane == 0) R->cut = 0;
    __syncwarp();
    double acc = 0.0;
    int n = C.N;
    const float total = ln_factorial((float)C.N);
    const int top = C.has_mid ? C.N / 2 : C.i_hi;
    add_chain_warp(L.t, acc, n, top, total, nullptr);
    add_chain_warp(L.t, acc, n, C.i_lo, total, R);
    return;
  }
  for (int k = lane; k < C.items; k += 32) L.item_contract[L.item_start[c] + k] = c;
  if (lane == 0) L.tickets[c] = 0u;
  if (C.wide) return;
  // (lanes 3 and 4 for the accurate mode)
  const double arg = lane == 0 ? C.u : lane == 1 ? C.d : lane == 2 ? C.S0 : lane == 3 ? C.p : C.q;
  const __int128 g = lane < (L.mode ? 5 : 3) ? log2_q96(arg) : 0;
  unsigned long long gh = (unsigned long long)(g >> 64), gl = (unsigned long long)g;
  auto from = [&](int src) {
    const unsigned long long h = __shfl_sync(0xffffffffu, gh, src);
    const unsigned long long l = __shfl_sync(0xffffffffu, gl, src);
    return (__int128)(((unsigned __int128)h << 64) | l);
  };
  const __int128 lu = from(0), ld = from(1), ls = from(2), lp = from(3), lq = from(4);
  if (lane == 0) {
    auto put = [](unsigned long long (&w)[2], __int128 v) {
      w[0] = (unsigned long long)(v >> 64);
      w[1] = (unsigned long long)v;
    };
    put(R->y1, ls + C.N * ld);
    put(R->y2, ls + C.N * lu);
    put(R->dy, lu - ld);
    if (L.mode) {
      // |log2(p/q)| ln 2, still in units of 2^-96, as a sum of two doubles. q is
      // 1 - p rounded: log(1 - p) = log q + (1 - q - p)/q.
      const unsigned __int128 a = lp > lq ? lp - lq : lq - lp;
      const unsigned long long ln2 = 0xB17217F7D1CF79ACULL;  // ln 2 2^64
      const unsigned __int128 v = (a >> 64) * ln2 + __umul64hi((unsigned long long)a, ln2);
      const double hi = (double)(long long)(v >> 46);  // below 2^60
      const long long lo = (long long)((__int128)v - ((__int128)(long long)hi << 46));
      const double dq = __ddiv_rn(__dsub_rn(__dsub_rn(1.0, C.q), C.p), C.q);
      R->ratio[0] = -hi * 0x1p-50;
      R->ratio[1] = -((double)lo * 0x1p-96) + (lp > lq ? dq : -dq);
    }
  }
}

// comb(N, i) from the contract's recorded stretches.
__device__ double comb_from(const BinomTables& T, int N, int i, const BinomPrep& R) {
  if (i == 0 || i == N) return 0.0;
  if (i == 1 || i == N - 1) return T.logt[N];
  int s = 0;
  while (s + 1 < R.segs && R.seg_n[s + 1] >= i) ++s;
  double acc = R.seg_acc[s];
  const int n = R.seg_n[s];
  if (n > i) {
    if (R.cut && s + 1 == R.segs) {
      acc = add_chain_desc(T, acc, n, i);
    } else {
      const int e = binade(acc);
      const unsigned long long* P = T.pref + (size_t)(e - kEmin) * (T.nmax + 1);
      acc = from_units(to_units(acc) + (long long)(P[n] - P[i]), e);
    }
  }
  return sub_chain_asc(T, acc, N - i);
}

// max(pf (S - E), 0); the sign and the comparison on the bits, off the FP64 pipe.
__device__ __forceinline__ double payoff_bits(double S, double E, int pf) {
  const long long a = __double_as_longlong(__dsub_rn(S, E)) ^
                      (pf < 0 ? (long long)0x8000000000000000ULL : 0LL);
  return __longlong_as_double(a < 0 ? 0LL : a);
}

// src/binom_embar.cpp:35-45: pair index i's terms in the reference's order
// (the middle term of an even N is its one term).
__global__ void __launch_bounds__(kBinomBlock) binom_kernel(BinomLaunch L) {
  __shared__ double sh[kBinomBlock];
  __shared__ unsigned long long T[256];
  __shared__ BinomPrep R;
  int c, j;
  if (!binom_item(L, false, c, j)) return;
  for (int k = threadIdx.x; k < 256; k += kBinomBlock) T[k] = L.exp2t[k];
  for (int k = threadIdx.x; k < (int)(sizeof(BinomPrep) / 4); k += kBinomBlock)
    ((int*)&R)[k] = ((const int*)(L.prep + c))[k];
  __syncthreads();
  const BinomContract& C = L.cs[c];
  const int ti = j * kBinomBlock + threadIdx.x;
  double v = 0.0;
  if (ti < C.terms) {
    const int N = C.N;
    const bool mid = C.i_lo + ti > C.i_hi;
    const int i = mid ? N / 2 : C.i_lo + ti;
    double b1, b2;
    if (L.mode == 0) {
      const double cv = comb_from(L.t, N, i, R);
      const double di = small_to_double(i), dj = small_to_double(N - i);
      b1 = __dadd_rn(__dadd_rn(cv, __dmul_rn(di, C.lp)), __dmul_rn(dj, C.lq));
      b2 = __dadd_rn(__dadd_rn(cv, __dmul_rn(dj, C.lp)), __dmul_rn(di, C.lq));
    } else {
      // The larger weight of the pair by its own logarithm, the smaller one from
      // it: their ratio is ((1-p)/p)^(N-2i) where p > 1/2. Both terms of the sum
      // are negative, so it is as good as the smaller weight's own logarithm; the
      // larger one from the smaller would carry the smaller's absolute error
      // (1e-12 of the price at N = 50,001 and p = 0.64).
      const bool up = __double_as_longlong(C.p) > __double_as_longlong(C.q);
      const double b = log_dbinom_shared(up ? N - i : i, C, C.stirl_n, L.stirl);
      const double n2 = small_to_double(N - 2 * i);
      const double m = __fma_rn(n2, R.ratio[1], __fma_rn(n2, R.ratio[0], b));
      b1 = up ? m : b;
      b2 = up ? b : m;
    }
    const unsigned __int128 iy = u128(R.dy) * (unsigned)i;
    const double s1 = exp2_q96(u128(R.y1) + iy, T), s2 = exp2_q96(u128(R.y2) - iy, T);
    v = __dmul_rn(exp_weight(b1, T), payoff_bits(s1, C.E, C.pf));
    if (!mid) v = __dadd_rn(v, __dmul_rn(exp_weight(b2, T), payoff_bits(s2, C.E, C.pf)));
  }
  // One warp adds the block's terms: 12 FP64 additions a block instead of the
  // shuffle tree's 45.
  sh[threadIdx.x] = v;
  __syncthreads();
  double tot[1] = {0.0};
  if (threadIdx.x < 32) {
    double x = sh[threadIdx.x];
    for (int k = 32; k < kBinomBlock; k += 32) x = __dadd_rn(x, sh[threadIdx.x + k]);
    tot[0] = warp_sum(x);
  }
  grid_finalize<1>(tot, L.partial + L.item_start[c], L.tickets + c, L.out + c, C.items, j);
}

// ---- host side ----

struct HostTables {
  std::vector<double> logt;
  std::vector<unsigned long long> pref;
  std::vector<int> tie_idx, tie_pos;
};
int tie_pitch(int nmax) { return (nmax >> kTieShift) + 2; }

// D_e[n] = round-half-away... of log n / u_e: floor plus [frac > 1/2], with
// frac == 1/2 recorded as a tie. Exact: log n * 2^{52-e} is a power-of-two
// scaling of a double, so floor and fraction are exact.
void build_tables(int nmax, HostTables& H) {
  H.logt.resize((size_t)nmax + 1);
  H.logt[0] = -INFINITY;
  for (int n = 1; n <= nmax; ++n) H.logt[n] = log((double)n);
  H.pref.assign((size_t)kNbin * (nmax + 1), 0ULL);
  const int pitch = tie_pitch(nmax);
  H.tie_idx.assign((size_t)kNbin * pitch, 0);
  H.tie_pos.clear();
  for (int b = 0; b < kNbin; ++b) {
    const int e = b + kEmin;
    unsigned long long run = 0;
    unsigned long long* P = &H.pref[(size_t)b * (nmax + 1)];
    P[0] = 0;
    int* idx = &H.tie_idx[(size_t)b * pitch];
    idx[0] = (int)H.tie_pos.size();
    for (int n = 1; n <= nmax; ++n) {
      if ((n & ((1 << kTieShift) - 1)) == 0) idx[n >> kTieShift] = (int)H.tie_pos.size();
      const double x = ldexp(H.logt[n], 52 - e);
      const double F = floor(x);
      const double f = x - F;
      unsigned long long D = (unsigned long long)F;
      if (f > 0.5) D += 1;
      else if (f == 0.5) H.tie_pos.push_back(n);
      run += D;
      P[n] = run;
    }
    idx[pitch - 1] = (int)H.tie_pos.size();
  }
}

// stirlerr(n) = log(n!) - (n + 1/2) log n + n - log(sqrt(2 pi)), n = 1..15, in
// long double; stirlerr(0) is unused (k = 0 has its own formula).
void stirlerr_table(double* out) {
  out[0] = 0.0;
  for (int n = 1; n <= 15; ++n) {
    const long double ln = (long double)n;
    out[n] = (double)(lgammal(ln + 1) - (ln + 0.5L) * logl(ln) + ln -
                      0.5L * logl(2 * 3.14159265358979323846264338327950288L));
  }
}

size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

int ensure_tables(pcf_ctx* c, int nmax) {
  if (c->d_logtab && c->logtab_n >= nmax) return PCF_OK;
  // Grown by doubling from 4096 entries: a one-off small N builds a small
  // table (its build is ~0.1 microsecond per entry and binade), a sequence
  // of growing N rebuilds it a logarithmic number of times.
  int want = 4096;
  while (want < nmax && want < kMaxN) want *= 2;
  want = std::min(std::max(want, nmax), kMaxN);
  HostTables H;
  build_tables(want, H);
  const size_t b_log = sizeof(double) * (want + 1);
  const size_t b_pref = sizeof(unsigned long long) * H.pref.size();
  const size_t b_off = sizeof(int) * H.tie_idx.size();
  const size_t b_pos = sizeof(int) * std::max<size_t>(1, H.tie_pos.size());
  const size_t o_pref = a256(b_log), o_off = a256(o_pref + b_pref), o_pos = a256(o_off + b_off);
  const size_t o_stir = a256(o_pos + b_pos);
  const size_t o_exp2 = a256(o_stir + 16 * sizeof(double));
  const size_t total = a256(o_exp2 + 256 * sizeof(unsigned long long));
  if (c->d_logtab) cudaFree(c->d_logtab);
  c->d_logtab = nullptr;
  c->logtab_n = 0;
  if (c->budget_bytes && total > c->budget_bytes)
    return set_error(PCF_ENOMEM, "binomial tables of %zu bytes exceed the context budget", total);
  void* d = nullptr;
  int st = cuda_status(cudaMalloc(&d, total), "cudaMalloc(binomial tables)");
  if (st) return st;
  std::vector<char> h(total, 0);
  memcpy(&h[0], H.logt.data(), b_log);
  memcpy(&h[o_pref], H.pref.data(), b_pref);
  memcpy(&h[o_off], H.tie_idx.data(), b_off);
  if (!H.tie_pos.empty()) memcpy(&h[o_pos], H.tie_pos.data(), sizeof(int) * H.tie_pos.size());
  stirlerr_table((double*)&h[o_stir]);
  for (int j = 0; j < 256; ++j)  // 2^(-j/256) in units of 2^-63
    ((unsigned long long*)&h[o_exp2])[j] =
        (unsigned long long)roundl(ldexpl(exp2l(-(long double)j / 256), 63));
  // On the context's stream and waited for: a copy from pageable memory on the
  // default stream may still be on its way when the call returns, and nothing
  // orders it before this stream's launches.
  st = cuda_status(cudaMemcpyAsync(d, h.data(), total, cudaMemcpyHostToDevice, c->stream),
                   "H2D binomial tables");
  const int landed = cuda_status(cudaStreamSynchronize(c->stream), "H2D binomial tables");
  if (!st) st = landed;
  if (st) {
    cudaFree(d);
    return st;
  }
  c->d_logtab = (double*)d;
  c->logtab_n = want;
  c->binom_off[0] = o_pref;
  c->binom_off[1] = o_off;
  c->binom_off[2] = o_pos;
  c->binom_off[3] = o_stir;
  c->binom_off[4] = o_exp2;
  return PCF_OK;
}

int setup_contract(const pcf_binom_contract& k, int idx, BinomContract& C) {
  const int pf = k.payoff_fun;
  if (pf != 1 && pf != -1)
    return set_error(PCF_EINVAL, "contract %d: Unknown payoff function", idx);
  if (!(k.S0 > 0) || !(k.E >= 0) || !(k.sigma > 0) || !(k.T > 0) || !std::isfinite(k.r) ||
      !std::isfinite(k.S0) || !std::isfinite(k.E) || !std::isfinite(k.sigma) ||
      !std::isfinite(k.T))
    return set_error(PCF_EINVAL, "contract %d: need S0 > 0, E >= 0, sigma > 0, T > 0", idx);
  if (k.N < 1 || k.N > kMaxN)
    return set_error(PCF_EINVAL, "contract %d: N must be in [1, %d]", idx, kMaxN);
  const int N = k.N;
  double u, d, p, q, R;
  lattice(k.r, k.sigma, k.T, N, u, d, p, q, R);
  if (!(p > 0 && p < 1)) return set_error(PCF_EINVAL, "contract %d: lattice p = %g not in (0,1)", idx, p);
  memset(&C, 0, sizeof C);
  C.S0 = k.S0;
  C.E = k.E;
  C.u = u;
  C.d = d;
  C.p = p;
  C.q = q;
  C.lp = log(p);
  C.lq = log(q);
  C.twopi_n = 2 * 3.14159265358979323846 / N;
  if (N <= 15) {
    double small[16];
    stirlerr_table(small);
    C.stirl_n = small[N];
  } else {
    C.stirl_n = stirlerr_series((double)N);
  }
  // The reference's pow(u, i), pow(d, N - i) and S0 pow(u, i) stay inside the
  // FP64 range for every i <= N.
  const double span = std::max(fabs(log(u)), fabs(log(d))) * N + fabs(log(k.S0));
  C.wide = span < 690.0 ? 0 : 1;
  C.N = N;
  C.pf = pf;
  const int until = (N % 2 != 0) ? (N + 1) / 2 : N / 2;  // src/binom_embar.cpp:31-33
  const double ps = p * u / R;
  const double w = kWindow * sqrt((double)N) + 2;
  const double klo = std::max(0.0, floor(N * std::min(p, ps) - w));
  const double khi = std::min((double)N, ceil(N * std::max(p, ps) + w));
  const long long ilo = (long long)std::max(0.0, std::min(klo, N - khi));
  const long long ihi = std::min((long long)until - 1, (long long)std::max(khi, N - klo));
  C.i_lo = (int)ilo;
  C.i_hi = (int)ihi;
  C.has_mid = (N % 2 == 0 && N / 2 >= klo && N / 2 <= khi) ? 1 : 0;
  C.terms = std::max(0, C.i_hi - C.i_lo + 1) + C.has_mid;
  C.items = std::max(1, (C.terms + kBinomBlock - 1) / kBinomBlock);
  return PCF_OK;
}

}  // namespace

}  // namespace pcf

using namespace pcf;

extern "C" int pcf_binom_embar_batch(pcf_ctx* ctx, int n, const pcf_binom_contract* ks, int mode,
                                     double* prices) {
  return pcf::abi_guard([&]() -> int {
    if (n < 0 || (n > 0 && (!ks || !prices))) return set_error(PCF_EINVAL, "bad arguments");
    if (mode != 0 && mode != 1) return set_error(PCF_EINVAL, "mode must be 0 or 1");
    if (n == 0) return PCF_OK;
    std::vector<BinomContract> cs((size_t)n);
    int nmax = 1;
    for (int i = 0; i < n; ++i) {
      int st = setup_contract(ks[i], i, cs[i]);
      if (st) return st;
      nmax = std::max(nmax, ks[i].N);
    }
    int st;
    pcf_ctx* c = resolve_ctx(ctx, &st);
    if (!c) return st;
    st = ensure_tables(c, nmax);
    if (st) return st;
    std::vector<int> start((size_t)n + 1, 0);
    for (int i = 0; i < n; ++i) start[i + 1] = start[i] + cs[i].items;
    const int items = start[n];
    const size_t o_cs = 0;
    const size_t o_start = a256(sizeof(BinomContract) * n);
    const size_t h2d = a256(o_start + sizeof(int) * (n + 1));
    const size_t o_part = h2d;
    const size_t o_tick = a256(o_part + sizeof(double) * items);
    const size_t o_prep = a256(o_tick + sizeof(unsigned) * n);
    const size_t o_map = a256(o_prep + sizeof(BinomPrep) * n);
    const size_t total = a256(o_map + sizeof(int) * items);
    if (n > 1 && !ctx_fits(c, total)) {
      // The memory limit has no room for the whole batch (a contract takes some
      // 500 bytes, most of them its BinomPrep): in two parts.
      st = pcf_binom_embar_batch(c, n / 2, ks, mode, prices);
      return st ? st : pcf_binom_embar_batch(c, n - n / 2, ks + n / 2, mode, prices + n / 2);
    }
    st = ctx_ensure(c, total, h2d + sizeof(double) * n);
    if (st) return st;
    char* h = (char*)c->h_buf;
    char* d = (char*)c->d_buf;
    memcpy(h + o_cs, cs.data(), sizeof(BinomContract) * n);
    memcpy(h + o_start, start.data(), sizeof(int) * (n + 1));
    st = cuda_status(cudaMemcpyAsync(d, h, h2d, cudaMemcpyHostToDevice, c->stream), "H2D binom");
    if (st) return st;
    double* out = (double*)(h + h2d);  // the kernels write the sums to the pinned buffer
    BinomLaunch L;
    L.cs = (const BinomContract*)(d + o_cs);
    L.item_start = (const int*)(d + o_start);
    L.ncontracts = n;
    L.partial = (double*)(d + o_part);
    L.tickets = (unsigned*)(d + o_tick);
    L.out = out;
    L.mode = mode;
    char* tb = (char*)c->d_logtab;
    L.t.logt = (const double*)tb;
    L.t.pref = (const unsigned long long*)(tb + c->binom_off[0]);
    L.t.tie_idx = (const int*)(tb + c->binom_off[1]);
    L.t.tie_pos = (const int*)(tb + c->binom_off[2]);
    L.stirl = (const double*)(tb + c->binom_off[3]);
    L.t.nmax = c->logtab_n;
    L.t.tie_pitch = tie_pitch(c->logtab_n);
    L.exp2t = (const unsigned long long*)(tb + c->binom_off[4]);
    L.prep = (BinomPrep*)(d + o_prep);
    L.item_contract = (int*)(d + o_map);
    int wide = 0;
    for (const BinomContract& k : cs) wide += k.wide;
    const int per = kPrepBlock / 64;
    binom_prep_kernel<<<(n + per - 1) / per, kPrepBlock, 0, c->stream>>>(L);
    if (wide < n) binom_kernel<<<items, kBinomBlock, 0, c->stream>>>(L);
    if (wide) binom_wide_kernel<<<items, kBinomBlock, 0, c->stream>>>(L);
    c->launches += 1 + (wide < n) + (wide > 0);
    st = cuda_status(cudaGetLastError(), "binom kernel launch");
    if (st) return st;
    st = cuda_status(cudaStreamSynchronize(c->stream), "binom kernel");
    if (st) return st;
    for (int i = 0; i < n; ++i) prices[i] = exp(-ks[i].r * ks[i].T) * out[i];  // :49
    return PCF_OK;
  });
}

extern "C" int pcf_binom_embar(pcf_ctx* ctx, double S0, double E, double r, double sigma,
                               double T, int N, int payoff_fun, int mode, double* price) {
  return pcf::abi_guard([&]() -> int {
    if (!price) return set_error(PCF_EINVAL, "price is NULL");
    pcf_binom_contract k{S0, E, r, sigma, T, N, payoff_fun};
    return pcf_binom_embar_batch(ctx, 1, &k, mode, price);
  });
}
