// Binomial-lattice backward induction (the reference's binom_vanilla_eur and
// binom_vanilla_amer) on one GPU.
//
// Reference: binom() of src/binom_vanilla_eur.cpp:5-39 and
// src/binom_vanilla_amer.cpp:5-40, on the beta-lattice of
// src/binom_vanilla_eur.cpp:14-22. Level N holds payoff(S0 u^i d^{N-i}),
// i = 0..N; each level n < N replaces v[i] by (p v[i+1] + q v[i]) / R, and the
// American version by the larger of that and payoff(S0 u^i d^{n-i}). v[0] of
// level 0 is the price.
//
// The result is the reference's bit for bit: node prices are
// (S0 * u^i) * d^j with u^i and d^j from host tables made by the same libm
// pow the reference calls; the arithmetic is IEEE FP64 in the reference's
// order (explicit _rn operations, and the unit is compiled with -fmad=false);
// and every level is a pure function of the level above, so computing a
// level's nodes in parallel changes nothing.
//
// The division by R is Markstein's: with y = RN(1/R) correctly rounded,
// q0 = RN(s y), rem = RN(s - q0 R) (exact, an FMA) and q = RN(q0 + rem y) is
// the correctly rounded quotient (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34,
// 1990): three FP64 operations. On GB300 an FP64 instruction occupies an SM
// quarter's pipe for 64 cycles (measured, at any number of active lanes; 19
// cycles per SM with four warps), and IEEE division takes 560 cycles there,
// so the FP64 operations of a node are the whole cost: 8 for an American node
// (6 European) with this division against 16. The exponent of the remainder
// limits the proof to s >= 2^-960; nodes below that differ by at most the last
// bit of a value that weighs below 2^-260 of any price of 2^-700 or more, and
// a smaller or non-finite price is computed again with the IEEE division
// (EXACT), as is every lattice whose R, p or q is out of the ordinary range or
// whose nodes may be infinite or not a number (lat_leaves_range).
//
// Two kernels (where a memory limit leaves no room for the strips' rings, the
// blocked one alone):
//   strips   columns i are cut into strips of 24 W (W = 1..4 warps, 24 columns
//            each). A level needs only v[i] and v[i+1], so values flow from
//            right to left and a node stays in its thread's register for the
//            column's whole life. A warp carries its right neighbour's first 8
//            columns as a halo and advances 8 levels between two exchanges:
//            within a thread block through shared memory, between blocks
//            through a ring of 8-byte words in global memory, where "not
//            written yet" is a NaN pattern no node takes. There is no grid
//            barrier: a block lags its right neighbour by the exchange's
//            latency once and then keeps pace. A courier warp polls the ring
//            and hands the words on through shared memory, so that the L2
//            latency stays off the level chain; with an SM quarter idle
//            (W < 4) another warp computes the exercise values ahead. Level by
//            level exchange (32 columns a warp, no halo) measured 0.44 us a
//            level against 0.24 us (European, N = 1000): the exchange costs
//            about as much as the level's own chain of five dependent FP64
//            operations (424 cycles), and the lanes that the halo wastes cost
//            nothing, since an FP64 instruction takes as long with one lane.
//   blocked  lattices with more columns than resident strips (N + 1 >
//            kStripsPerSm x 96 x SMs): a grid step advances kLatSteps levels;
//            a block loads its share of the nodes plus kLatSteps to the right,
//            advances them in shared memory and writes them to the other of
//            two level arrays, one bounded grid barrier per step. The strips
//            take over once the level fits them.
// Measured on GB300 (whole call; before: the blocked kernel with IEEE
// division, whose block 0 ran the last 2048 levels alone): American put N =
// 10,000 38.2 -> 3.1 ms, of which 0.2 ms are the host's pow tables and 0.1 ms
// the strips' start-up lag; N = 1000 5.4 -> 0.33 ms.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "pcf_api_internal.h"
#include "pcf_device.cuh"

namespace pcf {

namespace {

constexpr int kLatBlock = 256;     // blocked kernel
constexpr int kLatSteps = 128;     // blocked kernel: levels per grid step
constexpr int kLatMaxN = 2000000;
constexpr int kStripWarps = 4;     // strips: most compute warps per block
constexpr int kStripsPerSm = 6;    // strips: most blocks per SM
constexpr int kHalo = 8;           // strips: levels between two exchanges, a power of two
constexpr int kOwn = 32 - kHalo;   // strips: columns a warp owns, a multiple of kHalo
constexpr int kRing = 1024;        // strips: words of a ring between two blocks of threads
constexpr int kInRing = 64;        // strips: words of the shared-memory ring
constexpr int kRingCheck = 32;     // strips: level blocks between two overrun checks
constexpr int kKept = 64;          // strips, test hook: words the courier hands on before it stops
constexpr unsigned long long kEmpty = ~0ULL;  // a NaN pattern no node takes

struct LatticeParams {
  double S0, E, p, q, R, invR;
  int N, pf, american;
  const double* up;  // pow(u, i), i = 0..N
  const double* dn;  // pow(d, j), j = 0..N
  double* A;         // blocked: two level arrays of N + 1 nodes
  double* B;
  unsigned* barrier;
  int* err;
  unsigned wait_limit;     // blocked: polls at the grid barrier before giving up
  unsigned barrier_extra;  // blocked, test hook: arrivals the barrier expects beyond the grid
  double* out;
  // strips
  int top;                     // level the strips start from
  const double* src;           // its nodes (NULL: level N, the payoffs)
  int warps;                   // compute warps per block
  int strips;                  // blocks
  int sms;
  unsigned long long* ring;    // strips x kRing words, filled with kEmpty
  unsigned* taken;             // strips: words of the ring its reader has taken
  unsigned word_limit;         // polls before giving up: the courier's for a neighbour's word,
  unsigned reader_limit;       // a strip's for its ring's reader,
  unsigned hand_limit;         // and a lane's for a word from the courier (shared memory)
  int withhold;                // test hook: what strip 1 (kLatWord) or strip 0's courier keeps back
};

// What P.err says gave up, and the host's words for it. The first one stays.
enum LatWait : int { kLatBarrier = 1, kLatWord = 2, kLatReader = 3, kLatHandOver = 4 };
const char* lat_wait_name(int w) {
  return w == kLatWord     ? "wait for the right neighbour's nodes"
         : w == kLatReader ? "wait for the ring's reader"
         : w == kLatHandOver ? "wait for the courier's words"
                             : "grid barrier";
}

// include/common.h:56-60: std::max(payoff_fun * (St - E), 0.0).
__device__ __forceinline__ double lat_payoff(const LatticeParams& P, int n, int i) {
  const double S = __dmul_rn(__dmul_rn(P.S0, P.up[i]), P.dn[n - i]);
  const double a = __dmul_rn((double)P.pf, __dsub_rn(S, P.E));
  return a < 0.0 ? 0.0 : a;
}

// (p v[i+1] + q v[i]) / R, each operation rounded.
template <bool EXACT>
__device__ __forceinline__ double lat_hold(const LatticeParams& P, double vi, double vi1) {
  const double s = __dadd_rn(__dmul_rn(P.p, vi1), __dmul_rn(P.q, vi));
  if (EXACT) return __ddiv_rn(s, P.R);
  const double q0 = __dmul_rn(s, P.invR);
  return __fma_rn(__fma_rn(-q0, P.R, s), P.invR, q0);
}

// Node i of level n from nodes i, i+1 of level n+1
// (src/binom_vanilla_amer.cpp:33-35; the European version stops at jatk).
template <bool EXACT>
__device__ __forceinline__ double lat_node(const LatticeParams& P, double vi, double vi1, int n,
                                           int i) {
  const double jatk = lat_hold<EXACT>(P, vi, vi1);
  if (!P.american) return jatk;
  const double sij = lat_payoff(P, n, i);
  return jatk < sij ? sij : jatk;  // std::max(jatk, sij)
}

// ---- strips ----

__device__ __forceinline__ unsigned long long ring_load(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void ring_store(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// A node value as a ring word (any NaN will do for a NaN, but not kEmpty).
__device__ __forceinline__ unsigned long long ring_word(double v) {
  const unsigned long long x = (unsigned long long)__double_as_longlong(v);
  return x == kEmpty ? 0x7ff8000000000000ULL : x;
}
__device__ __forceinline__ bool lat_stopped(const LatticeParams& P) {
  return *((volatile int*)P.err) != 0;
}
__device__ __forceinline__ void lat_give_up(const LatticeParams& P, LatWait w) {
  atomicCAS(P.err, 0, (int)w);
}

// The courier warp of strip b: takes the words k = 0 .. words-1 from the ring
// of strip b + 1 in batches of 32, one word per lane, empties each ring slot
// and puts the word into the shared ring once its slot there is empty. Every
// 32 words it reports how many ring slots are free again.
__device__ void strip_courier(const LatticeParams& P, int b, int words,
                              volatile unsigned long long* in) {
  const int lane = threadIdx.x & 31;
  unsigned long long* ring = P.ring + (size_t)(b + 1) * kRing;
  // Test hook: strip 0's courier reports where nobody looks.
  unsigned* taken = P.taken + (P.withhold == kLatReader && b == 0 ? 0 : b + 1);
  for (int k0 = 0; k0 < words; k0 += 32) {
    const int k = k0 + lane;
    bool have = k >= words, done = have;
    unsigned long long v = kEmpty;
  #pragma unroll 1
    for (unsigned polls = 0;; ++polls) {
      if (!have) {
        v = ring_load(ring + (k & (kRing - 1)));
        if (v != kEmpty) {
          ring_store(ring + (k & (kRing - 1)), kEmpty);
          have = true;
        }
      }
      if (have && !done && in[k & (kInRing - 1)] == kEmpty) {
        in[k & (kInRing - 1)] = v;
        done = true;
      }
      if (__all_sync(0xffffffffu, done)) break;
      if ((polls & 63u) == 63u && (polls > P.word_limit || lat_stopped(P))) {
        if (lane == 0) lat_give_up(P, kLatWord);
        return;  // the compute warps see P.err in their own wait
      }
    }
    // The emptied slots before the report (a release store: __threadfence would
    // also empty the SM's L1, which holds the d^j).
    __syncwarp();
    if (lane == 0)
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(taken),
                   "r"((unsigned)min(k0 + 32, words))
                   : "memory");
  }
}

// HELP: an extra warp computes the exercise values of the strip's columns a
// block of levels ahead (blocks of at most three compute warps, whose fourth
// SM quarter is idle); otherwise each thread computes its own.
template <bool AMER, bool EXACT, bool HELP>
__global__ void __launch_bounds__(32 * (kStripWarps + 1), kStripsPerSm)
    lattice_strip_kernel(LatticeParams P) {
  constexpr int kPayCols = HELP ? kOwn * (kStripWarps - 1) + kHalo : 1;
  __shared__ double first[2][kStripWarps][kHalo];  // each warp's first nodes, by block parity
  __shared__ double pay[2][kHalo][kPayCols];       // HELP: exercise values, by block parity
  __shared__ unsigned long long in[kInRing];
  __shared__ int fail;
  const int W = P.warps, C = kOwn * W;
  // Rows of `sms` strips in alternating directions, so that an SM's strips
  // are long- and short-lived ones (a strip ends at its own first column).
  int b = blockIdx.x;
  const int row = b / P.sms, r0 = row * P.sms;
  if (row & 1) b = r0 + min(P.strips - r0, P.sms) - 1 - (b - r0);
  const int a0 = b * C, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool right = b + 1 < P.strips;  // a strip to the right feeds this one
  for (int k = threadIdx.x; k < kInRing; k += blockDim.x) in[k] = kEmpty;
  if (threadIdx.x == 0) fail = 0;
  __syncthreads();
  // Blocks of levels end at multiples of kHalo, as the strips' first columns
  // are; the first block takes the rest of the top level.
  const int n1 = (P.top - 1) & ~(kHalo - 1);  // the first block's last level
  if (w == W) {
    const int ar = a0 + C;  // the right strip's first column: it ends at level ar
    int words = kHalo * (1 + (P.top > ar ? (n1 - ar) / kHalo + 1 : 0));
    if (P.withhold == kLatHandOver && b == 0) words = min(words, kKept);  // test hook
    if (right) strip_courier(P, b, words, in);
    return;
  }
  const int meet = 32 * (HELP ? W + 1 : W);  // threads of the block's barrier
  auto block_sync = [&]() {
    asm volatile("bar.sync 1, %0;" ::"r"(meet) : "memory");
  };
  const long long flip = P.pf < 0 ? (long long)0x8000000000000000ULL : 0;
  // Column i's S0 u^i: RN(S0 u^i) is the first product of every payoff.
  auto up = [&](int i) { return i <= P.N ? __dmul_rn(P.S0, P.up[i]) : 0.0; };
  auto down = [&](int n, int i) { return P.dn[max(n - i, 0)]; };  // beyond the level: unused
  auto payoff_of = [&](double su, double dni) {  // lat_payoff from S0 u^i and d^{n-i}
    const double S = __dmul_rn(su, dni);
    if (EXACT) {
      const double a = __dmul_rn((double)P.pf, __dsub_rn(S, P.E));
      return a < 0.0 ? 0.0 : a;
    }
    // times +-1 and the comparison with 0 on the bits, off the FP64 pipe
    const long long a = __double_as_longlong(__dsub_rn(S, P.E)) ^ flip;
    return __longlong_as_double(a < 0 ? 0LL : a);
  };
  int n = P.top;
  if (HELP && w == W + 1) {
    constexpr int kChunks = (kPayCols + 31) / 32;
    double su[kChunks];
#pragma unroll
    for (int t = 0; t < kChunks; ++t) su[t] = up(a0 + 32 * t + lane);
    // Exercise values of the levels n-1 .. m of block kb.
    auto fill = [&](int kb, int lev, int m) {
#pragma unroll
      for (int t = 0; t < kChunks; ++t) {
        const int col = 32 * t + lane;
        if (32 * t < C + kHalo) {
          double d[kHalo];
#pragma unroll
          for (int j = 0; j < kHalo; ++j) d[j] = down(lev - 1 - j, a0 + col);
#pragma unroll
          for (int j = 0; j < kHalo; ++j) {
            const double x = payoff_of(su[t], d[j]);
            if (col < kPayCols) pay[kb & 1][j][col] = x;
          }
        }
      }
    };
    fill(0, n, n1);
    for (int kb = 0; n > a0; ++kb) {
      if ((kb & (kRingCheck - 1)) == kRingCheck - 1) {
        block_sync();
        const int f = *((volatile int*)&fail);
        block_sync();
        if (f) return;
      }
      const int m = kb == 0 ? n1 : n - kHalo;
      block_sync();  // block kb's values are there; kb + 1's slots were read in block kb - 1
      if (m > a0) fill(kb + 1, m, m - kHalo);
      n = m;
    }
    return;
  }
  const int i = a0 + w * kOwn + lane;
  const double su = up(i);
  auto step = [&](double v, double x) {  // one level; x: exercise value, or d^{n-i} without HELP
    const double v1 = __shfl_down_sync(0xffffffffu, v, 1);
    const double sum = __dadd_rn(__dmul_rn(P.p, v1), __dmul_rn(P.q, v));
    if (EXACT) {
      const double nv = __ddiv_rn(sum, P.R);
      if (!AMER) return nv;
      const double sij = HELP ? x : payoff_of(su, x);
      return nv < sij ? sij : nv;
    }
    const double q0 = __dmul_rn(sum, P.invR);
    const double rem = __fma_rn(-q0, P.R, sum);
    if (!AMER) return __fma_rn(rem, P.invR, q0);
    // max(quotient, sij). Both are non-negative, so they are ordered as their
    // bits are; q0 is within two units of the quotient's last place, so q0
    // decides unless it is that close to sij, while the quotient is on its way.
    const long long y = __double_as_longlong(HELP ? x : payoff_of(su, x));
    const long long x0 = __double_as_longlong(q0);
    bool ex = x0 < y;
    const bool close = (unsigned long long)(x0 - y + 4) <= 8ULL;
    const bool any_close = __any_sync(0xffffffffu, close);
    const double nv = __fma_rn(rem, P.invR, q0);
    if (any_close) ex = __double_as_longlong(nv) < y;
    return ex ? __longlong_as_double(y) : nv;
  };
  double v = 0.0;
  if (i <= P.top) v = P.src ? P.src[i] : payoff_of(su, down(P.top, i));
  unsigned long long* ring = P.ring + (size_t)b * kRing;  // strip 0's is written, never read
  if (P.withhold == kLatWord && b == 1) ring -= kRing;    // test hook: as strip 0's
  const bool edge = lane < kHalo;    // the nodes the left neighbour needs
  const bool halo = lane >= kOwn;    // the right neighbour's first nodes
  const bool fed = halo && w + 1 == W && right;
  volatile unsigned long long* vin = in;
  bool dead = false;
  double dn[kHalo];
  if (AMER && !HELP) {
#pragma unroll
    for (int j = 0; j < kHalo; ++j) dn[j] = down(P.top - 1 - j, i);
  }
#pragma unroll 1
  for (int kb = 0;; ++kb) {  // block kb: levels n-1 .. m from level n
    // The strip's nodes at level n, to the left neighbours.
    if (edge) {
      first[kb & 1][w][lane] = v;
      if (w == 0) ring_store(ring + ((kb * kHalo + lane) & (kRing - 1)), ring_word(v));
    }
    if (n <= a0) break;
    if ((kb & (kRingCheck - 1)) == kRingCheck - 1) {
      if (b > 0 && threadIdx.x == 0) {
        // The words of blocks up to kb + kRingCheck reuse slots whose words
        // the reader must have taken.
        const int need = (kb + kRingCheck + 1) * kHalo - kRing;
        for (unsigned polls = 0; (int)*((volatile unsigned*)(P.taken + b)) < need;) {
          if (++polls > P.reader_limit || lat_stopped(P)) {
            lat_give_up(P, kLatReader);
            fail = 1;
            break;
          }
        }
        __threadfence();
      }
      block_sync();
      const int f = *((volatile int*)&fail);
      block_sync();
      if (f) return;  // between the two barriers nothing writes `fail`: all warps agree
    }
    const int m = kb == 0 ? n1 : n - kHalo;
    double dnext[kHalo];
    if (AMER && !HELP) {  // the next block's d^{n-i} are on their way while this one runs
#pragma unroll
      for (int j = 0; j < kHalo; ++j) dnext[j] = down(m - 1 - j, i);
    }
    block_sync();
    if (AMER && HELP) {
#pragma unroll
      for (int j = 0; j < kHalo; ++j) dn[j] = pay[kb & 1][j][w * kOwn + lane];
    }
    if (halo && w + 1 < W) v = first[kb & 1][w + 1][lane - kOwn];
    if (fed && n >= a0 + C && !dead) {
      unsigned polls = 0;
      unsigned long long x;
      const int slot = (kb * kHalo + lane - kOwn) & (kInRing - 1);
      while ((x = vin[slot]) == kEmpty) {
        if ((++polls & 1023u) == 0 && (polls > P.hand_limit || lat_stopped(P))) {
          lat_give_up(P, kLatHandOver);
          fail = 1;
          dead = true;
          break;
        }
      }
      vin[slot] = kEmpty;
      v = __longlong_as_double((long long)x);
    }
    __syncwarp();
    if (n - m == kHalo) {
#pragma unroll
      for (int j = 0; j < kHalo; ++j) v = step(v, AMER ? dn[j] : 0.0);
    } else {
#pragma unroll 1
      for (int j = 0; j < n - m; ++j)
        v = step(v, !AMER ? 0.0 : HELP ? pay[0][j][w * kOwn + lane] : down(n - 1 - j, i));
    }
    n = m;
    if (AMER && !HELP) {
#pragma unroll
      for (int j = 0; j < kHalo; ++j) dn[j] = dnext[j];
    }
  }
  if (b == 0 && threadIdx.x == 0) *P.out = v;
}

// ---- blocked ----

// Advances `cnt0` nodes of level `top` (starting at node `a`) by `k` levels
// in shared memory; on return cur holds the new level's first cnt0 - k nodes.
template <bool EXACT>
__device__ double* advance(const LatticeParams& P, double* cur, double* nxt, int cnt0, int top,
                           int k, int a) {
  for (int j = 1; j <= k; ++j) {
    const int n = top - j, cnt = cnt0 - j;
    for (int t = threadIdx.x; t < cnt; t += kLatBlock)
      nxt[t] = lat_node<EXACT>(P, cur[t], cur[t + 1], n, a + t);
    __syncthreads();
    double* x = cur;
    cur = nxt;
    nxt = x;
  }
  return cur;
}

// Levels N .. P.top; the last one written is in P.B after an odd number of
// steps, in P.A after an even one.
template <bool EXACT>
__global__ void __launch_bounds__(kLatBlock) lattice_kernel(LatticeParams P, int seg_cap) {
  extern __shared__ double sm[];
  const int G = gridDim.x, b = blockIdx.x;
  // Level N (src/binom_vanilla_eur.cpp:27-28 writes max((S - E) pf, 0), the
  // same value as payoff()).
  for (int i = b * kLatBlock + threadIdx.x; i <= P.N; i += G * kLatBlock)
    P.A[i] = lat_payoff(P, P.N, i);
  if (!group_barrier(P.barrier, (unsigned)G + P.barrier_extra, P.err, P.wait_limit)) return;
  double* src = P.A;
  double* dst = P.B;
  int top = P.N;
  while (top > P.top) {
    const int k = min(kLatSteps, top - P.top);
    const int bot = top - k;  // the new level has bot + 1 nodes
    const int seg = (bot + 1 + G - 1) / G;
    const int a = b * seg, e = min(a + seg, bot + 1);
    if (a < e) {
      const int cnt0 = e - a + k;  // nodes [a, e + k) of level top; e + k <= top + 1
      double* cur = sm;
      double* nxt = sm + seg_cap + kLatSteps;
      for (int t = threadIdx.x; t < cnt0; t += kLatBlock) cur[t] = src[a + t];
      __syncthreads();
      cur = advance<EXACT>(P, cur, nxt, cnt0, top, k, a);
      for (int t = threadIdx.x; t < e - a; t += kLatBlock) dst[a + t] = cur[t];
    }
    if (!group_barrier(P.barrier, (unsigned)G + P.barrier_extra, P.err, P.wait_limit)) return;
    double* x = src;
    src = dst;
    dst = x;
    top = bot;
  }
}

// Whether a node may be infinite or not a number where the fast strips would
// lose it: they take a payoff's sign, and an American node's larger value, from
// the bits, and their division turns an infinite node into a NaN of either sign.
//   put       S0 u^i = inf where d^(n-i) = 0 is a NaN share price; other
//             infinite share prices have payoff 0;
//   American  every value, at most the largest payoff grown by R^-N, has to be
//             finite. (European strips compare nothing: what is not finite
//             reaches the root, and that is computed again.)
bool lat_leaves_range(double S0, double E, double R, int N, int pf, bool american,
                      const double* up, const double* dn) {
  if (pf < 0 && !std::isfinite(S0 * up[N]))
    for (int i = N; i >= 0 && !std::isfinite(S0 * up[i]); --i)
      if (dn[N - i] == 0.0) return true;
  if (!american) return false;
  const double top = (pf > 0 ? S0 * std::max(1.0, up[N]) * std::max(1.0, dn[N]) : 0.0) + E;
  return !(top * std::max(1.0, pow(1.0 / R, (double)N)) < 0x1p1023);
}

typedef void (*StripKernel)(LatticeParams);
StripKernel strip_kernel(bool amer, bool exact, bool help) {
  if (!amer) return exact ? lattice_strip_kernel<false, true, false> : lattice_strip_kernel<false, false, false>;
  if (help) return exact ? lattice_strip_kernel<true, true, true> : lattice_strip_kernel<true, false, true>;
  return exact ? lattice_strip_kernel<true, true, false> : lattice_strip_kernel<true, false, false>;
}

}  // namespace

}  // namespace pcf

using namespace pcf;

extern "C" int pcf_binom_vanilla(pcf_ctx* ctx, double S0, double E, double r, double sigma,
                                 double T, int N, int payoff_fun, int american, double* price) {
  return pcf::abi_guard([&]() -> int {
    if (!price) return set_error(PCF_EINVAL, "price is NULL");
    int st = check_common(S0, E, r, sigma, T, N, payoff_fun);
    if (st) return st;
    if (N > kLatMaxN) return set_error(PCF_EINVAL, "N must be <= %d", kLatMaxN);
    pcf_ctx* c = resolve_ctx(ctx, &st);
    if (!c) return st;
    double u, d, p, q, R;
    lattice(r, sigma, T, N, u, d, p, q, R);
    // The ordinary range of the three-operation division and of comparing
    // node values as integers (all of them non-negative and finite: see
    // lat_leaves_range).
    bool exact = !(R >= 0.5 && R <= 2.0 && p > 0 && p < 1 && q > 0);

    // Strips from level `top`: the level N, or the largest that fits. (One block
    // on an SM always does; how many more is asked only where it matters, which
    // spares a lattice of 30 levels 0.7 of its 31 us.)
    int occ = 1;
    if (N >= c->sm_count * kOwn * kStripWarps) {
      occ = kStripsPerSm;
      for (bool ex : {false, true}) {
        int n = 0;
        st = cuda_status(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                             &n, strip_kernel(american != 0, ex, false), 32 * (kStripWarps + 1), 0),
                         "occupancy(lattice strips)");
        if (st) return st;
        occ = std::min(occ, n);
      }
      if (occ < 1) return set_error(PCF_EINVAL, "the lattice strip block does not fit on an SM");
    }
    const int cap = occ * c->sm_count * kOwn * kStripWarps;
    int top = std::min(N, cap - 1);
    if (c->test_strip_level) top = std::min(top, c->test_strip_level);  // test hook
    const size_t nodes = (size_t)N + 1;
    int W = 0, strips = 0;
    size_t o_ring = 0, ring_bytes = 0, o_cnt = 0, cnt_bytes = 0, o_A = 0, total = 0;
    auto lay_out = [&]() {
      // The fewest warps per block that give each strip an SM of its own: up to
      // three warps of a block an FP64 instruction takes 64 cycles, four share
      // the pipe at 76 (measured).
      W = kStripWarps;
      for (int k = 1; k < kStripWarps; ++k)
        if ((long long)k * kOwn * c->sm_count >= (long long)top + 1) {
          W = k;
          break;
        }
      strips = top ? (top + kOwn * W) / (kOwn * W) : 0;
      // Scratch: up | dn | rings | counters (barrier, err, out, taken) and, for
      // the blocked levels, A | B.
      auto a256 = [](size_t x) { return (x + 255) & ~(size_t)255; };
      o_ring = a256(16 * nodes);
      ring_bytes = sizeof(unsigned long long) * kRing * (size_t)strips;
      o_cnt = a256(o_ring + ring_bytes);
      cnt_bytes = 256 + a256(sizeof(unsigned) * (size_t)strips);
      o_A = o_cnt + cnt_bytes;
      total = o_A + (top < N ? 16 * nodes : 0);
    };
    lay_out();
    // Where the memory limit has no room for the rings, the blocked kernel runs
    // every level: slower, and no more scratch than two level arrays.
    if (!ctx_fits(c, total)) {
      top = 0;
      lay_out();
    }
    const bool help = american && W < kStripWarps;
    const size_t o_up = 0, o_dn = 8 * nodes, o_B = o_A + 8 * nodes;
    const size_t o_out = o_cnt + 128;  // beside the error word: one copy brings both
    st = ctx_ensure(c, total, 16 * nodes + 256);
    if (st) return st;
    char* dv = (char*)c->d_buf;
    double* h = (double*)c->h_buf;
    // The reference's pow(u, i) and pow(d, n - i) (src/binom_vanilla_amer.cpp:28,32).
    for (size_t i = 0; i < nodes; ++i) {
      h[i] = pow(u, (double)i);
      h[nodes + i] = pow(d, (double)i);
    }
    exact = exact || lat_leaves_range(S0, E, R, N, payoff_fun, american != 0, h, h + nodes);
    st = cuda_status(cudaMemcpyAsync(dv + o_up, h, 16 * nodes, cudaMemcpyHostToDevice, c->stream),
                     "H2D lattice tables");
    if (st) return st;
    LatticeParams P;
    memset(&P, 0, sizeof P);
    P.S0 = S0;
    P.E = E;
    P.p = p;
    P.q = q;
    P.R = R;
    P.invR = 1.0 / R;
    P.N = N;
    P.pf = payoff_fun;
    P.american = american ? 1 : 0;
    P.up = (const double*)(dv + o_up);
    P.dn = (const double*)(dv + o_dn);
    P.A = (double*)(dv + o_A);
    P.B = (double*)(dv + o_B);
    P.barrier = (unsigned*)(dv + o_cnt);
    P.err = (int*)(dv + o_cnt + 64);
    P.taken = (unsigned*)(dv + o_cnt + 256);
    P.ring = (unsigned long long*)(dv + o_ring);
    P.wait_limit = P.word_limit = P.reader_limit = 1u << 22;  // seconds
    P.hand_limit = 1u << 28;
    // Test hooks: waits that cannot complete. Only the starved one is cut short;
    // the others end when they see that it gave up.
    P.barrier_extra = c->test_barrier_extra;
    P.withhold = c->test_barrier_extra ? kLatWord : c->test_lattice;
    if (P.barrier_extra) P.wait_limit = c->test_poll_limit;
    if (P.withhold == kLatWord) P.word_limit = c->test_poll_limit;
    if (P.withhold == kLatReader) P.reader_limit = c->test_poll_limit;
    if (P.withhold == kLatHandOver) P.hand_limit = c->test_poll_limit;
    P.out = (double*)(dv + o_out);
    P.top = top;
    P.warps = W;
    P.strips = strips;
    P.sms = c->sm_count;

    double root = 0;
    for (;;) {
      st = cuda_status(cudaMemsetAsync(dv + o_cnt, 0, cnt_bytes, c->stream),
                       "memset lattice counters");
      if (!st && strips > 1)  // (one strip's ring has no reader: 4 of 24 us)
        st = cuda_status(cudaMemsetAsync(dv + o_ring, 0xff, ring_bytes, c->stream),
                         "memset lattice rings");
      if (st) return st;
      if (top < N) {
        const int G = c->sm_count;
        int seg_cap = (N + 1 + G - 1) / G;
        const size_t smem = sizeof(double) * 2 * (size_t)(seg_cap + kLatSteps);
        void (*kernel)(LatticeParams, int) = exact ? lattice_kernel<true> : lattice_kernel<false>;
        st = cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)smem),
                         "lattice smem attribute");
        if (st) return st;
        void* args[] = {&P, &seg_cap};
        st = cuda_status(cudaLaunchCooperativeKernel((void*)kernel, dim3(G), dim3(kLatBlock), args,
                                                     smem, c->stream),
                         "lattice kernel launch");
        if (st) return st;
        c->launches += 1;
        P.src = ((N - top + kLatSteps - 1) / kLatSteps) % 2 ? P.B : P.A;
      }
      if (strips) {
        void* args[] = {&P};
        st = cuda_status(
            cudaLaunchCooperativeKernel((void*)strip_kernel(american != 0, exact, help),
                                        dim3(strips), dim3(32 * (W + 1 + help)), args, 0, c->stream),
            "lattice strip launch");
        if (!st) c->launches += 1;
      } else {
        st = cuda_status(cudaMemcpyAsync(P.out, P.src, 8, cudaMemcpyDeviceToDevice, c->stream),
                         "lattice root");
      }
      if (st) return st;
      st = cuda_status(cudaMemcpyAsync(h, dv + o_cnt, 256, cudaMemcpyDeviceToHost, c->stream),
                       "D2H lattice");
      if (!st) st = cuda_status(cudaStreamSynchronize(c->stream), "lattice kernel");
      if (st) return st;
      if (const int w = ((const int*)h)[16])
        return set_error(PCF_ETIMEOUT, "lattice %s gave up", lat_wait_name(w));
      root = h[16];
      if (exact || (root >= 0x1p-700 && std::isfinite(root))) break;
      exact = true;  // too small (or not finite) for the three-operation division
    }
    *price = root;
    return PCF_OK;
  });
}
