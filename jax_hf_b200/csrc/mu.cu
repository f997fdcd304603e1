// Chemical potential: mu such that sum_k w_k sum_j f(eps_kj - mu) = N.
//
// One thread-block cluster (up to 16 CTAs) runs the whole root find: every
// iteration each CTA reduces its slice, publishes the partial in its shared
// memory, one cluster barrier, and warp 0 of every CTA then reads all partials
// through distributed shared memory and reduces them with a fixed shuffle tree.
// All CTAs therefore hold bit-identical (mu, lo, hi) and take identical
// branches; no global-memory round trip and no second launch per iteration.
// The bisection evaluates two levels per pass (the 3 midpoints of the next two
// levels in one reduction, then the two decisions in order).  Each pass costs a
// chain of block and cluster reductions whose latency grows with the number of
// sums: on 2304 eigenvalues (9 CTAs) the 54 steps take 49.7 us at two levels per
// pass (27 passes) and 51.4 at three; before the trees of a pass ran side by side 52, 59,
// and 65 us at one, 91 at four levels; storing the
// warp partials into every CTA's shared memory behind a single cluster barrier
// instead of the two-stage reduction measured slower (63 us at two levels, before).
//
// Methods (reference):
//   0  _find_mu_bisection  utils.py:353-382 (maxiter 54 f64 / 30 f32)
//   1  _find_mu_newton     utils.py:385-442 (maxiter 25 f64 / 15 f32)
//   2  _solve_mu           solver.py:62-101 (maxiter 25, warm start mu0)
// The iterations replay the reference update rules.  Bisection stops early
// only at an exact fixed point of (lo, hi); the Newton variants stop once the
// accepted Newton step is below 4 ulp of mu (the reference keeps iterating
// there, moving mu by at most a few ulp).
#include <cooperative_groups.h>

#include <climits>
#include <map>
#include <mutex>
#include <utility>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace hf {

constexpr int kMuThreads = 1024;
constexpr int kMuMaxCluster = 16;  // non-portable size, used when the device schedules it
constexpr int kBisLevels = 2;  // bisection levels per pass of the 256-thread variant
constexpr int kMuCertPasses = 6;  // Newton passes of a hinted bisection (certified bracket)
constexpr int kMuCertPassesCold = 12;  // from the middle of the spectrum

struct MuArgs {
  const void* eps;
  const void* w;
  int n, nb, method, maxiter;
  double target, T;
  const double* mu0;
  double* out;
  const int* active;  // optional device flag: return at once when *active == 0
  int cache;          // elements per thread kept in shared memory as (eps, w); 0: read from L2
  int certify;        // bisection: certify a bracket from the middle of the spectrum (without a hint)
  int kpt;                    // eigenvalues per thread of the cluster kernel
  const struct MuState* pre;  // what the grid-wide passes found, or nullptr
};

// Root-find state of the grid-wide passes (device memory, in the caller's workspace).
struct MuState {
  unsigned counter;  // CTAs of the running pass that have published; zero between passes
  int done, it, fixed;      // fixed: the bisection's interval no longer changes
  double lo, hi, mu;        // bracket; method 2: iterate
  double mn, mx, W;         // extreme eigenvalues, total weight
  double A, B, m, d;        // bisection: certified bracket, next iterate and probe offset
};
// loads in flight per thread when the elements are read from L2
constexpr int kMuCacheU = 4;
// the shared-memory cache holds up to this many (eps, w) entries per thread (layout
// [u][thread]; 192 KB for 1024 threads): a 144 x 144 x 8 spectrum on 16 CTAs needs 11
constexpr int kMuCacheMax = 12;

template <typename RT>
__device__ __forceinline__ double load_eps(const MuArgs& a, int e) {
  return (double)static_cast<const RT*>(a.eps)[e];
}
template <typename RT>
__device__ __forceinline__ double load_w(const MuArgs& a, int e) {
  return (double)static_cast<const RT*>(a.w)[e / a.nb];
}

// Visits the elements e = gt, gt + gs, ... < n in batches of U with all U loads of
// a batch issued before any use, so each thread keeps U L2 requests in flight
// instead of one (the passes are load-latency bound, not exp bound).
template <typename RT, int U, class F>
__device__ __forceinline__ void for_each_eps(const MuArgs& a, int gt, int gs, F&& f) {
  for (int base = gt; base < a.n; base += U * gs) {
    double ev[U], wv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = base + u * gs;
      ev[u] = e < a.n ? load_eps<RT>(a, e) : 0.0;
      wv[u] = e < a.n ? load_w<RT>(a, e) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (base + u * gs < a.n) f(ev[u], wv[u]);
  }
}

// Cluster-wide sum of (x, y); every thread of every CTA receives the total.
// Each CTA publishes its block sum in its `slots`; after the cluster barrier,
// lane r of warp 0 reads CTA r's slot (one distributed-shared-memory read per
// lane, all in flight together) and warp 0 reduces them with a fixed shuffle
// tree, so every CTA obtains bit-identical totals.  slots is double-buffered by
// `parity`: a CTA may publish the next pass while a slower one still reads this.
__device__ __forceinline__ void cluster_sum2(cg::cluster_group& cl, double& x, double& y,
                                             double (*slots)[2], double* wsm, int parity) {
  x = warp_sum(x);
  y = warp_sum(y);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) { wsm[2 * wid] = x; wsm[2 * wid + 1] = y; }
  __syncthreads();
  if (wid == 0) {  // the warp partials, reduced by one warp
    double sx = lane < nw ? wsm[2 * lane] : 0.0, sy = lane < nw ? wsm[2 * lane + 1] : 0.0;
    sx = warp_sum(sx);
    sy = warp_sum(sy);
    if (lane == 0) {
      slots[parity][0] = sx;
      slots[parity][1] = sy;
    }
  }
  cl.sync();
  if (wid == 0) {
    double tx = 0.0, ty = 0.0;
    if (lane < (int)cl.num_blocks()) {
      double(*rs)[2] = cl.map_shared_rank(slots, lane);
      tx = rs[parity][0];
      ty = rs[parity][1];
    }
    tx = warp_sum(tx);
    ty = warp_sum(ty);
    if (lane == 0) { wsm[64] = tx; wsm[65] = ty; }
  }
  __syncthreads();
  x = wsm[64];
  y = wsm[65];
}

// Cluster-wide sums of K values (as cluster_sum2) over CTAs of NW warps; v[] holds this
// thread's terms on entry and the totals on return.  bsm: 33 K doubles, slots: [2][K].
// RANGE: v[0] is a minimum and v[1] a maximum instead.  A pass is a chain of three shuffle
// trees and a cluster barrier; the trees of the K values advance level by level (one tree
// after the other, a store between them, made a pass of 3 sums 2.0 us instead of 1.8), and
// levels that would only add the zeros of absent warps and CTAs are left out.
template <int K, int NW, bool RANGE = false>
__device__ __forceinline__ void cluster_sum_n(cg::cluster_group& cl, double (&v)[K], double (*slots)[K], double* bsm,
                                              int parity) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  auto reduce = [](double (&x)[K], int first) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      if (off > first) continue;
      double y[K];
#pragma unroll
      for (int j = 0; j < K; ++j) y[j] = __shfl_xor_sync(0xffffffffu, x[j], off);
#pragma unroll
      for (int j = 0; j < K; ++j) x[j] = !RANGE || j > 1 ? x[j] + y[j] : j ? fmax(x[j], y[j]) : fmin(x[j], y[j]);
    }
  };
  auto none = [](int j) { return !RANGE || j > 1 ? 0.0 : j ? -INFINITY : INFINITY; };
  reduce(v, 16);
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < K; ++j) bsm[wid * K + j] = v[j];
  }
  __syncthreads();
  if (wid == 0) {
    double t[K];
#pragma unroll
    for (int j = 0; j < K; ++j) t[j] = lane < NW ? bsm[lane * K + j] : none(j);
    reduce(t, NW / 2);
    if (lane == 0) {
#pragma unroll
      for (int j = 0; j < K; ++j) slots[parity][j] = t[j];
    }
  }
  cl.sync();
  if (wid == 0) {
    double(*rs)[K] = lane < (int)cl.num_blocks() ? cl.map_shared_rank(slots, lane) : nullptr;
    double t[K];
#pragma unroll
    for (int j = 0; j < K; ++j) t[j] = rs ? rs[parity][j] : none(j);
    reduce(t, kMuMaxCluster / 2);
    if (lane == 0) {
#pragma unroll
      for (int j = 0; j < K; ++j) bsm[32 * K + j] = t[j];
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < K; ++j) v[j] = bsm[32 * K + j];
}

__device__ __forceinline__ void cluster_minmax(cg::cluster_group& cl, double& mn, double& mx,
                                               double (*slots)[2], double* wsm) {
  for (int off = 16; off > 0; off >>= 1) {
    mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, off));
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) { wsm[2 * wid] = mn; wsm[2 * wid + 1] = mx; }
  __syncthreads();
  if (wid == 0) {
    double a = lane < nw ? wsm[2 * lane] : INFINITY, b = lane < nw ? wsm[2 * lane + 1] : -INFINITY;
    for (int off = 16; off > 0; off >>= 1) {
      a = fmin(a, __shfl_xor_sync(0xffffffffu, a, off));
      b = fmax(b, __shfl_xor_sync(0xffffffffu, b, off));
    }
    if (lane == 0) {
      slots[2][0] = a;
      slots[2][1] = b;
    }
  }
  cl.sync();
  if (wid == 0) {
    double a = INFINITY, b = -INFINITY;
    if (lane < (int)cl.num_blocks()) {
      double(*rs)[2] = cl.map_shared_rank(slots, lane);
      a = rs[2][0];
      b = rs[2][1];
    }
    for (int off = 16; off > 0; off >>= 1) {
      a = fmin(a, __shfl_xor_sync(0xffffffffu, a, off));
      b = fmax(b, __shfl_xor_sync(0xffffffffu, b, off));
    }
    if (lane == 0) { wsm[64] = a; wsm[65] = b; }
  }
  __syncthreads();
  mn = wsm[64];
  mx = wsm[65];
}

__device__ __forceinline__ double expit(double x) { return 1.0 / (1.0 + exp(-x)); }

// x / b, correctly rounded, for a divisor b fixed over a pass with rb = 1 / b (correctly
// rounded).  q0 = x rb is within 1.5 ulp of x / b; one fma remainder step x - q0 b and
// correction makes it faithful, and by Markstein's theorem (P. Markstein, IBM J. Res.
// Dev. 34 (1990) 111-119: with y the correctly rounded 1/b and q faithful, r = x - q b is
// exact under an fma and q + r y rounds to the correctly rounded x / b) a second step
// gives the correctly rounded quotient, the bits of x / b.  The remainder must not
// underflow nor the products overflow, so numerators outside [2^-900, 2^900] in
// magnitude (and NaN and infinities) take the division, and so does every x when
// rb = 0 (recip_of: divisors outside [2^-64, 2^64]).  Five fp64 operations in place
// of a division routine per element, at the same bits.
__device__ __forceinline__ double recip_of(double b) {
  return (fabs(b) >= 0x1p-64 && fabs(b) <= 0x1p+64) ? 1.0 / b : 0.0;
}
__device__ __forceinline__ double div_by(double x, double b, double rb) {
  const double ax = fabs(x);
  if (!(ax >= 0x1p-900 && ax <= 0x1p+900) || rb == 0.0) return x / b;
  double q = x * rb;
  double r = fma(-q, b, x);
  q = fma(r, rb, q);
  r = fma(-q, b, x);
  return fma(r, rb, q);
}

// Twice the error bound of two evaluations of N with ka and kb terms summed per thread (the
// sum below twice the evaluation's rounding error, see the certified bracket below), with
// 25% to spare: evaluations by different kernels may be compared with each other.
__device__ __forceinline__ double cert_margin(int ka, int kb, double W) {
  return 1.25 * ((double)ka + (double)kb + 60.0) * 1.1102230246251565e-16 * W;
}

// What the margin is worth on the axis of x, and no less than the spacing of the numbers at m: probes any
// closer are m itself.  Infinite where N is flat.
__device__ __forceinline__ double probe_noise(double margin, double Z, double m) {
  return Z > 0.0 ? fmax(margin / Z, 0x1p-52 * fabs(m)) : INFINITY;
}

// Whether a bracket of this width is as narrow as evaluations with this margin make it: a few times the noise
// at an iterate m whose count n is next to the target (where N is flat at the target, at once: every
// level inside has to be evaluated).  Away from the target the noise at m says nothing.
__device__ __forceinline__ bool bracket_done(double width, double n, double target, double margin, double noise) {
  return fabs(n - target) <= 16.0 * margin && width <= 4.0 * noise;
}

// Offset of the two probes around a Newton iterate of N(x) = target that was moved by `step`.
// |N''| <= N' / Td for every sum of Fermi functions, so a step of at most Td / 2 leaves the
// iterate within step^2 / Td of the root; longer steps take twice the step.  `noise`: probe_noise.
__device__ __forceinline__ double probe_offset(double step, double iTd, double noise) {
  return step * iTd <= 0.5 ? fma(step * step, iTd, 1.5 * noise) : fmax(2.0 * step, 1.5 * noise);
}

// Bisection levels that need no evaluation: every midpoint >= A is decided "above", every one
// <= B "below".  True when the interval stops changing.
__device__ __forceinline__ bool replay_levels(double A, double B, int maxiter, double& lo, double& hi, int& it) {
  while (it < maxiter) {
    const double mid = 0.5 * (lo + hi);
    double nl, nh;
    if (mid >= A) { nl = lo; nh = mid; }
    else if (mid <= B) { nl = mid; nh = hi; }
    else return false;
    if (nl == lo && nh == hi) return true;
    lo = nl;
    hi = nh;
    ++it;
  }
  return false;
}

// One step of the Newton-bracket rule (solver.py:62-101) from g = N(mu) - target and
// Z = N'(mu); true once the accepted Newton step is below 4 ulp of mu.
__device__ __forceinline__ bool newton_step(double g, double Z, double& lo, double& hi, double& mu) {
  if (g < 0) lo = mu;
  if (g > 0) hi = mu;
  double mn2 = mu - g / fmax(Z, 1e-18);
  const double mb = 0.5 * (lo + hi);
  bool newton = true;
  if (mn2 <= lo || mn2 >= hi) { mn2 = mb; newton = false; }
  mn2 = fmin(fmax(mn2, lo), hi);
  if (!isfinite(mn2)) { mn2 = mb; newton = false; }
  const double step = fabs(mn2 - mu);
  mu = mn2;
  return newton && step <= 4.0 * 2.220446049250313e-16 * fmax(1.0, fabs(mu));
}

// ------------------------------------------------------------ grid-wide passes ---
// The cluster kernel below has 16 SMs: from a few ten thousand eigenvalues on it is bound
// by their FP64 pipes (one exp and one division per eigenvalue and evaluation).  These
// passes run one evaluation each over the whole grid; the last CTA to publish its sums
// (atomic ticket, no spin) takes the step, and the cluster kernel finishes from MuState.
// Every pass returns at once when the state says done.  The bisection's passes certify a
// bracket (see the hinted bisection below), the levels inside it are evaluated two per pass,
// and the cluster kernel finishes what is left (with its shared-memory cache: inside a gap that is
// some forty levels).
constexpr int kPassThreads = 256;
constexpr int kPassBlocks = 296;   // two CTAs per SM
constexpr int kPassSums = 8;
// Eigenvalues from which a call with a workspace certifies a bracket for the bisection, in the cluster kernel
// (kCertMin) or by the passes (kGridMin).  What that gives depends on the spectrum, in us against every level
// in the cluster kernel: for a metal (T = 0.1) 44 against 118 on 16384, 60 against 164 on 38416, 78 against 235
// on 98304, 77 against 281 on 131072.  With the target inside a gap (gap 2, T = 0.01) the count is flat to its
// rounding and every level there is evaluated: 121 against 118, 168 against 164, 238 against 235, 284 against 281
// (one pass to see it).  Passes from 65536 on would take 70 for the metal of 98304, but 202 against 188 in the gap
// on 65536, where the idle ones show.  kGridMinNewton: the warm-started Newton rule has only 4 to 8
// evaluations, each a launch here and a cluster barrier there: 39 us in the cluster kernel against 39, 70 against
// 50 and 95 against 61 by the passes on 165888 (T = 0.1, 0.01, 0.001), 21.1 against 22.9 where a gap ends it
// after one; on 131072 39 against 40, 55 against 44, 17.2 against 21.0.
constexpr int kCertMin = 16384, kGridMin = 131072, kGridMinNewton = 163840;
constexpr int kNewtonPasses = 5;   // method 2: Newton steps queued ahead of the cluster kernel
constexpr int kLevelPasses = 5;    // bisection: passes of two levels each behind them
constexpr int kCertPasses = 7;     // bisection: certifying passes, the first one a scan of 8 points
constexpr size_t kMuWsBytes = 256 + sizeof(double) * kPassBlocks * kPassSums;  // also 3 per warp of k_mu_levels
static_assert(kPassBlocks * kPassSums >= 3 * 32 * kMuMaxCluster, "workspace of k_mu_levels");

enum MuStage { kStageRange, kStageScan, kStageCertify };

template <typename RT, int STAGE>
__global__ void __launch_bounds__(kPassThreads) k_mu_pass(const MuArgs a, MuState* st, double* part, bool final_pass) {
  pdl_begin();
  if (a.active && !*a.active) return;
  if (STAGE != kStageRange && st->done) return;
  constexpr int K = STAGE == kStageRange ? 4 : STAGE == kStageScan ? 8 : 5;
  __shared__ double red[(kPassThreads / 32) * K];
  __shared__ bool last;
  const int gt = blockIdx.x * blockDim.x + threadIdx.x, gs = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double Td = a.T + 1e-12;
  double v[K];
#pragma unroll
  for (int j = 0; j < K; ++j) v[j] = 0.0;
  auto fermi = [](double x) { return recip_seeded(1.0 + exp(x > 600.0 ? 600.0 : x)); };  // a NaN stays one
  if constexpr (STAGE == kStageRange) {  // extremes, total and least weight
    v[0] = v[3] = INFINITY;
    v[1] = -INFINITY;
    for_each_eps<RT, kMuCacheU>(a, gt, gs, [&](double e, double w) {
      v[0] = fmin(v[0], e);
      v[1] = fmax(v[1], e);
      v[2] += w;
      v[3] = fmin(v[3], w);
    });
  } else if constexpr (STAGE == kStageScan) {  // N at 8 points inside [mn, mx]
    const double r = 1.0 / Td, m0 = st->mn, h = (st->mx - st->mn) * (1.0 / 9.0);
    for_each_eps<RT, kMuCacheU>(a, gt, gs, [&](double e, double w) {
#pragma unroll
      for (int j = 0; j < K; ++j) v[j] += w * fermi((e - fma(j + 1.0, h, m0)) * r);
    });
  } else {
    const double r = 1.0 / Td, m = st->m, pl = m - st->d, ph = m + st->d;
    for_each_eps<RT, kMuCacheU>(a, gt, gs, [&](double e, double w) {
      const double f = fermi((e - m) * r);
      v[0] += w * f;
      v[1] += w * (f * (1.0 - f));
      v[2] += w * fermi((e - pl) * r);
      v[3] += w * fermi((e - ph) * r);
      v[4] += w;
    });
  }
  // block, then grid: fixed trees, so the sums do not depend on the order of arrival
  auto combine = [](int j, double x, double y) {
    if (STAGE != kStageRange || j == 2) return x + y;
    return j == 1 ? fmax(x, y) : fmin(x, y);
  };
  auto block_all = [&]() {  // v: the block's values in thread 0
#pragma unroll
    for (int j = 0; j < K; ++j) {
      for (int off = 16; off > 0; off >>= 1) v[j] = combine(j, v[j], __shfl_xor_sync(0xffffffffu, v[j], off));
      if (lane == 0) red[wid * K + j] = v[j];
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
      for (int j = 0; j < K; ++j) {
        v[j] = red[(lane & (kPassThreads / 32 - 1)) * K + j];
        for (int off = kPassThreads / 64; off > 0; off >>= 1) v[j] = combine(j, v[j], __shfl_xor_sync(0xffffffffu, v[j], off));
      }
    }
  };
  block_all();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int j = 0; j < K; ++j) part[blockIdx.x * K + j] = v[j];
    __threadfence();
    last = atomicAdd(&st->counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int j = 0; j < K; ++j) v[j] = STAGE != kStageRange || j == 2 ? 0.0 : j == 1 ? -INFINITY : INFINITY;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += kPassThreads)
#pragma unroll
    for (int j = 0; j < K; ++j) v[j] = combine(j, v[j], __ldcg(part + b * K + j));
  block_all();
  if (threadIdx.x != 0) return;
  st->counter = 0u;
  if constexpr (STAGE == kStageRange) {
    const double mn = v[0], mx = v[1];
    st->mn = mn;
    st->mx = mx;
    st->W = v[2];
    // a bracket decides levels only while N increases: with a negative weight every level is evaluated
    st->done = v[3] < 0.0;
    st->A = INFINITY;
    st->B = -INFINITY;
    st->m = 0.5 * (mn + mx);
    st->d = 0.0;
    const double span = mx - mn + 10.0 * fmax(a.T, 1e-6);
    st->lo = mn - span;
    st->hi = mx + span;
    st->it = 0;
    st->fixed = 0;
  } else {
    const int gk = (a.n + gs - 1) / gs;
    const double margin = cert_margin(gk, a.kpt, st->W);
    double A = st->A, B = st->B;
    auto note = [&](double x, double n) {
      if (n > a.target + margin) A = fmin(A, x);
      if (n < a.target - margin) B = fmax(B, x);
    };
    double r = 0.0, d = 0.0;
    if constexpr (STAGE == kStageScan) {
      const double m0 = st->mn, h = (st->mx - st->mn) * (1.0 / 9.0);
      double xl = m0, nl = 0.0, xh = st->mx, nh = st->W;  // the points next to the target
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const double x = fma(j + 1.0, h, m0);
        note(x, v[j]);
        if (v[j] < a.target) { xl = x; nl = v[j]; }
        else if (x < xh) { xh = x; nh = v[j]; }
      }
      r = nh > nl ? xl + (xh - xl) * fmin(fmax((a.target - nl) / (nh - nl), 0.0), 1.0) : 0.5 * (xl + xh);
    } else {
      const double m = st->m;
      note(m, v[0]);
      note(m - st->d, v[2]);
      note(m + st->d, v[3]);
      const double span = st->mx - st->mn + 10.0 * fmax(a.T, 1e-6);
      const double bl = fmax(B, st->mn - span), bh = fmin(A, st->mx + span), Z = v[1] / Td;
      r = m - (v[0] - a.target) / Z;
      const bool newton = Z > 0.0 && isfinite(r) && r > bl && r < bh;
      if (!newton) r = 0.5 * (bl + bh);
      const double fw = probe_noise(margin, Z, m);
      st->done = bracket_done(bh - bl, v[0], a.target, margin, fw);
      d = newton ? probe_offset(fabs(r - m), 1.0 / Td, fw) : 0.0;  // no probes around a middle
    }
    st->A = A;
    st->B = B;
    st->m = r;
    st->d = d;
    if (STAGE == kStageCertify && (st->done || final_pass)) {
      // the levels that the bracket decides (none outside [B, A] needs an evaluation)
      const double span = st->mx - st->mn + 10.0 * fmax(a.T, 1e-6);
      double lo = st->mn - span, hi = st->mx + span;
      int it = 0;
      st->fixed = replay_levels(A, B, a.maxiter, lo, hi, it);
      st->lo = lo;
      st->hi = hi;
      st->it = it;
    }
  }
}

// Evaluations over the whole grid in the summation order of the cluster kernel: its csize
// CTAs of 32 warps are spread over csize * 8 CTAs of four of them.  kOrdParts threads share
// the elements of one of "its" threads: they form the terms, the first of them adds them in
// order from shared memory, and the last CTA combines the warp sums by the same trees.  The
// results are the cluster kernel's bit for bit, which its callers need: a last-digit change
// of mu moves the plateau stop of the conjugate-gradient solver on some problems.
constexpr int kOrdWarps = 4, kOrdParts = 4, kOrdThreads = 32 * kOrdWarps * kOrdParts;

// term(e, w, t): the K term values of an element; add(t, w, acc): acc += them.  acc is the
// thread's own sum (part 0 only).
template <typename RT, int K, class Term, class Add>
__device__ __forceinline__ void ordered_terms(const MuArgs& a, int csize, double (*buf)[kOrdParts][32 * kOrdWarps][K + 1],
                                              Term&& term, Add&& add) {
  const int vt = threadIdx.x % (32 * kOrdWarps), part = threadIdx.x / (32 * kOrdWarps);
  const int gt = blockIdx.x * 32 * kOrdWarps + vt, gs = csize * kMuThreads;
  int side = 0;
  for (int base = gt - vt; base < a.n; base += kOrdParts * gs, side ^= 1) {  // uniform over the CTA
    const int e = base + vt + part * gs;
    double* t = buf[side][part][vt];
    if (e < a.n) {
      const double w = load_w<RT>(a, e);
      term(load_eps<RT>(a, e), w, t);
      t[K] = w;
    }
    __syncthreads();
    if (part == 0) {
#pragma unroll
      for (int q = 0; q < kOrdParts; ++q)
        if (base + vt + q * gs < a.n) add(buf[side][q][vt]);
    }
  }
}

// v: sums of the virtual threads (part 0); publishes the warp sums and returns true in the
// last CTA, where warp 0 then holds the totals in every lane.
template <int K>
__device__ __forceinline__ bool ordered_totals(double (&v)[K], int csize, MuState* st, double* part) {
  __shared__ double sb[kMuMaxCluster][K];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (wid < kOrdWarps) {
    const int vw = blockIdx.x * kOrdWarps + wid;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      v[j] = warp_sum(v[j]);
      if (lane == 0) part[K * vw + j] = v[j];
    }
    if (lane == 0) __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&st->counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  if (wid < csize) {  // one warp per CTA of the cluster kernel (csize <= kOrdThreads / 32)
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const double x = warp_sum(__ldcg(part + K * (wid * 32 + lane) + j));
      if (lane == 0) sb[wid][j] = x;
    }
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int j = 0; j < K; ++j) v[j] = warp_sum(lane < csize ? sb[lane][j] : 0.0);
  }
  return true;
}
static_assert(kOrdThreads / 32 >= kMuMaxCluster, "a warp per CTA of the cluster kernel");

// One evaluation of the Newton-bracket rule.  FIRST: at mu0, with the extremes already in st.
template <typename RT, bool FIRST>
__global__ void __launch_bounds__(kOrdThreads) k_mu_newton(const MuArgs a, int csize, MuState* st, double* part) {
  pdl_begin();
  if (a.active && !*a.active) return;
  if (!FIRST && st->done) return;
  __shared__ double buf[2][kOrdParts][32 * kOrdWarps][3];
  const double Tj = fmax(a.T, 1e-12), rTj = recip_of(Tj);
  const double mu0 = FIRST ? a.mu0[0] : 0.0, mu = FIRST ? mu0 : st->mu;
  double v[2] = {0.0, 0.0};
  ordered_terms<RT, 2>(
      a, csize, buf,
      [&](double ev, double w, double* t) {
        const double p = expit(div_by(mu - ev, Tj, rTj));
        t[0] = p;
        t[1] = div_by(w * (p * (1.0 - p)), Tj, rTj);
      },
      [&](const double* t) {
        v[0] = fma(t[2], t[0], v[0]);
        v[1] += t[1];
      });
  if (!ordered_totals<2>(v, csize, st, part) || threadIdx.x != 0) return;
  st->counter = 0u;
  double lo, hi, m;
  int it, done = 0;
  bool have = true;
  if (FIRST) {
    lo = st->mn - 50.0 * Tj;
    hi = st->mx + 50.0 * Tj;
    m = fmin(fmax(mu0, lo), hi);
    it = 0;
    have = m == mu0;  // the first Newton evaluation is in hand
  } else {
    lo = st->lo;
    hi = st->hi;
    m = mu;
    it = st->it;
  }
  if (have) {
    done = newton_step(v[0] - a.target, v[1], lo, hi, m);
    done = ++it >= a.maxiter || done;
  }
  st->done = done;
  st->it = it;
  st->lo = lo;
  st->hi = hi;
  st->mu = m;
}

// Two levels of the bisection: the counts at the three midpoints, then the two decisions.
template <typename RT>
__global__ void __launch_bounds__(kOrdThreads) k_mu_levels(const MuArgs a, int csize, MuState* st, double* part) {
  pdl_begin();
  if (a.active && !*a.active) return;
  if (st->fixed || st->it >= a.maxiter) return;
  __shared__ double buf[2][kOrdParts][32 * kOrdWarps][4];
  const double iTd = 1.0 / (a.T + 1e-12);
  double lo = st->lo, hi = st->hi;
  const double m1 = 0.5 * (lo + hi), m2 = 0.5 * (lo + m1), m3 = 0.5 * (m1 + hi);
  double v[3] = {0.0, 0.0, 0.0};
  ordered_terms<RT, 3>(
      a, csize, buf,
      [&](double ev, double w, double* t) {
        t[0] = w / (1.0 + exp((ev - m1) * iTd));
        t[1] = w / (1.0 + exp((ev - m2) * iTd));
        t[2] = w / (1.0 + exp((ev - m3) * iTd));
      },
      [&](const double* t) {
        v[0] += t[0];
        v[1] += t[1];
        v[2] += t[2];
      });
  if (!ordered_totals<3>(v, csize, st, part) || threadIdx.x != 0) return;
  st->counter = 0u;
  int it = st->it;
  bool fixed = false;
  double cn = v[0], mid = m1;
  for (int l = 0; l < 2 && !fixed && it < a.maxiter; ++l) {
    const bool above = cn > a.target;
    const double nl = above ? lo : mid, nh = above ? mid : hi;
    if (nl == lo && nh == hi) {
      fixed = true;
    } else {
      lo = nl;
      hi = nh;
      ++it;
      cn = above ? v[1] : v[2];
      mid = above ? m2 : m3;
    }
  }
  st->lo = lo;
  st->hi = hi;
  st->it = it;
  st->fixed = fixed;
}

// BT threads per CTA; the bisection evaluates L levels per pass (L = 2 for the
// 256-thread variant, 1 for the 1024-thread variant, whose register budget is 64).
// NEWTON: methods 1 and 2 only (1024 threads); otherwise the bisection only, so that
// neither variant carries the other's registers (1024-thread CTAs have 64 per thread).
template <typename RT, int BT, bool NEWTON>
__global__ void __launch_bounds__(BT) k_find_mu(const MuArgs a) {
  pdl_begin();
  constexpr int L = BT <= 256 ? kBisLevels : 1, NODES = (1 << L) - 1;
  if (a.active && !*a.active) return;  // uniform across the cluster: no barrier is skipped by a subset
  // the grid-wide passes got there (uniform as well)
  if (a.pre && (NEWTON ? a.pre->done : a.pre->fixed || a.pre->it >= a.maxiter)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) a.out[0] = NEWTON ? a.pre->mu : 0.5 * (a.pre->lo + a.pre->hi);
    return;
  }
  cg::cluster_group cl = cg::this_cluster();
  __shared__ double slots[3][2];
  __shared__ double wsm[66];
  __shared__ double bslots[2][NODES];
  __shared__ double bsm[33 * NODES];
  __shared__ double cslots[2][5];  // the certifying Newton passes of a hinted bisection
  __shared__ double csm[33 * 5];
  extern __shared__ double2 mu_cache[];  // a.cache: (eps, w) of this thread's elements, [u][thread]
  const int gt = cl.block_rank() * blockDim.x + threadIdx.x;
  const int gs = cl.num_blocks() * blockDim.x;
  // every pass visits this thread's elements in the same order, from shared memory when
  // they fit (each thread reads back only what it stored: no barrier), else from L2
  if (a.cache) {
    for (int u = 0; u < a.cache; ++u) {
      const int e = gt + u * gs;
      mu_cache[u * blockDim.x + threadIdx.x] =
          e < a.n ? make_double2(load_eps<RT>(a, e), load_w<RT>(a, e)) : make_double2(0.0, 0.0);
    }
  }
  auto visit = [&](auto&& f) {
    if (a.cache) {  // the same elements in the same order as the L2 path
      for (int u = 0; u < a.cache; ++u)
        if (gt + u * gs < a.n) {
          const double2 c = mu_cache[u * blockDim.x + threadIdx.x];
          f(c.x, c.y);
        }
    } else {
      for_each_eps<RT, kMuCacheU>(a, gt, gs, f);
    }
  };

  // method 0 with a hint (the caller's previous mu): read before any CTA can write a.out
  const double hint = (!NEWTON && a.mu0 != nullptr) ? a.mu0[0] : 0.0;
  const bool has_hint = !NEWTON && a.mu0 != nullptr && isfinite(hint) && a.pre == nullptr;
  // Method 2 with a warm start: the min/max pass also forms N and Z at mu0, which
  // are the first Newton evaluation whenever mu0 lies inside the bracket.
  const bool fuse_first = NEWTON && a.method == 2 && a.mu0 != nullptr && a.pre == nullptr;
  const double mu0v = fuse_first ? a.mu0[0] : 0.0;
  const double Tf = fmax(a.T, 1e-12), rTf = recip_of(Tf);
  double mn = INFINITY, mx = -INFINITY, N0 = 0.0, Z0 = 0.0;
  double hv[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // has_hint: extremes, N and N' Td at the hint, W
  // 1 / (1 + x) for x = exp(.), kept inside the range of recip_seeded; a NaN stays one
  auto cert_fermi = [](double x) { return recip_seeded(1.0 + (x > 0x1p+860 ? 0x1p+860 : x)); };
  int parity = 0;
  if (fuse_first) {
    visit([&](double v, double w) {
      mn = fmin(mn, v);
      mx = fmax(mx, v);
      const double p = expit(div_by(mu0v - v, Tf, rTf));
      N0 = fma(w, p, N0);  // as k_mu_newton adds
      Z0 += div_by(w * (p * (1.0 - p)), Tf, rTf);
    });
  } else if (has_hint) {  // the first Newton evaluation of the hinted bisection with the extremes
    hv[0] = mn;
    hv[1] = mx;
    const double r = 1.0 / (a.T + 1e-12);
    visit([&](double v, double w) {
      hv[0] = fmin(hv[0], v);
      hv[1] = fmax(hv[1], v);
      const double f = cert_fermi(exp((v - hint) * r));
      hv[2] += w * f;
      hv[3] += w * (f * (1.0 - f));
      hv[4] += w < 0.0 ? NAN : w;  // N does not increase then: no bracket
    });
  } else if (!a.pre) {
    visit([&](double v, double) {
      mn = fmin(mn, v);
      mx = fmax(mx, v);
    });
  }
  if (a.pre) {
    mn = a.pre->mn;
    mx = a.pre->mx;
  } else if (has_hint) {
    if constexpr (!NEWTON) cluster_sum_n<5, BT / 32, true>(cl, hv, cslots, csm, parity);
    parity ^= 1;
    mn = hv[0];
    mx = hv[1];
  } else {
    cluster_minmax(cl, mn, mx, slots, wsm);
  }
  if (fuse_first) {
    cluster_sum2(cl, N0, Z0, slots, wsm, parity);
    parity ^= 1;
  }

  double result;
  if constexpr (!NEWTON) {
    // L levels of the bisection per pass: the counts at all 2^L - 1
    // midpoints of the next L levels (a binary tree of intervals, each midpoint
    // formed exactly as the one-level loop would form it) come from one cluster
    // reduction, then the L decisions are replayed in order; same decisions and
    // result as one level per pass, with L times fewer dependent reductions.
    const double T = a.T;
    const double span = mx - mn + 10.0 * fmax(T, 1e-6);
    double lo = mn - span, hi = mx + span;
    const double Td = T + 1e-12, iTd = 1.0 / Td;
    int it = 0;
    bool fixed = false;
    double A = INFINITY, B = -INFINITY;
    constexpr bool COLD = BT > 256;  // a.certify is for large spectra only
    if (has_hint || (COLD && a.certify)) {
      // Certified bracket from the hint, or from the middle of the spectrum.  For weights >= 0
      // N(x) = sum w / (1 + exp((e - x) / Td)) is increasing in x; an evaluation N~(x) differs from it by at most E = (kpt + 24) u W
      // (kpt terms summed per thread, a reduction tree of depth <= 14, about 6 u per term, and u W for the
      // rounding of the exponent's argument y, whose error u |y| moves a term by f (1 - f) u |y| < 0.23 u;
      // as a product of two exponentials with |z| <= 2 in the second, by less than 1.3 u, and by 2 u for
      // the second exponential and the product; W = sum w).  So once
      // N~(A) > target + margin with margin = cert_margin(...) >= 2E, every x >= A has
      // N~(x) > target: the bisection's decision at a midpoint m >= A is "above" without
      // an evaluation, and likewise "below" for m <= B once N~(B) < target - margin.
      // Newton passes from the hint put A and B within a few margin / N' of the root,
      // each evaluating N and N' at the iterate and N at two probes around it; then the
      // levels whose midpoints lie outside (B, A) are replayed without evaluations and
      // only the last few levels are evaluated.  The decisions, and so the result, are
      // those of evaluating every level.
      // With a hint the first evaluation came with the extremes, at the hint itself: a call on 2304
      // eigenvalues (T = 0.1) takes 16.0 us with a hint 1e-7 off the root and 17.8 with one 1e-2 off,
      // 49 without a hint.
      const int kpt = (a.n + gs - 1) / gs, passes = !COLD || has_hint ? kMuCertPasses : kMuCertPassesCold;
      double m = !COLD || has_hint ? hint : 0.5 * (mn + mx), d = 0.0, width = INFINITY;
      double nA = INFINITY, nB = 0.0;  // the counts at A and B (without a hint)
      double v[5] = {hv[2], hv[3], hv[2], hv[2], hv[4]};  // N(m), N'(m) Td, N(m - d), N(m + d), W
      auto evaluate = [&] {
        // The probes are the rounded m - d and m + d, as they are recorded in A and B: what counts is the
        // count at the recorded number (one half ulp of m beside it is more than the margin for a band
        // that is narrow against its offset from zero).  exp((e - x) / Td) is the product of the
        // exponential at m and the factor of the realised offset m - x where that is small.
        const double pl = m - d, ph = m + d, zl = (m - pl) * iTd, zh = (m - ph) * iTd;
        const bool fac = zl <= 2.0 && zh >= -2.0;
        const double up = exp(zl), dn = exp(zh);
#pragma unroll
        for (int j = 0; j < 5; ++j) v[j] = 0.0;
        visit([&](double ev, double w) {
          const double g = exp((ev - m) * iTd);
          const double f = cert_fermi(g);
          v[0] += w * f;
          v[1] += w * (f * (1.0 - f));
          v[2] += w * cert_fermi(fac ? g * up : exp((ev - pl) * iTd));
          v[3] += w * cert_fermi(fac ? g * dn : exp((ev - ph) * iTd));
          v[4] += w < 0.0 ? NAN : w;  // N does not increase then: no bracket
        });
        cluster_sum_n<5, BT / 32>(cl, v, cslots, csm, parity);
        parity ^= 1;
      };
      for (int t = 0;;) {
        // one copy of the evaluation in each kernel: a loop's calls find the instruction cache cold
        if constexpr (COLD) {
          if (t > 0 || !has_hint) evaluate();
        }
        const double margin = cert_margin(kpt, kpt, v[4]);
        if (isnan(margin)) break;
        const double xs[3] = {m, m - d, m + d}, ns[3] = {v[0], v[2], v[3]};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          if (ns[q] > a.target + margin) A = fmin(A, xs[q]);
          if (ns[q] < a.target - margin) B = fmax(B, xs[q]);
        }
        const double Z = v[1] * iTd;
        const double bl = fmax(B, lo), bh = fmin(A, hi);
        double r = m - (v[0] - a.target) / Z;
        // a step that left more than half of the bracket is followed by its middle
        const bool slow = bh - bl > 0.5 * width;
        width = bh - bl;
        const bool newton = Z > 0.0 && isfinite(r) && r > bl && r < bh && !slow;
        if (!newton) r = 0.5 * (bl + bh);
        const double floor_w = probe_noise(margin, Z, m);
        if (bracket_done(width, v[0], a.target, margin, floor_w) || ++t == passes) break;
        // fewer than one level in 30 Td over the bracket: N is a staircase, which Newton's rule does not climb
        if (COLD && !has_hint) {
          if (v[0] > a.target) nA = fmin(nA, v[0]);
          else nB = fmax(nB, v[0]);
          if ((fmin(nA, v[4]) - nB) * Td * a.n < 0.03 * v[4] * width) break;
        }
        d = newton ? probe_offset(fabs(r - m), iTd, floor_w) : 0.0;  // no probes around a middle
        m = r;
        if constexpr (!COLD) evaluate();
      }
    } else if (a.pre) {  // what the grid-wide passes left
      A = a.pre->A;
      B = a.pre->B;
      lo = a.pre->lo;
      hi = a.pre->hi;
      it = a.pre->it;
      fixed = a.pre->fixed != 0;
    }
    // the levels decided by the certified bracket (none without one)
    if (!fixed) fixed = replay_levels(A, B, a.maxiter, lo, hi, it);
    while (it < a.maxiter && !fixed) {
      double nlo[NODES + 1], nhi[NODES + 1], mid[NODES + 1];
      nlo[1] = lo;
      nhi[1] = hi;
#pragma unroll
      for (int j = 1; j <= NODES; ++j) {
        mid[j] = 0.5 * (nlo[j] + nhi[j]);
        if (2 * j + 1 <= NODES) {
          nlo[2 * j] = nlo[j];
          nhi[2 * j] = mid[j];
          nlo[2 * j + 1] = mid[j];
          nhi[2 * j + 1] = nhi[j];
        }
      }
      // exp((e - m_j) / Td) = exp((e - m_1) / Td) * exp((m_1 - m_j) / Td) where the
      // second factor is finite and nonzero; direct exp for the other midpoints
      // the factors are the same for every thread: lane j - 1 of each warp evaluates
      // factor j and the warp shares them
      double r[NODES + 1];
      bool fac[NODES + 1];
      {
        const int ln = threadIdx.x & 31;
        double zl = 0.0;
#pragma unroll
        for (int j = 1; j <= NODES; ++j)
          if (ln == j - 1) zl = (mid[1] - mid[j]) * iTd;
        const double rl = fabs(zl) < 700.0 ? exp(zl) : 0.0;
#pragma unroll
        for (int j = 1; j <= NODES; ++j) {
          fac[j] = fabs((mid[1] - mid[j]) * iTd) < 700.0;
          r[j] = __shfl_sync(0xffffffffu, rl, j - 1);
        }
      }
      double cnt[NODES];
#pragma unroll
      for (int j = 0; j < NODES; ++j) cnt[j] = 0.0;
      visit([&](double ev, double w) {
        const double g = exp((ev - mid[1]) * iTd);
#pragma unroll
        for (int j = 1; j <= NODES; ++j) {
          const double x = fac[j] ? g * r[j] : exp((ev - mid[j]) * iTd);
          cnt[j - 1] += w / (1.0 + x);
        }
      });
      cluster_sum_n<NODES, BT / 32>(cl, cnt, bslots, bsm, parity);
      parity ^= 1;
      int node = 1;
#pragma unroll
      for (int l = 0; l < L; ++l) {
        if (fixed || it >= a.maxiter) break;
        // node's count and midpoint by select chains (no dynamically indexed arrays)
        double cn = 0.0, mn_ = 0.0;
#pragma unroll
        for (int j = 1; j <= NODES; ++j)
          if (j == node) { cn = cnt[j - 1]; mn_ = mid[j]; }
        const bool above = cn > a.target;
        const double nl = above ? lo : mn_;
        const double nh = above ? mn_ : hi;
        if (nl == lo && nh == hi) {  // exact fixed point
          fixed = true;
          break;
        }
        lo = nl;
        hi = nh;
        node = 2 * node + (above ? 0 : 1);
        ++it;
      }
    }
    result = 0.5 * (lo + hi);
  } else {
    const double Tj = fmax(a.T, 1e-12), rTj = recip_of(Tj);
    double lo, hi, mu;
    if (a.method == 1) {
      const double span = mx - mn + 10.0 * fmax(Tj, 1e-6);
      lo = mn - span;
      hi = mx + span;
      mu = 0.5 * (lo + hi);
    } else {
      lo = mn - 50.0 * Tj;
      hi = mx + 50.0 * Tj;
      const double m0 = a.mu0 ? a.mu0[0] : 0.0;
      mu = fmin(fmax(m0, lo), hi);
    }
    int it = 0;
    if (a.pre) {  // method 2, carried on from the grid-wide passes
      lo = a.pre->lo;
      hi = a.pre->hi;
      mu = a.pre->mu;
      it = a.pre->it;
    }
    const bool have_first = fuse_first && mu == mu0v;
    for (; it < a.maxiter; ++it) {
      double N = 0.0, Z = 0.0;
      if (it == 0 && have_first) {
        N = N0;
        Z = Z0;
      } else {
        visit([&](double ev, double w) {
          const double p = expit(div_by(mu - ev, Tj, rTj));
          N = fma(w, p, N);
          Z += div_by(w * (p * (1.0 - p)), Tj, rTj);
        });
        cluster_sum2(cl, N, Z, slots, wsm, parity);
        parity ^= 1;
      }
      if (newton_step(N - a.target, Z, lo, hi, mu)) break;
    }
    if (a.method == 1) {
      double N = 0.0, dummy = 0.0;
      visit([&](double ev, double w) { N += w * expit(div_by(mu - ev, Tj, rTj)); });
      cluster_sum2(cl, N, dummy, slots, wsm, parity);
      parity ^= 1;
      if (fabs(N - a.target) > 1e-12) mu = 0.5 * (lo + hi);
    }
    result = mu;
  }
  if (cl.block_rank() == 0 && threadIdx.x == 0) a.out[0] = result;
  cl.sync();  // keep every CTA's shared memory alive until all remote reads are done
}

}  // namespace hf

using namespace hf;

namespace hf {
int find_mu_internal(void* stream, int dtype, int method, int nk1, int nk2, int nb, const void* eps,
                     const void* weights, double n_electrons, double T, int maxiter, const double* mu0,
                     double* mu_out, const int* active, void* ws, size_t ws_bytes, bool ws_ready);

// Queues the grid-wide passes in front of the cluster kernel (a.kpt set).
template <typename RT>
static int launch_passes(cudaStream_t s, const MuArgs& a, int csize, MuState* st, double* part, bool ready) {
  if (!ready) HF_CUDA(cudaMemsetAsync(st, 0, sizeof(MuState), s));  // the ticket; the passes set the rest
  int blocks = (a.n + kPassThreads - 1) / kPassThreads;
  if (blocks > kPassBlocks) blocks = kPassBlocks;
  const int ord = csize * (kMuThreads / (32 * kOrdWarps));
  launch_pdl(k_mu_pass<RT, kStageRange>, blocks, kPassThreads, 0, s, a, st, part, false);
  if (a.method == 2) {
    launch_pdl(k_mu_newton<RT, true>, ord, kOrdThreads, 0, s, a, csize, st, part);
    for (int i = 0; i < kNewtonPasses; ++i) launch_pdl(k_mu_newton<RT, false>, ord, kOrdThreads, 0, s, a, csize, st, part);
    HF_LAUNCH_CHECK("k_mu_newton");
    return HF_OK;
  }
  launch_pdl(k_mu_pass<RT, kStageScan>, blocks, kPassThreads, 0, s, a, st, part, false);
  for (int i = 1; i < kCertPasses; ++i)
    launch_pdl(k_mu_pass<RT, kStageCertify>, blocks, kPassThreads, 0, s, a, st, part, i == kCertPasses - 1);
  for (int i = 0; i < kLevelPasses; ++i) launch_pdl(k_mu_levels<RT>, ord, kOrdThreads, 0, s, a, csize, st, part);
  HF_LAUNCH_CHECK("k_mu_pass");
  return HF_OK;
}
}

extern "C" int hf_mu_workspace_size(size_t* bytes) {
  if (!bytes) return fail(HF_ERR_INVALID, "bytes is NULL");
  *bytes = kMuWsBytes;
  return HF_OK;
}

extern "C" int hf_find_mu_ws(void* stream, int dtype, int method, int nk1, int nk2, int nb, const void* eps,
                             const void* weights, double n_electrons, double T, int maxiter, const double* mu0,
                             double* mu_out, void* workspace, size_t workspace_bytes) {
  if (!workspace || workspace_bytes < kMuWsBytes)
    return fail(HF_ERR_WORKSPACE, "workspace too small: need " + std::to_string(kMuWsBytes) + " bytes");
  if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0)
    return fail(HF_ERR_WORKSPACE, "workspace must be 256-byte aligned");
  return hf::find_mu_internal(stream, dtype, method, nk1, nk2, nb, eps, weights, n_electrons, T, maxiter, mu0,
                              mu_out, nullptr, workspace, workspace_bytes, false);
}

extern "C" int hf_find_mu(void* stream, int dtype, int method, int nk1, int nk2, int nb,
                          const void* eps, const void* weights, double n_electrons, double T,
                          int maxiter, const double* mu0, double* mu_out) {
  return hf::find_mu_internal(stream, dtype, method, nk1, nk2, nb, eps, weights, n_electrons, T, maxiter, mu0,
                              mu_out, nullptr, nullptr, 0, false);
}

int hf::find_mu_internal(void* stream, int dtype, int method, int nk1, int nk2, int nb, const void* eps,
                         const void* weights, double n_electrons, double T, int maxiter, const double* mu0,
                         double* mu_out, const int* active, void* ws, size_t ws_bytes, bool ws_ready) {
  if (dtype != HF_C128 && dtype != HF_C64) return fail(HF_ERR_INVALID, "bad dtype");
  if (method < 0 || method > 2) return fail(HF_ERR_INVALID, "method must be 0, 1 or 2");
  if (nk1 < 1 || nk2 < 1 || nb < 1) return fail(HF_ERR_INVALID, "bad shape");
  if (!eps || !weights || !mu_out) return fail(HF_ERR_INVALID, "NULL argument");
  const bool single = dtype == HF_C64;
  if (maxiter <= 0) {
    if (method == 0) maxiter = single ? 30 : 54;
    else if (method == 1) maxiter = single ? 15 : 25;
    else maxiter = 25;
  }
  const size_t n_all = (size_t)nk1 * (size_t)nk2 * (size_t)nb;
  if (n_all > (size_t)INT_MAX) return fail(HF_ERR_UNSUPPORTED, "more than 2^31 - 1 eigenvalues");
  MuArgs a = {};
  a.eps = eps; a.w = weights;
  a.n = (int)n_all; a.nb = nb; a.method = method; a.maxiter = maxiter;
  a.target = n_electrons; a.T = T; a.mu0 = mu0; a.out = mu_out; a.active = active;
  // bisection: every pass evaluates 3 midpoints per eigenvalue, so small
  // meshes use 256-thread CTAs with one eigenvalue per thread, spread over up to 16
  // SMs; the Newton variants (one evaluation per pass, bound by the cluster barrier
  // of each pass): up to four per thread of 1024-thread CTAs
  const int threads = (method == 0 && a.n <= kMuMaxCluster * 256) ? 256 : kMuThreads;
  const int per_cta = method == 0 ? threads : kMuCacheU * kMuThreads;
  int csize = (a.n + per_cta - 1) / per_cta;
  if (csize < 1) csize = 1;
  if (csize > kMuMaxCluster) csize = kMuMaxCluster;
  const void* fn = method != 0 ? (single ? (const void*)k_find_mu<float, kMuThreads, true>
                                         : (const void*)k_find_mu<double, kMuThreads, true>)
                   : threads == 256 ? (single ? (const void*)k_find_mu<float, 256, false>
                                              : (const void*)k_find_mu<double, 256, false>)
                                    : (single ? (const void*)k_find_mu<float, kMuThreads, false>
                                              : (const void*)k_find_mu<double, kMuThreads, false>);
  unsigned long long ctx = 0;
  if (int cst = context_id(&ctx)) return cst;
  // per (kernel, context), set up once under a lock: the largest schedulable cluster
  // size (beyond the portable 8 only as large as the device can co-schedule) and the
  // opt-in for the shared-memory cache of the largest block
  static std::mutex mu_setup;
  static std::map<std::pair<const void*, unsigned long long>, int> max_cluster;
  {
    std::lock_guard<std::mutex> lk(mu_setup);
    auto key = std::make_pair(fn, ctx);
    auto it = max_cluster.find(key);
    if (it == max_cluster.end()) {
      int mc = 8;
      if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
        cudaLaunchConfig_t q = {};
        q.gridDim = dim3(kMuMaxCluster, 1, 1);
        q.blockDim = dim3(threads, 1, 1);
        cudaLaunchAttribute qa[1];
        qa[0].id = cudaLaunchAttributeClusterDimension;
        qa[0].val.clusterDim.x = kMuMaxCluster;
        qa[0].val.clusterDim.y = 1;
        qa[0].val.clusterDim.z = 1;
        q.attrs = qa;
        q.numAttrs = 1;
        int c = 0;
        if (cudaOccupancyMaxPotentialClusterSize(&c, fn, &q) == cudaSuccess && c >= 8) mc = c < kMuMaxCluster ? c : kMuMaxCluster;
      }
      cudaGetLastError();  // a refused query leaves the portable size
      HF_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)((size_t)kMuCacheMax * kMuThreads * sizeof(double2))));
      it = max_cluster.emplace(key, mc).first;
    }
    if (csize > it->second) csize = it->second;
  }
  {
    const long long per = ((long long)a.n + (long long)csize * threads - 1) / ((long long)csize * threads);
    a.cache = per <= kMuCacheMax ? (int)per : 0;
    a.kpt = (int)per;
  }
  // the grid-wide passes, given a workspace: for the bisection without a hint (with one, or below
  // kGridMin, the cluster kernel certifies its own bracket) and the warm-started Newton rule
  const bool bisect = method == 0 && !mu0 && T + 1e-12 > 0.0 && a.n >= kCertMin;
  const bool grid = ws && ws_bytes >= kMuWsBytes;
  if (grid && bisect && a.n < kGridMin) a.certify = 1;
  if (grid && (method == 2 ? mu0 != nullptr && a.n >= kGridMinNewton : bisect && a.n >= kGridMin)) {
    MuState* st = static_cast<MuState*>(ws);
    double* part = reinterpret_cast<double*>(static_cast<char*>(ws) + 256);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int e = single ? launch_passes<float>(s, a, csize, st, part, ws_ready)
                         : launch_passes<double>(s, a, csize, st, part, ws_ready);
    if (e) return e;
    a.pre = st;
  }
  const size_t cache_bytes = (size_t)a.cache * threads * sizeof(double2);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(csize, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = a.cache ? cache_bytes : 0;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (method != 0) {
    if (single) HF_CUDA(cudaLaunchKernelEx(&cfg, k_find_mu<float, kMuThreads, true>, a));
    else HF_CUDA(cudaLaunchKernelEx(&cfg, k_find_mu<double, kMuThreads, true>, a));
  } else if (threads == 256) {
    if (single) HF_CUDA(cudaLaunchKernelEx(&cfg, k_find_mu<float, 256, false>, a));
    else HF_CUDA(cudaLaunchKernelEx(&cfg, k_find_mu<double, 256, false>, a));
  } else {
    if (single) HF_CUDA(cudaLaunchKernelEx(&cfg, k_find_mu<float, kMuThreads, false>, a));
    else HF_CUDA(cudaLaunchKernelEx(&cfg, k_find_mu<double, kMuThreads, false>, a));
  }
  return HF_OK;
}
