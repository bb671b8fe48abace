// cov_fit.cu -- binned maximum-likelihood gamma fit of the null tail with
// the likelihood evaluated on the GPU (FP64).
//
// esl_gam_FitCompleteBinned (called at src/covariation.c:1956) is restated
// as: location mu = phi (the tail's lower bound, fixed), rate lambda and
// shape tau maximising sum_b obs_b log(S(lo_b) - S(hi_b)) over the tail bins
// [cmin, imax], S(x) = Q(tau, lambda (x - mu)); Nelder-Mead (1965) on
// (log lambda, log tau) from moment estimates.  The whole search (Newton
// rounds, Nelder-Mead if they do not converge; see k_gam_fit) is one
// cooperative launch: each round evaluates all its likelihood points
// together, each block summing a fixed chunk of the non-empty tail bins;
// after a grid barrier every block adds the block sums in the same fixed
// order, so all blocks hold bit-identical likelihoods and take the same
// decisions without a second barrier.  Results do not depend on timing.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "cov_dev.cuh"
#include "cov_div.cuh"
#include "cov_fit.h"

namespace covgpu {

// On this chip a warp issues an FP64 instruction every ~64 cycles, whatever
// its lanes do and whether or not it depends on the one before (an SM's four
// schedulers: one in 16 cycles).  So what counts in these kernels is the
// number of FP64 instructions of the longest warp, comparisons and
// conversions from integers among them: tests are made on the words where
// the words decide, and independent parts go to different warps.

// |t| < eps |s| (or <=): where the exponents are at most `far` apart it is
// false and from `near` on true, for an eps between 2^-(near - 1) and
// 2^-(far + 1); the comparison itself between
template <bool EQ>
__device__ __forceinline__ bool negligible(double t, double s, double eps, int far, int near) {
  const int et = (__double2hiint(t) >> 20) & 0x7ff, es = (__double2hiint(s) >> 20) & 0x7ff;
  if (et != 0 && es != 0x7ff) {
    if (es - et <= far) return false;
    if (es - et >= near) return true;
  }
  return EQ ? fabs(t) <= eps * fabs(s) : fabs(t) < fabs(s) * eps;
}

// regularised upper incomplete gamma Q(a, x): series for x < a + 1, Lentz's
// continued fraction otherwise (Abramowitz & Stegun 6.5.29, 6.5.31), as the
// part that is summed and the prefactor
//   Q = 1 - sum pre  (x < a + 1),  Q = pre h  (else),  pre = x^a e^-x / Gamma(a)
__device__ double gamma_q_sum(double a, double x) {
  if (x < a + 1.0) {
    double sum = 1.0 / a, del = sum, ap = a;
    const bool in = div_range(x) && a < 1e30;
    for (int n = 0; n < 10000; n++) {
      ap += 1.0;
      const double q = in ? div_fast(x, ap) : x / ap;
      del = __dmul_rn(del, q);
      sum = __dadd_rn(sum, del);
      if (negligible<false>(del, sum, 1e-16, 52, 55)) break;
    }
    return sum;
  }
  double b = x + 1.0 - a, c = 1.0 / 1e-300, d = 1.0 / b, h = d, di = 0.0;
  for (int i = 1; i < 10000; i++) {
    di += 1.0;
    const double an = -di * (di - a);
    b += 2.0;
    d = __fma_rn(an, d, b);
    if (div_range(d) && div_range(c) && (__double2hiint(an) & 0x7fffffff) < 0x46293e59) {
      c = __dadd_rn(b, div_fast(an, c));
      d = div_fast(1.0, d);
    } else {   // the first step (c = 1e300) and arguments far out
      if (fabs(d) < 1e-300) d = 1e-300;
      c = b + an / c;
      d = 1.0 / d;
    }
    if ((__double2hiint(c) & 0x7fffffff) < 0x01a56e20 && fabs(c) < 1e-300) c = 1e-300;
    const double del = __dmul_rn(d, c);
    h = __dmul_rn(h, del);
    if (__double_as_longlong(del) == 0x3ff0000000000000ll) break;   // |del - 1| < 1e-16: only 1 itself
  }
  return h;
}
// log of the prefactor without Gamma(a): a log x - x
__device__ __forceinline__ double gamma_q_lpre(double a, double x) { return __fma_rn(a, log(x), -x); }
__device__ __forceinline__ double gamma_q_join(double a, double x, double sum, double lpre, double lga) {
  const double pre = exp(__dsub_rn(lpre, lga));
  return x < a + 1.0 ? __fma_rn(-sum, pre, 1.0) : __dmul_rn(pre, sum);
}
__device__ double gamma_q_dev(double a, double x, double lga) {
  if (x <= 0.0) return 1.0;
  return gamma_q_join(a, x, gamma_q_sum(a, x), gamma_q_lpre(a, x), lga);
}

struct FitPoint { double lambda, tau, lga, lconst; };   // lconst = tau log lambda - lgamma(tau)

// log of the gamma probability of the bin [lo, lo + h), location mu, with
// logx = log(lo - mu) when lo > mu.
// Far enough above mu (h <= (lo - mu) / 16, lambda h <= 1/2) the probability
// is computed as f(x) * integral_0^h exp(g(t)) dt,  x = lo - mu,
//   g(t) = (tau - 1) log(1 + t/x) - lambda t,
// with exp(g) = sum_k c_k t^k from (x + t) E' = (tau - 1 - lambda (x + t)) E:
//   c_{k+1} = ((tau - 1 - lambda x - k) c_k - lambda c_{k-1}) / (x (k + 1)),
// summed as d_k = c_k h^k, which needs one log and avoids the cancellation
// of Q(lo) - Q(hi); closer to mu the difference of Q is used.
__constant__ double c_inv[64];   // c_inv[k] = 1 / (k + 1)
__constant__ double c_num[60] = {0,  1,  2,  3,  4,  5,  6,  7,  8,  9,  10, 11, 12, 13, 14, 15, 16, 17, 18, 19,
                                 20, 21, 22, 23, 24, 25, 26, 27, 28, 29, 30, 31, 32, 33, 34, 35, 36, 37, 38, 39,
                                 40, 41, 42, 43, 44, 45, 46, 47, 48, 49, 50, 51, 52, 53, 54, 55, 56, 57, 58, 59};

// a non-empty bin [lo, lo + h) of the tail: x = lo - mu, x2 = lo + h - mu,
// logx = log x (x > 0); r = h / x where h <= x / 16, else -1
struct FitBin { double x, h, r, logx, x2; };

__device__ __forceinline__ bool gam_bin_far(const FitBin& B, const FitPoint& P) { return B.r >= 0.0 && P.lambda * B.h <= 0.5; }
// log of h sum_k d_k / (k + 1)
__device__ __forceinline__ double gam_far_sum(const FitBin& B, const FitPoint& P) {
  const double r = B.r, s = P.lambda * B.h, tm1 = P.tau - 1.0;
  double dkm1 = 0.0, dk = 1.0, sum = 1.0;
  for (int k = 0; k < 60; k++) {
    const double dk1 = (((tm1 - c_num[k]) * r - s) * dk - s * r * dkm1) * c_inv[k];
    const double term = dk1 * c_inv[k + 1];
    sum += term;
    dkm1 = dk; dk = dk1;
    if (negligible<true>(term, sum, 1e-17, 55, 58)) break;
  }
  return log(B.h * sum);
}
__device__ __forceinline__ double gam_far_join(const FitBin& B, const FitPoint& P, double ls) {
  return P.lconst + (P.tau - 1.0) * B.logx - P.lambda * B.x + ls;
}
// Q at the lower or upper bound of a bin near mu
__device__ __forceinline__ double gam_near_x(const FitBin& B, bool upper, const FitPoint& P) {
  const double x = upper ? B.x2 : B.x;
  return x > 0.0 ? P.lambda * x : 0.0;
}
__device__ __forceinline__ double gam_near_join(double ql, double qu) {
  const double p = ql - qu;
  return log(p > 0.0 ? p : 1e-300);
}

__device__ __forceinline__ uint64_t fit_clock() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

constexpr uint64_t kFitWaitNs = 2000000000ull;   // grid barrier gives up after 2 s
constexpr int kFitMaxPts = 6;                      // likelihood points per evaluation round

struct FitOut { double lambda, tau; int evals, status; };

struct FitGrid {
  const int* bins;       // non-empty tail bins, in bin order
  const double* cnts;    // their counts
  FitBin* geo;           // scratch: the bins' geometry
  int nnz;
  double bmin, w, mu;
  double* part;          // [2][6][gridDim.x] block sums
  unsigned* bar;         // arrival counter, zero at launch
  double* val;           // [6][nnz]: the items' terms (a search on a cluster)
  FitOut* out;
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

constexpr int kFitNear = 192;   // bins near mu whose parts a block shares out
constexpr int kFitOwn = 8;      // of which one thread owns at most these

struct FitShared {
  FitPoint pts[kFitMaxPts];
  double F[kFitMaxPts], red[8 * kFitMaxPts], pc[kFitMaxPts][2], tmp[16];
  int flag, ctl, nnear;
  int near_it[kFitNear];
  double near_r[4][kFitNear];
};

// the lanes' sums of six values, pairwise over lanes 16, 8, 4, 2 and 1 apart
// (each value's sum is the one its own butterfly gives), a lane keeping half
// of its values at each step: 8 additions instead of 30.  The total of value
// q is in lane fold_lane(q)'s group of four.
__device__ __forceinline__ double fold6(const double (&a)[kFitMaxPts], int lane) {
  const bool u = lane & 16, v = lane & 8, w = lane & 4;
  double x[3];
#pragma unroll
  for (int k = 0; k < 3; k++) x[k] = (u ? a[3 + k] : a[k]) + __shfl_xor_sync(0xffffffffu, u ? a[k] : a[3 + k], 16);
  const double y0 = (v ? x[2] : x[0]) + __shfl_xor_sync(0xffffffffu, v ? x[0] : x[2], 8);
  const double y1 = (v ? 0.0 : x[1]) + __shfl_xor_sync(0xffffffffu, v ? x[1] : 0.0, 8);
  double z = (w ? y1 : y0) + __shfl_xor_sync(0xffffffffu, w ? y0 : y1, 4);
  z += __shfl_xor_sync(0xffffffffu, z, 2);
  return z + __shfl_xor_sync(0xffffffffu, z, 1);
}
// the value whose total fold6 leaves in this lane, or -1
__device__ __forceinline__ int fold_value(int lane) {
  if (lane & 3) return -1;
  const int v = (lane & 8) ? 2 : (lane & 4) ? 1 : 0;
  return (lane & 12) == 12 ? -1 : ((lane & 16) ? 3 : 0) + v;
}

// evaluates the npts points of simplex coordinates sh.pc (written by thread
// 0) over the tail.  The work items (point q, bin k), point-major, are spread
// over the first `own` threads of each block of the grid.  Each block sums
// its items per point, arrives at the grid barrier, then adds all block sums
// in block order into sh.F.  False when the barrier timed out.
//
// A bin near mu takes two incomplete gammas.  They, the far bins' series and
// the points' lgamma are independent, so they go to different warps: far
// series to the owners, sums of the lower and upper bounds to the next two
// warps, the prefactors' logarithms to the one after, lgamma and log lambda
// to the last; the values meet in shared memory.
//
// The list's size: the bins within 17 widths of mu make up to 102 items in a
// round; more only when lambda w > 0.5, and those past the list are computed
// where they are.
//
// The tail of a 30 x 61 family with 20 nulls (16 bins): 209 us with
// everything of an item in its thread, 156 us with the near bins' parts in
// four warps, 99 us so.
//
// VAL: the blocks are a cluster that computes the items of a one-block search
// (own threads).  The terms go to memory, and after the cluster's barrier
// every block sums them all in the one block's order.
template <bool VAL>
__device__ bool fit_eval(const FitGrid& g, FitShared& sh, int npts, unsigned& phase, int own, int G, int bid) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int T = G * own, now = own >> 5, nw = blockDim.x >> 5;   // at least four warps
  const int nitems = npts * g.nnz, first = bid * own + tid;
  double* part = g.part + (size_t)(phase & 1u) * kFitMaxPts * G;
  if (tid == 0) sh.nnear = 0;
  __syncthreads();
  if (lane < npts && warp == 0) sh.pts[lane].tau = exp(sh.pc[lane][1]);
  if (lane < npts && warp == 1) sh.pts[lane].lambda = exp(sh.pc[lane][0]);
  __syncthreads();
  int slot[kFitOwn], nslot = 0;
  if (tid < own) {
    for (int it = first; it < nitems; it += T) {
      const int q = it / g.nnz;
      if (gam_bin_far(g.geo[it - q * g.nnz], sh.pts[q]) || nslot == kFitOwn) continue;
      const int s = atomicAdd(&sh.nnear, 1);
      slot[nslot++] = s;
      if (s < kFitNear) sh.near_it[s] = it;
    }
  }
  __syncthreads();
  const int nnear = min(sh.nnear, kFitNear);
  double fls = 0.0;   // the far series of the thread's first item
  if (tid < own && first < nitems) {
    const int q = first / g.nnz;
    const FitBin B = g.geo[first - q * g.nnz];
    if (gam_bin_far(B, sh.pts[q])) fls = gam_far_sum(B, sh.pts[q]);
  }
  if (warp == nw - 1 && lane < npts) {
    FitPoint& P = sh.pts[lane];
    const double lga = lgamma(P.tau);
    P.lga = lga;
    P.lconst = P.tau * log(P.lambda) - lga;
  }
  for (int c = 0; c * 32 < nnear; c++) {
    const int role = (warp - 4 * c) & (nw - 1), e = c * 32 + lane;   // nw is 4 or 8
    if (role < 1 || role > 3 || e >= nnear) continue;
    const int it = sh.near_it[e], q = it / g.nnz;
    const FitBin B = g.geo[it - q * g.nnz];
    const FitPoint& P = sh.pts[q];
    const double tau = P.tau;
    if (role < 3) {
      const double x = gam_near_x(B, role == 2, P);
      sh.near_r[role - 1][e] = x > 0.0 ? gamma_q_sum(tau, x) : 0.0;
    } else {
#pragma unroll 1
      for (int k = 0; k < 2; k++) {
        const double x = gam_near_x(B, k, P);
        sh.near_r[2 + k][e] = x > 0.0 ? gamma_q_lpre(tau, x) : 0.0;
      }
    }
  }
  __syncthreads();
  if (nnear > 0) {   // Q at the bounds, in the warps that made the sums
    for (int c = 0; c * 32 < nnear; c++) {
      const int role = (warp - 4 * c) & (nw - 1), e = c * 32 + lane;
      if (role < 1 || role > 2 || e >= nnear) continue;
      const int it = sh.near_it[e], q = it / g.nnz;
      const FitBin B = g.geo[it - q * g.nnz];
      const FitPoint& P = sh.pts[q];
      const double x = gam_near_x(B, role == 2, P);
      sh.near_r[role - 1][e] =
          x > 0.0 ? gamma_q_join(P.tau, x, sh.near_r[role - 1][e], sh.near_r[role + 1][e], P.lga) : 1.0;
    }
    __syncthreads();
  }
  double acc[kFitMaxPts];
#pragma unroll
  for (int q = 0; q < kFitMaxPts; q++) acc[q] = 0.0;
  if (tid < own) {
    int ns = 0;
    for (int it = first; it < nitems; it += T) {
      const int q = it / g.nnz, k = it - q * g.nnz;
      const FitBin B = g.geo[k];
      const FitPoint& P = sh.pts[q];
      double lp;
      if (gam_bin_far(B, P)) {
        lp = gam_far_join(B, P, it == first ? fls : gam_far_sum(B, P));
      } else {
        double ql, qu;
        const int s = ns < nslot ? slot[ns] : kFitNear;
        ns++;
        if (s < kFitNear) {
          ql = sh.near_r[0][s];
          qu = sh.near_r[1][s];
        } else {   // no room in the block's list
          ql = gamma_q_dev(P.tau, gam_near_x(B, false, P), P.lga);
          qu = gamma_q_dev(P.tau, gam_near_x(B, true, P), P.lga);
        }
        lp = gam_near_join(ql, qu);
      }
      const double v = g.cnts[k] * lp;
      if (VAL) {
        g.val[it] = v;
      } else {
#pragma unroll
        for (int r = 0; r < kFitMaxPts; r++)
          if (q == r) acc[r] -= v;
      }
    }
  }
  if (VAL) {
    cluster_sync();
    if (tid < own)
#pragma unroll
      for (int q = 0; q < kFitMaxPts; q++) {
        const int s = q * g.nnz, e = min((q + 1) * g.nnz, nitems);
#pragma unroll 4
        for (int it = s + ((tid - s) & (own - 1)); it < e; it += own) acc[q] -= __ldcg(g.val + it);
      }
  }
  if (tid < own) {
    const double z = fold6(acc, lane);
    const int q = fold_value(lane);
    if (q >= 0) sh.red[warp * kFitMaxPts + q] = z;
  }
  __syncthreads();
  if (VAL) {
    if (tid < npts) {
      double t = sh.red[tid];
      for (int i = 1; i < now; i++) t += sh.red[i * kFitMaxPts + tid];
      sh.F[tid] = t;
    }
    cluster_sync();   // the terms may be overwritten
    phase++;
    return true;
  }
  if (tid < npts) {
    double t = sh.red[tid];
    for (int i = 1; i < now; i++) t += sh.red[i * kFitMaxPts + tid];
    part[tid * G + bid] = t;
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    atomicAdd(g.bar, 1u);
    const unsigned target = (phase + 1u) * (unsigned)G;
    uint64_t t0 = 0;
    int ok = 1;
    while (ld_acquire(g.bar) < target) {
      const uint64_t now = fit_clock();
      if (t0 == 0) t0 = now;
      else if (now - t0 > kFitWaitNs) { ok = 0; break; }
    }
    sh.flag = ok;
  }
  __syncthreads();
  if (!sh.flag) return false;
  if (tid < 32) {
    double t[kFitMaxPts];   // the points' sums side by side
#pragma unroll
    for (int q = 0; q < kFitMaxPts; q++) t[q] = (q < npts && tid < G) ? __ldcg(part + q * G + tid) : 0.0;
    for (int i = tid + 32; i < G; i += 32)
#pragma unroll
      for (int q = 0; q < kFitMaxPts; q++) t[q] += q < npts ? __ldcg(part + q * G + i) : 0.0;
    const double z = fold6(t, lane);
    const int q = fold_value(lane);
    if (q >= 0 && q < npts) sh.F[q] = z;
  }
  __syncthreads();
  phase++;
  return true;
}

// The search.  Phase 1, Newton on theta = (log lambda, log tau): every round
// evaluates the 6-point stencil theta, theta +- h e1, theta +- h e2,
// theta + h (e1 + e2) (h = 1e-5) for the gradient and Hessian by central
// differences, steps -H^-1 g (a scaled gradient step where H is not
// positive definite, steps capped at 1 in log space), and halves a step that
// raised the likelihood's negative; it stops when the step is below 1e-10.
// Phase 2, only when phase 1 did not converge in 40 rounds: Nelder-Mead from
// the best point of phase 1, the same points a sequential Nelder-Mead
// visits, to 1e-12 in F and 1e-9 in theta.
// (G, bid): the blocks of the search and this block's index; a grouped
// launch runs one search per block (G = 1)
// own: the threads of a block that own items (the others help)
template <bool VAL>
__device__ __forceinline__ void gam_fit_body(const FitGrid& g, double s00, double s01, int own, int G, int bid) {
  __shared__ FitShared sh;
  double (&F)[kFitMaxPts] = sh.F;
  double (&pc)[kFitMaxPts][2] = sh.pc;
  int &flag = sh.flag, &ctl = sh.ctl;
  {
    const int T = G * blockDim.x;
    for (int k = bid * blockDim.x + threadIdx.x; k < g.nnz; k += T) {
      const double lo = g.w * g.bins[k] + g.bmin, hi = g.w * (g.bins[k] + 1) + g.bmin, h = hi - lo;
      FitBin B;
      B.x = lo - g.mu;
      B.h = h;
      B.r = (B.x > 0.0 && h <= 0.0625 * B.x) ? h / B.x : -1.0;
      B.logx = (B.x > 0.0) ? log(B.x) : 0.0;
      B.x2 = (lo + h) - g.mu;
      g.geo[k] = B;
    }
  }
  // the bins' geometry is read by other blocks' threads: a barrier round with
  // no points publishes them grid-wide
  unsigned phase = 0;
  int evals = 0, status = 0;
  if (!fit_eval<VAL>(g, sh, 0, phase, own, G, bid)) status = 2;

  // ---- phase 1: Newton ----
  // Steps below kNewtonTol in (log lambda, log tau) end the search: the
  // 6-point stencil's gradient carries the FP64 rounding of -log L (~1e-16
  // |F|) divided by H, which for tails of ~1e5 scores puts the smallest
  // reachable step near 1e-11-1e-10; the oracle's Nelder-Mead stops at ~1e-8.
  constexpr double H = 1e-5, kNewtonTol = 1e-9;
  double th0 = s00, th1 = s01;               // thread 0's state
  double bth0 = s00, bth1 = s01, bF = INFINITY;
  double d0 = 0.0, d1 = 0.0;                 // last step
  int converged = 0;
  for (int r = 0; r < 40 && !status; r++) {
    if (threadIdx.x == 0) {
      pc[0][0] = th0;     pc[0][1] = th1;
      pc[1][0] = th0 + H; pc[1][1] = th1;
      pc[2][0] = th0 - H; pc[2][1] = th1;
      pc[3][0] = th0;     pc[3][1] = th1 + H;
      pc[4][0] = th0;     pc[4][1] = th1 - H;
      pc[5][0] = th0 + H; pc[5][1] = th1 + H;
    }
    if (!fit_eval<VAL>(g, sh, 6, phase, own, G, bid)) { status = 2; break; }
    evals += 6;
    if (threadIdx.x < 32) {   // the five difference quotients, a lane each
      const int k = threadIdx.x;
      double num, den = H * H;
      if (k == 0)      { num = F[1] - F[2]; den = 2.0 * H; }
      else if (k == 1) { num = F[3] - F[4]; den = 2.0 * H; }
      else if (k == 2) num = F[1] - 2.0 * F[0] + F[2];
      else if (k == 3) num = F[3] - 2.0 * F[0] + F[4];
      else             num = F[5] - F[1] - F[3] + F[0];
      const double qt = num / den;
      if (k < 5) sh.tmp[k] = qt;
      __syncwarp();
      // -H^-1 g, a lane per component
      const double h00 = sh.tmp[2], h11 = sh.tmp[3], h01 = sh.tmp[4];
      const double det = h00 * h11 - h01 * h01;
      const double ga = sh.tmp[k == 0 ? 0 : 1], gb = sh.tmp[k == 0 ? 1 : 0], hh = k == 0 ? h11 : h00;
      const double nd = -(hh * ga - h01 * gb);
      const double dd = nd / det;
      if (k < 2) sh.tmp[5 + k] = dd;
      if (k == 0) sh.tmp[7] = det;
      __syncwarp();
    }
    if (threadIdx.x == 0) {
      ctl = 1;
      const double F0 = F[0];
      if (!(F0 <= bF) && r > 0) {
        // the step raised -log L (or gave NaN): back off towards the best point
        d0 *= 0.5; d1 *= 0.5;
        th0 = bth0 + d0; th1 = bth1 + d1;
        if (fabs(d0) < kNewtonTol && fabs(d1) < kNewtonTol) { th0 = bth0; th1 = bth1; converged = 1; ctl = 0; }
      } else {
        bth0 = th0; bth1 = th1; bF = F0;
        const double g0 = sh.tmp[0], g1 = sh.tmp[1], h00 = sh.tmp[2], h11 = sh.tmp[3], det = sh.tmp[7];
        if (h00 > 0.0 && h11 > 0.0 && det > 0.0) {
          d0 = sh.tmp[5];
          d1 = sh.tmp[6];
        } else {
          const double sc = fmax(fmax(fabs(h00), fabs(h11)), 1.0);
          d0 = -g0 / sc; d1 = -g1 / sc;
        }
        const double m = fmax(fabs(d0), fabs(d1));
        if (m > 1.0) { d0 /= m; d1 /= m; }
        if (m < kNewtonTol) { converged = 1; ctl = 0; }
        else { th0 = bth0 + d0; th1 = bth1 + d1; }
      }
    }
    __syncthreads();
    if (!ctl) break;
    __syncthreads();
  }

  // ---- phase 2: Nelder-Mead when Newton did not converge ----
  double S[3][2], SF[3];   // the simplex, kept by thread 0
  if (threadIdx.x == 0) {
    flag = converged;
    const double c0 = isfinite(bF) ? bth0 : s00, c1 = isfinite(bF) ? bth1 : s01;
    S[0][0] = c0;       S[0][1] = c1;
    S[1][0] = c0 + 0.5; S[1][1] = c1;
    S[2][0] = c0;       S[2][1] = c1 + 0.5;
    for (int k = 0; k < 3; k++) { pc[k][0] = S[k][0]; pc[k][1] = S[k][1]; }
  }
  __syncthreads();
  const bool need_nm = !flag;
  __syncthreads();
  if (need_nm && !status) {
    if (!fit_eval<VAL>(g, sh, 3, phase, own, G, bid)) status = 2;
    evals += 3;
    if (threadIdx.x == 0) for (int k = 0; k < 3; k++) SF[k] = F[k];
    for (int it = 0; it < 4000 && !status; it++) {
      int lo = 0, hi = 0, md = 0;
      if (threadIdx.x == 0) {
        for (int k = 1; k < 3; k++) { if (SF[k] < SF[lo]) lo = k; if (SF[k] > SF[hi]) hi = k; }
        md = 3 - lo - hi;
        if (md == lo || md == hi || md < 0 || md > 2)
          md = (hi == 0) ? ((lo == 1) ? 2 : 1) : ((hi == 1) ? ((lo == 0) ? 2 : 0) : ((lo == 0) ? 1 : 0));
        if (fabs(SF[hi] - SF[lo]) <= 1e-12 * (fabs(SF[lo]) + 1e-30) && fabs(S[hi][0] - S[lo][0]) < 1e-9 &&
            fabs(S[hi][1] - S[lo][1]) < 1e-9) {
          ctl = 0;
        } else {
          const double c0 = 0.5 * (S[lo][0] + S[md][0]), c1 = 0.5 * (S[lo][1] + S[md][1]);
          pc[0][0] = c0 + (c0 - S[hi][0]);       pc[0][1] = c1 + (c1 - S[hi][1]);         // reflection
          pc[1][0] = c0 + 2.0 * (c0 - S[hi][0]); pc[1][1] = c1 + 2.0 * (c1 - S[hi][1]);   // expansion
          pc[2][0] = c0 + 0.5 * (S[hi][0] - c0); pc[2][1] = c1 + 0.5 * (S[hi][1] - c1);   // contraction
          ctl = 1;
        }
      }
      __syncthreads();
      if (!ctl) break;
      if (!fit_eval<VAL>(g, sh, 3, phase, own, G, bid)) { status = 2; break; }
      evals += 3;
      if (threadIdx.x == 0) {
        const double fr = F[0];
        ctl = 1;
        if (fr < SF[lo]) {
          if (F[1] < fr) { S[hi][0] = pc[1][0]; S[hi][1] = pc[1][1]; SF[hi] = F[1]; }
          else           { S[hi][0] = pc[0][0]; S[hi][1] = pc[0][1]; SF[hi] = fr; }
        } else if (fr < SF[md]) {
          S[hi][0] = pc[0][0]; S[hi][1] = pc[0][1]; SF[hi] = fr;
        } else if (F[2] < SF[hi]) {
          S[hi][0] = pc[2][0]; S[hi][1] = pc[2][1]; SF[hi] = F[2];
        } else {   // shrink towards the best vertex
          int nq = 0;
          for (int k = 0; k < 3; k++)
            if (k != lo) {
              pc[nq][0] = S[lo][0] + 0.5 * (S[k][0] - S[lo][0]);
              pc[nq][1] = S[lo][1] + 0.5 * (S[k][1] - S[lo][1]);
              nq++;
            }
          ctl = 2;
        }
      }
      __syncthreads();
      if (ctl == 2) {
        if (!fit_eval<VAL>(g, sh, 2, phase, own, G, bid)) { status = 2; break; }
        evals += 2;
        if (threadIdx.x == 0) {
          int nq = 0;
          for (int k = 0; k < 3; k++)
            if (k != lo) { S[k][0] = pc[nq][0]; S[k][1] = pc[nq][1]; SF[k] = F[nq]; nq++; }
        }
      }
      __syncthreads();
    }
  }
  if (bid == 0 && threadIdx.x == 0) {
    double l0 = bth0, l1 = bth1;
    if (need_nm) {
      int lo = 0;
      for (int k = 1; k < 3; k++) if (SF[k] < SF[lo]) lo = k;
      l0 = S[lo][0]; l1 = S[lo][1];
    }
    g.out->lambda = exp(l0);
    g.out->tau = exp(l1);
    g.out->evals = evals;
    g.out->status = status;
  }
}

__global__ void __launch_bounds__(256, 3)
k_gam_fit(FitGrid g, double s00, double s01, int own) {
  gam_fit_body<false>(g, s00, s01, own, (int)gridDim.x, (int)blockIdx.x);
}

// one search per cluster of C blocks (a block when C is 1): fit e of the
// batch's fits
template <bool VAL>
__global__ void __launch_bounds__(256, 3)
k_gam_fit_grp(const FitGrid* __restrict__ gs, const double2* __restrict__ start, int C) {
  const int e = VAL ? (int)blockIdx.x / C : (int)blockIdx.x;
  const FitGrid g = gs[e];
  const double2 s0 = start[e];
  gam_fit_body<VAL>(g, s0.x, s0.y, 256, C, VAL ? (int)blockIdx.x % C : 0);
}

// Blocks per fit of a batch: FP64 throughput is an SM's, and a search on one
// block leaves the other SMs idle while the batch waits for it, so clusters of
// up to 8 (the portable size) while the fits' blocks do not exceed the SMs.
// The two launches of 64 families (47 fits on clusters of three, 17 on eight):
// 3.77 ms with a block each, 1.04 ms so.
static int fit_cluster(int nl) {
  int dev = 0, nsm = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return std::max(1, std::min(8, nsm / std::max(nl, 1)));
}

struct FitWork {
  int* d_bins = nullptr;
  double* d_cnts = nullptr;
  FitBin* d_geo = nullptr;
  int cap_bins = 0;
  double* d_part = nullptr;
  unsigned* d_bar = nullptr;
  FitOut* d_out = nullptr;
  FitOut* h_out = nullptr;   // pinned
  int max_grid = 0;
};

FitWork* fitwork_create() { return new FitWork(); }
void fitwork_destroy(FitWork* fw) {
  if (!fw) return;
  if (fw->d_bins) cudaFree(fw->d_bins);
  if (fw->d_cnts) cudaFree(fw->d_cnts);
  if (fw->d_geo) cudaFree(fw->d_geo);
  if (fw->d_part) cudaFree(fw->d_part);
  if (fw->d_bar) cudaFree(fw->d_bar);
  if (fw->d_out) cudaFree(fw->d_out);
  if (fw->h_out) cudaFreeHost(fw->h_out);
  delete fw;
}

// survfit[b] = mass * S(upper bound of bin b) for b in [cmin, 2 nb), 0 below
// (cov_histogram_SetSurvFitTail, src/covariation.c:1676-1699)
__device__ __forceinline__ double surv_bin(int b, int cmin, double bmin, double w, double mass, int doexp, double mu,
                                           double lambda, double tau, double lga) {
  if (b < cmin) return 0.0;
  const double x = w * (b + 1) + bmin;
  double S;
  if (x <= mu) S = 1.0;
  else if (doexp) S = exp(-lambda * (x - mu));
  else S = gamma_q_dev(tau, lambda * (x - mu), lga);
  return mass * S;
}
__global__ void k_survfit(int cmin, int nb, double bmin, double w, double mass, int doexp, double mu, double lambda,
                          double tau, double lga, double* __restrict__ sf) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < 2 * nb; b += gridDim.x * blockDim.x)
    sf[b] = surv_bin(b, cmin, bmin, w, mass, doexp, mu, lambda, tau, lga);
}

// the gamma survival with two lanes to a bin, a warp to a block: the even
// lane carries the fraction's C, the odd lane its 1/D, so that a step is one
// division of the warp instead of two; the steps' factors -i (i - a) are the
// same for every bin and come from a table.
constexpr int kFracTab = 96;
__global__ void __launch_bounds__(32)
k_survfit_pair(int cmin, int nb, double bmin, double w, double mass, double mu, double lambda, double tau, double lga,
               double* __restrict__ sf) {
  __shared__ double tab[kFracTab];
  const int lane = threadIdx.x, odd = lane & 1, bin = blockIdx.x * 16 + (lane >> 1);
  for (int i = lane; i < kFracTab; i += 32) tab[i] = -(double)(i + 1) * ((double)(i + 1) - tau);
  __syncwarp();
  const double xb = w * (bin + 1) + bmin;
  const double x = xb <= mu ? 0.0 : lambda * (xb - mu);
  const bool in = bin >= cmin && bin < 2 * nb && x > 0.0, frac = in && !(x < tau + 1.0);
  double sum = 0.0;
  if (in && !frac) sum = gamma_q_sum(tau, x);
  __syncwarp();
  if (__any_sync(0xffffffffu, frac)) {
    double b = x + 1.0 - tau;
    double v = 1.0 / b, h = v;
    if (!odd) v = 1.0 / 1e-300;
    bool done = !frac;
    for (int i = 1; i < 10000 && !__all_sync(0xffffffffu, done); i++) {
      const double an = i <= kFracTab ? tab[i - 1] : -(double)i * ((double)i - tau);
      b += 2.0;
      const double t = __fma_rn(an, v, b);
      double den = odd ? t : v;
      const double num = odd ? 1.0 : an;
      double q;
      if (div_range(den) && (__double2hiint(num) & 0x7fffffff) < 0x46293e59) {
        q = div_fast(num, den);
      } else {
        if (odd && fabs(den) < 1e-300) den = 1e-300;
        q = num / den;
      }
      const double s = __dadd_rn(b, q);
      v = odd ? q : s;
      if (!odd && (__double2hiint(v) & 0x7fffffff) < 0x01a56e20 && fabs(v) < 1e-300) v = 1e-300;
      const double del = __dmul_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
      const double hn = __dmul_rn(h, del);
      if (!done) h = hn;
      done = done || __double_as_longlong(del) == 0x3ff0000000000000ll;
    }
    if (frac) sum = h;
  }
  if (bin >= 2 * nb || odd) return;
  double S = 0.0;
  if (bin >= cmin) S = mass * (x > 0.0 ? gamma_q_join(tau, x, sum, gamma_q_lpre(tau, x), lga) : 1.0);
  sf[bin] = S;
}

cudaError_t launch_survfit(int cmin, int nb, double bmin, double w, double mass, int doexp, double mu, double lambda,
                           double tau, double* d_sf, cudaStream_t st) {
  const int n = 2 * nb;
  int dev = 0, nsm = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const double lga = doexp ? 0.0 : std::lgamma(tau);
  // The time is that of the warp with the most FP64 instructions (the bins
  // next to x = tau + 1 take ~60 steps of the fraction, the others ~10): two
  // lanes to a bin until the short warps, several to a scheduler, take as long
  // as that one, then a lane each.  1,440 bins (30 x 61): 69 us a lane per bin
  // with IEEE divisions, 57 us with div_fast, 48 us in pairs.
  if (!doexp && n <= 64 * 4 * nsm) {
    k_survfit_pair<<<std::max(1, (n + 15) / 16), 32, 0, st>>>(cmin, nb, bmin, w, mass, mu, lambda, tau, lga, d_sf);
  } else {
    const int thr = 32 * std::max(1, std::min(8, (n + 32 * nsm - 1) / (32 * nsm)));
    k_survfit<<<std::max(1, std::min(1024, (n + thr - 1) / thr)), thr, 0, st>>>(cmin, nb, bmin, w, mass, doexp, mu,
                                                                            lambda, tau, lga, d_sf);
  }
  return cudaGetLastError();
}

// the start of a gamma fit (moment estimates, log lambda and log tau) and
// the non-empty tail bins; 1 when the tail is empty
static int fit_prepare(const uint64_t* h_obs, int cmin, int imax, double bmin, double w, double mu,
                       std::vector<int>& bins, std::vector<double>& cnts, double* s00, double* s01) {
  double m = 0.0, v = 0.0, n = 0.0;
  bins.clear();
  cnts.clear();
  for (int b = cmin; b <= imax; b++) {
    const double mid = (w * b + bmin) + 0.5 * w - mu;
    n += (double)h_obs[b]; m += (double)h_obs[b] * mid;
    if (h_obs[b]) { bins.push_back(b); cnts.push_back((double)h_obs[b]); }
  }
  if (n <= 0) return 1;
  m /= n;
  for (int b = cmin; b <= imax; b++) {
    const double mid = (w * b + bmin) + 0.5 * w - mu;
    v += (double)h_obs[b] * (mid - m) * (mid - m);
  }
  v /= n;
  if (!(v > 0.0) || !(m > 0.0)) { v = w * w; if (!(m > 0.0)) m = w; }
  *s00 = std::log(m / v);
  *s01 = std::log(m * m / v);
  return 0;
}

// 0 ok, 1 empty tail, 90 CUDA error; the result is read by gamma_fit_collect
// once the stream has passed the launch
int gamma_fit_launch(FitWork* fwp, const uint64_t* h_obs, int cmin, int imax, double bmin, double w, double phi,
                     cudaStream_t st) {
  FitWork& fw = *fwp;
  const double mu = phi;
  std::vector<int> bins;
  std::vector<double> cnts;
  double s00 = 0.0, s01 = 0.0;
  if (fit_prepare(h_obs, cmin, imax, bmin, w, mu, bins, cnts, &s00, &s01)) return 1;

  if (!fw.max_grid) {
    int dev = 0, nsm = 0, occ = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 90;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_gam_fit, 256, 0) != cudaSuccess || !coop || occ < 1)
      return 90;
    fw.max_grid = nsm;   // one block per SM is co-resident
    double inv[64];
    for (int k = 0; k < 64; k++) inv[k] = 1.0 / (k + 1);
    if (cudaMemcpyToSymbol(c_inv, inv, sizeof(inv)) != cudaSuccess) return 90;
    if (cudaMalloc(&fw.d_part, sizeof(double) * 2 * kFitMaxPts * fw.max_grid) != cudaSuccess) return 90;
    if (cudaMalloc(&fw.d_bar, sizeof(unsigned)) != cudaSuccess) return 90;
    if (cudaMalloc(&fw.d_out, sizeof(FitOut)) != cudaSuccess) return 90;
    if (cudaMallocHost(&fw.h_out, sizeof(FitOut)) != cudaSuccess) return 90;
  }
  const int nnz = (int)bins.size();
  if (fw.cap_bins < nnz) {
    if (fw.d_bins) cudaFree(fw.d_bins);
    if (fw.d_cnts) cudaFree(fw.d_cnts);
    if (fw.d_geo) cudaFree(fw.d_geo);
    fw.d_bins = nullptr; fw.d_cnts = nullptr; fw.d_geo = nullptr; fw.cap_bins = 0;
    if (cudaMalloc(&fw.d_bins, sizeof(int) * nnz) != cudaSuccess) return 90;
    if (cudaMalloc(&fw.d_cnts, sizeof(double) * nnz) != cudaSuccess) return 90;
    if (cudaMalloc(&fw.d_geo, sizeof(FitBin) * nnz) != cudaSuccess) return 90;
    fw.cap_bins = nnz;
  }
  if (cudaMemcpyAsync(fw.d_bins, bins.data(), sizeof(int) * nnz, cudaMemcpyHostToDevice, st) != cudaSuccess) return 90;
  if (cudaMemcpyAsync(fw.d_cnts, cnts.data(), sizeof(double) * nnz, cudaMemcpyHostToDevice, st) != cudaSuccess) return 90;
  if (cudaMemsetAsync(fw.d_bar, 0, sizeof(unsigned), st) != cudaSuccess) return 90;

  FitGrid g;
  g.bins = fw.d_bins; g.cnts = fw.d_cnts; g.geo = fw.d_geo; g.nnz = nnz;
  g.bmin = bmin; g.w = w; g.mu = mu;
  g.part = fw.d_part; g.bar = fw.d_bar; g.val = nullptr; g.out = fw.d_out;
  int own = 0;
  void* args[] = {&g, &s00, &s01, &own};
  // one warp per SM until every SM has one, then up to 8 warps per block
  const int nitems = kFitMaxPts * nnz;
  const int W = std::max(1, std::min(8, (nitems + 32 * fw.max_grid - 1) / (32 * fw.max_grid)));
  const int G = std::max(1, std::min(fw.max_grid, (nitems + 32 * W - 1) / (32 * W)));
  own = 32 * W;
  // four or eight warps, for the independent parts of an evaluation
  if (cudaLaunchCooperativeKernel((const void*)k_gam_fit, dim3(G), dim3(own > 128 ? 256 : 128), args, 0, st) !=
      cudaSuccess)
    return 90;
  if (cudaMemcpyAsync(fw.h_out, fw.d_out, sizeof(FitOut), cudaMemcpyDeviceToHost, st) != cudaSuccess) return 90;
  return 0;
}

// 0 ok, 2 barrier timeout, else the search's status
int gamma_fit_collect(FitWork* fwp, double* ret_lambda, double* ret_tau, int* ret_evals) {
  const FitWork& fw = *fwp;
  if (fw.h_out->status) return fw.h_out->status;
  *ret_lambda = fw.h_out->lambda;
  *ret_tau = fw.h_out->tau;
  if (ret_evals) *ret_evals = fw.h_out->evals;
  return 0;
}




// ------------------------------------------------------------------------
// a batch of gamma fits (a cluster of blocks per fit, every search launched at once)
// and the survival tables of a batch of tails
// ------------------------------------------------------------------------
struct FitBatch {
  int cap_fit = 0, cap_bins = 0;
  FitGrid* d_grid = nullptr;
  double2* d_start = nullptr;
  int* d_bins = nullptr;
  double* d_cnts = nullptr;
  FitBin* d_geo = nullptr;
  double* d_val = nullptr;
  double* d_part = nullptr;
  unsigned* d_bar = nullptr;
  FitOut* d_out = nullptr;
  FitOut* h_out = nullptr;   // pinned
  std::vector<int> status;   // per fit: 1 empty tail (not launched)
  std::vector<int> slot;     // per fit: its block, or -1
  bool inv_set = false;
};

FitBatch* fitbatch_create() { return new FitBatch(); }
void fitbatch_destroy(FitBatch* fb) {
  if (!fb) return;
  void* p[] = {fb->d_grid, fb->d_start, fb->d_bins, fb->d_cnts, fb->d_geo, fb->d_val, fb->d_part, fb->d_bar, fb->d_out};
  for (void* x : p) if (x) cudaFree(x);
  if (fb->h_out) cudaFreeHost(fb->h_out);
  delete fb;
}

int gamma_fit_batch_launch(FitBatch* fb, int nfit, const FitReq* req, cudaStream_t st) {
  fb->status.assign(nfit, 0);
  fb->slot.assign(nfit, -1);
  if (!fb->inv_set) {
    double inv[64];
    for (int k = 0; k < 64; k++) inv[k] = 1.0 / (k + 1);
    if (cudaMemcpyToSymbol(c_inv, inv, sizeof(inv)) != cudaSuccess) return 90;
    fb->inv_set = true;
  }
  std::vector<int> bins_all, bins;
  std::vector<double> cnts_all, cnts;
  std::vector<int> boff;
  std::vector<double2> start;
  int nl = 0;
  for (int k = 0; k < nfit; k++) {
    double s00, s01;
    if (fit_prepare(req[k].obs, req[k].cmin, req[k].imax, req[k].bmin, req[k].w, req[k].phi, bins, cnts, &s00,
                    &s01)) {
      fb->status[k] = 1;
      continue;
    }
    fb->slot[k] = nl++;
    boff.push_back((int)bins_all.size());
    bins_all.insert(bins_all.end(), bins.begin(), bins.end());
    cnts_all.insert(cnts_all.end(), cnts.begin(), cnts.end());
    start.push_back(make_double2(s00, s01));
  }
  boff.push_back((int)bins_all.size());
  if (nl == 0) return 0;
  const int nb = (int)bins_all.size();
  if (fb->cap_fit < nl) {
    void* p[] = {fb->d_grid, fb->d_start, fb->d_part, fb->d_bar, fb->d_out};
    for (void* x : p) if (x) cudaFree(x);
    if (fb->h_out) cudaFreeHost(fb->h_out);
    fb->d_grid = nullptr; fb->d_start = nullptr; fb->d_part = nullptr; fb->d_bar = nullptr; fb->d_out = nullptr;
    fb->h_out = nullptr; fb->cap_fit = 0;
    const int cap = std::max(nl, 64);
    if (cudaMalloc(&fb->d_grid, sizeof(FitGrid) * cap) != cudaSuccess ||
        cudaMalloc(&fb->d_start, sizeof(double2) * cap) != cudaSuccess ||
        cudaMalloc(&fb->d_part, sizeof(double) * 2 * kFitMaxPts * cap) != cudaSuccess ||
        cudaMalloc(&fb->d_bar, sizeof(unsigned) * cap) != cudaSuccess ||
        cudaMalloc(&fb->d_out, sizeof(FitOut) * cap) != cudaSuccess ||
        cudaMallocHost(&fb->h_out, sizeof(FitOut) * cap) != cudaSuccess)
      return 90;
    fb->cap_fit = cap;
  }
  if (fb->cap_bins < nb) {
    if (fb->d_bins) cudaFree(fb->d_bins);
    if (fb->d_cnts) cudaFree(fb->d_cnts);
    if (fb->d_geo) cudaFree(fb->d_geo);
    if (fb->d_val) cudaFree(fb->d_val);
    fb->d_val = nullptr;
    fb->d_bins = nullptr; fb->d_cnts = nullptr; fb->d_geo = nullptr; fb->cap_bins = 0;
    const int cap = std::max(nb, 4096);
    if (cudaMalloc(&fb->d_bins, sizeof(int) * cap) != cudaSuccess ||
        cudaMalloc(&fb->d_cnts, sizeof(double) * cap) != cudaSuccess ||
        cudaMalloc(&fb->d_geo, sizeof(FitBin) * cap) != cudaSuccess ||
        cudaMalloc(&fb->d_val, sizeof(double) * kFitMaxPts * cap) != cudaSuccess)
      return 90;
    fb->cap_bins = cap;
  }
  std::vector<FitGrid> grid(nl);
  for (int k = 0; k < nfit; k++) {
    const int e = fb->slot[k];
    if (e < 0) continue;
    FitGrid& g = grid[e];
    g.bins = fb->d_bins + boff[e]; g.cnts = fb->d_cnts + boff[e]; g.geo = fb->d_geo + boff[e];
    g.nnz = boff[e + 1] - boff[e];
    g.bmin = req[k].bmin; g.w = req[k].w; g.mu = req[k].phi;
    g.part = fb->d_part + (size_t)e * 2 * kFitMaxPts;
    g.val = fb->d_val + (size_t)kFitMaxPts * boff[e];
    g.bar = fb->d_bar + e;
    g.out = fb->d_out + e;
  }
  if (cudaMemcpyAsync(fb->d_bins, bins_all.data(), sizeof(int) * nb, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(fb->d_cnts, cnts_all.data(), sizeof(double) * nb, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(fb->d_grid, grid.data(), sizeof(FitGrid) * nl, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(fb->d_start, start.data(), sizeof(double2) * nl, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemsetAsync(fb->d_bar, 0, sizeof(unsigned) * nl, st) != cudaSuccess)
    return 90;
  const int C = fit_cluster(nl);
  if (C == 1) {
    k_gam_fit_grp<false><<<nl, 256, 0, st>>>(fb->d_grid, fb->d_start, 1);
    if (cudaGetLastError() != cudaSuccess) return 90;
  } else {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nl * C);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, k_gam_fit_grp<true>, (const FitGrid*)fb->d_grid, (const double2*)fb->d_start, C) !=
        cudaSuccess)
      return 90;
  }
  if (cudaMemcpyAsync(fb->h_out, fb->d_out, sizeof(FitOut) * nl, cudaMemcpyDeviceToHost, st) != cudaSuccess) return 90;
  return 0;
}

int gamma_fit_batch_collect(FitBatch* fb, int k, double* ret_lambda, double* ret_tau, int* ret_evals) {
  if (fb->status[k]) return fb->status[k];
  const FitOut& o = fb->h_out[fb->slot[k]];
  if (o.status) return o.status;
  *ret_lambda = o.lambda;
  *ret_tau = o.tau;
  if (ret_evals) *ret_evals = o.evals;
  return 0;
}

__global__ void k_survfit_grp(const SurvReq* __restrict__ r, const int* __restrict__ pre, int nr) {
  const int e = grp_find(pre, nr, (int)blockIdx.x);
  const SurvReq& q = r[e];
  const int b = ((int)blockIdx.x - __ldg(pre + e)) * blockDim.x + threadIdx.x;
  if (b >= 2 * q.nb) return;
  q.sf[b] = surv_bin(b, q.cmin, q.bmin, q.w, q.mass, q.doexp, q.mu, q.lambda, q.tau, q.lga);
}

cudaError_t grp_survfit(const SurvReq* d_req, const int* pre, int nr, int nb, cudaStream_t st) {
  if (nb > 0) k_survfit_grp<<<nb, 256, 0, st>>>(d_req, pre, nr);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// helix aggregation of pair p-values (agg_FISHER, agg_LANCASTER,
// agg_WFISHER, agg_SIDAK of src/aggregate.c:141-322): one warp per helix
// ------------------------------------------------------------------------
// y >= 0 with Q(a, y) = p, by doubling then bisection on the upper tail (the
// chi-square quantile of the complement of p, formed without 1 - p)
__device__ double gamma_q_inv(double a, double p) {
  if (!(p > 0.0)) return INFINITY;
  if (p >= 1.0) return 0.0;
  const double lga = lgamma(a);
  double lo = 0.0, hi = fmax(1.0, a);
  for (int k = 0; k < 1000 && gamma_q_dev(a, hi, lga) > p; k++) { lo = hi; hi *= 2.0; }
  for (int k = 0; k < 200 && hi - lo > 1e-15 * hi; k++) {
    const double mid = 0.5 * (lo + hi);
    if (gamma_q_dev(a, mid, lga) > p) lo = mid; else hi = mid;
  }
  return 0.5 * (lo + hi);
}

__global__ void k_aggregate(int method, int nh, const int* __restrict__ off, const double* __restrict__ pval,
                            const double* __restrict__ aux, double* __restrict__ term, double* __restrict__ pagg) {
  const int h = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= nh) return;
  const int a = off[h], n = off[h + 1] - a;
  if (n <= 0) { if (lane == 0) pagg[h] = -1.0; return; }
  if (n == 1) { if (lane == 0) pagg[h] = pval[a]; return; }
  if (method == 1 || method == 2) {
    // weights: Lancaster 1 + substitutions; weighted Fisher (0.01 + power)
    // scaled to sum 2n (extract_rm_weights_*, src/aggregate.c:375-482)
    double wsum = 0.0;
    if (method == 2)
      for (int k = 0; k < n; k++) wsum += 0.01 + aux[a + k];
    const double f = (method == 2 && wsum > 0.0) ? 2.0 * n / wsum : 1.0;
    for (int k = lane; k < n; k += 32) {
      const double w = (method == 1) ? 1.0 + aux[a + k] : (0.01 + aux[a + k]) * f;
      term[2 * (a + k)] = w;
      term[2 * (a + k) + 1] = 2.0 * gamma_q_inv(0.5 * w, pval[a + k]);   // chi-square(w) quantile at 1 - p
    }
  }
  __syncwarp();
  if (lane != 0) return;
  double r;
  if (method == 0) {           // Fisher: chi-square with 2n degrees of freedom
    double chi = 0.0;
    for (int k = 0; k < n; k++) chi += -2.0 * log(pval[a + k]);
    r = isnan(chi) ? NAN : gamma_q_dev((double)n, 0.5 * chi, lgamma((double)n));
  } else if (method == 3) {    // Sidak
    double pmin = pval[a];
    for (int k = 1; k < n; k++) pmin = fmin(pmin, pval[a + k]);
    r = 1.0 - exp((double)n * log(1.0 - pmin));
  } else {                     // Lancaster / weighted Fisher
    double df = 0.0, chi = 0.0;
    for (int k = 0; k < n; k++) df += term[2 * (a + k)];
    for (int k = 0; k < n; k++) chi += term[2 * (a + k) + 1];
    r = isnan(chi) ? NAN : gamma_q_dev(0.5 * df, 0.5 * chi, lgamma(0.5 * df));
  }
  pagg[h] = r;
}

cudaError_t launch_aggregate(int method, int nh, const int* d_off, const double* d_pval, const double* d_aux,
                             double* d_term, double* d_pagg, cudaStream_t st) {
  if (nh <= 0) return cudaSuccess;
  k_aggregate<<<(nh + 7) / 8, 256, 0, st>>>(method, nh, d_off, d_pval, d_aux, d_term, d_pagg);
  return cudaGetLastError();
}

}  // namespace covgpu
