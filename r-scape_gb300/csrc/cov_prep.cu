// cov_prep.cu -- alignment preparation on the device: sequence weights and
// the gap-column filter of an alignment already resident in a context slot.
//
//   k_pb_colinv   per column the counts of the canonical residues and of the
//                 residue types; inv[c][x] = 1/(types * count_x)
//   k_pb_rows     one CTA per sequence: w_s = sum_c inv[c][a_sc] over its
//                 canonical residues (fixed-order block reduction)
//                 -- position-based weights, Henikoff & Henikoff 1994
//                 (esl_msaweight_PB, called at src/R-scape.c:1556 for
//                 nseq > 1000), renormalised to sum to N on the host
//   k_gapfilter   per column the weighted fraction of residues
//                 (ACGU and degenerate codes) among residues and gaps ('-',
//                 '*'; '~' is skipped) against 1 - gapthresh
//                 (msamanip_RemoveGapColumns, src/msamanip.c:461-501)
//   GSC weights   (Gerstein, Sonnhammer & Chothia 1994; esl_msaweight_GSC,
//                 called at src/R-scape.c:1555 for nseq <= 1000):
//     k_gsc_codes  residue codes with non-residues masked to values that
//                  match nothing (0xFE in the row role, 0xFF in the column
//                  role), and the residue count of every sequence
//     k_gsc_ident  32 x 32 tiles of sequence pairs: identities counted four
//                  columns at a time (__vcmpeq4) from shared-memory tiles;
//                  D = 1 - identities / min(len_a, len_b)
//     k_gsc_upgma  UPGMA, all merges in one launch of one cluster of CTAs:
//                  the closest pair of live clusters, ties to the first pair
//                  in row-major order (a < b); each side's new branch shared
//                  among its leaves in proportion to their weights (equally
//                  while those are 0); size-weighted average distances of the
//                  merged cluster (FP64 without contraction, the operations
//                  of the definition)
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <type_traits>

#include "cov_dev.cuh"
#include "cov_div.cuh"
#include "cov_prep.h"
#include "cov_batch.h"
#include "covgpu.h"

namespace covgpu {

// 32 columns by a CTA of 8 words x 32 slices of the sequences: a thread counts
// its word's four columns in packed bytes, emptied into the columns' counters
// before they can overflow.  One thread per column and all N rows in turn took
// 1.5 ms on 64 ragged families (N up to 2,000), 0.1 ms now.
constexpr int PB_COLS = 32;
__host__ __device__ __forceinline__ int pb_blocks_of(int L) { return (L + PB_COLS - 1) / PB_COLS; }
__device__ __forceinline__ void pb_colinv_body(
    const GridIdx g, const uint8_t* __restrict__ ax, int N, int L, int Lp, double* __restrict__ inv) {
  __shared__ int cnt[PB_COLS][4];
  const int tid = threadIdx.x, word = tid & 7, slice = tid >> 3, c0 = g.x * PB_COLS;
  if (tid < PB_COLS * 4) (&cnt[0][0])[tid] = 0;
  __syncthreads();
  const uint8_t* col = ax + c0 + 4 * word;   // Lp is a multiple of 32
  for (int s0 = slice; s0 < N; s0 += 32 * 255) {
    const int s1 = min(N, s0 + 32 * 255);
    uint32_t k[4] = {0, 0, 0, 0};
    for (int s = s0; s < s1; s += 32) {
      const uint32_t v = *reinterpret_cast<const uint32_t*>(col + (int64_t)s * Lp);
#pragma unroll
      for (int x = 0; x < 4; x++) k[x] = __vsub4(k[x], __vcmpeq4(v, 0x01010101u * x));
    }
#pragma unroll
    for (int x = 0; x < 4; x++)
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const int n = (k[x] >> (8 * b)) & 0xFF;
        if (n) atomicAdd(&cnt[4 * word + b][x], n);
      }
  }
  __syncthreads();
  if (tid < PB_COLS && c0 + tid < L) {
    const int* n = cnt[tid];
    const int types = (n[0] > 0) + (n[1] > 0) + (n[2] > 0) + (n[3] > 0);
#pragma unroll
    for (int x = 0; x < 4; x++)
      inv[(int64_t)(c0 + tid) * 4 + x] = (types > 0 && n[x] > 0) ? 1.0 / ((double)types * (double)n[x]) : 0.0;
  }
}
__global__ void __launch_bounds__(256)
k_pb_colinv(const uint8_t* __restrict__ ax, int N, int L, int Lp, double* __restrict__ inv) {
  pb_colinv_body(native_grid(), ax, N, L, Lp, inv);
}

__device__ __forceinline__ void pb_rows_body(
    const GridIdx g, const uint8_t* __restrict__ ax, int L, int Lp, const double* __restrict__ inv,
    double* __restrict__ w) {
  __shared__ double red[8];
  const int s = g.x;
  const uint8_t* row = ax + (int64_t)s * Lp;
  double acc = 0.0;
  for (int c = threadIdx.x; c < L; c += blockDim.x) {
    const int x = row[c];
    if (x < 4) acc += inv[(int64_t)c * 4 + x];
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += red[i];
    w[s] = t;
  }
}
__global__ void __launch_bounds__(256)
k_pb_rows(const uint8_t* __restrict__ ax, int L, int Lp, const double* __restrict__ inv, double* __restrict__ w) {
  pb_rows_body(native_grid(), ax, L, Lp, inv, w);
}

// A column's two sums (residues, residues and gaps) run over the sequences in
// their order in FP64: where the fraction lies on the threshold, the rounding of
// the sums decides, and any other order decides some columns differently.  But
// that chain of additions (~64 cycles each) is needed only there.  So 32 columns
// by a CTA of 8 words x 32 slices of the sequences sum the weights in FP32 first:
// non-negative terms, so the fraction is off by less than (N / 16 + 70) 2^-24 of
// itself, and a fraction further than twice that from the threshold is decided.
// The first warp adds the other columns' weights in order, a lane per (column,
// sum), while the others stage the next rows.  So are all columns where a weight is negative or not finite, the sums
// come near the ends of FP32's range or the threshold is below 1e-6.  Without weights the sums
// are counts, in integers.
// The whole call, weighted / without weights: 30 x 61 40 / 35 us with a thread per
// column that read its rows itself, 23 / 21 so; 2,000 x 1,500 410 / 344, 45 / 29
// so, 97 with every weighted sum in order; 194 with all columns on the threshold.
constexpr int GAP_COLS = 32, GAP_SLICES = 32, GAP_ROWS = 96;
template <bool UNIT>
__global__ void __launch_bounds__(8 * GAP_SLICES)
k_gapfilter(const uint8_t* __restrict__ ax, const double* __restrict__ wgt, int N, int L, int Lp, double idthresh,
            int* __restrict__ useme) {
  typedef typename std::conditional<UNIT, int, float>::type sum_t;
  __shared__ union {
    sum_t part[2][GAP_SLICES][GAP_COLS + 1];
    struct { uint4 code[2][GAP_ROWS][GAP_COLS / 16]; double w[2][GAP_ROWS]; } row;
  } sm;
  __shared__ unsigned some, left;   // columns with a weight other than 0; columns to be summed in order
  __shared__ int odd;               // a weight that is negative or not finite
  const int tid = threadIdx.x, word = tid & 7, slice = tid >> 3, c0 = blockIdx.x * GAP_COLS;
  if (tid == 0) { some = 0u; odd = 0; }
  __syncthreads();
  sum_t r[4] = {0, 0, 0, 0}, t[4] = {0, 0, 0, 0};
  unsigned any = 0u;
  bool bad = false;
  const uint8_t* col = ax + c0 + 4 * word;   // Lp is a multiple of 32
#pragma unroll 4
  for (int s = slice; s < N; s += GAP_SLICES) {
    const uint32_t v = *reinterpret_cast<const uint32_t*>(col + (int64_t)s * Lp);
    sum_t w = 1;
    bool nz = true;
    if constexpr (!UNIT) {
      const double wd = wgt[s];
      const int hi = __double2hiint(wd);
      bad |= (unsigned)hi >= 0x7ff00000u;
      nz = ((hi << 1) | __double2loint(wd)) != 0;
      w = (float)wd;
    }
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const uint32_t x = (v >> (8 * b)) & 0xFFu;
      const bool in = x <= 16;
      t[b] += in ? w : (sum_t)0;
      r[b] += (x <= 15 && x != 4) ? w : (sum_t)0;
      if constexpr (!UNIT) any |= (unsigned)(in && nz) << b;
    }
  }
#pragma unroll
  for (int b = 0; b < 4; b++) { sm.part[0][slice][4 * word + b] = r[b]; sm.part[1][slice][4 * word + b] = t[b]; }
  if (any) atomicOr(&some, any << (4 * word));
  if (bad) odd = 1;
  __syncthreads();
  if (tid < 32) {
    sum_t rs = 0, ts = 0;
    for (int k = 0; k < GAP_SLICES; k++) { rs += sm.part[0][k][tid]; ts += sm.part[1][k][tid]; }
    const bool ok = c0 + tid < L;
    if constexpr (UNIT) {
      if (ok) useme[c0 + tid] = (rs > 0 && (double)rs / (double)ts >= idthresh) ? 1 : 0;
    } else {
      const float id = (float)idthresh, q = rs / ts;
      const float margin = ((float)(N / GAP_SLICES) + 64.f) * 0x1p-22f * fmaxf(q, id);
      const bool none = !odd && !((some >> tid) & 1u);   // no weight at all: neither sum is positive
      const bool sure = none || (!odd && idthresh > 1e-6 && ts > 1e-20f && ts < 1e30f && fabsf(q - id) > margin);
      const unsigned hard = __ballot_sync(0xffffffffu, ok && !sure);
      if (ok && sure) useme[c0 + tid] = !none && q > id;
      if (tid == 0) left = hard;
    }
  }
  if constexpr (!UNIT) {
    __syncthreads();
    unsigned hard = left;
    const int row = tid - 32, k = tid & 15, top = (tid & 16) ? 16 : 15;   // residues up to 15, with gaps 16
    auto stage = [&](int buf, int s) {
      if (row < 0 || row >= GAP_ROWS || s + row >= N) return;
      const uint4* a = reinterpret_cast<const uint4*>(ax + (int64_t)(s + row) * Lp + c0);
      sm.row.code[buf][row][0] = a[0];
      sm.row.code[buf][row][1] = a[1];
      sm.row.w[buf][row] = wgt[s + row];
    };
    while (hard) {   // 16 columns at a time; the same in every thread
      unsigned m = hard;
      for (int j = 0; j < k; j++) m &= m - 1;
      const int c = m ? __ffs(m) - 1 : 0;
      double v = 0.0;
      stage(0, 0);
      __syncthreads();
      int buf = 0;
      for (int s0 = 0; s0 < N; s0 += GAP_ROWS, buf ^= 1) {
        stage(buf ^ 1, s0 + GAP_ROWS);
        if (row < 0) {
          const int n = min(GAP_ROWS, N - s0);
          const uint8_t* code = reinterpret_cast<const uint8_t*>(sm.row.code[buf]) + c;
#pragma unroll 8
          for (int s = 0; s < n; s++) {
            const int x = code[GAP_COLS * s];
            if (x <= top && (x != 4 || top == 16)) v += sm.row.w[buf][s];
          }
        }
        __syncthreads();
      }
      if (row < 0) {
        const double tot = __shfl_down_sync(0xffffffffu, v, 16);
        if (m && top == 15) useme[c0 + c] = (v > 0.0 && v / tot >= idthresh) ? 1 : 0;
      }
      for (int j = 0; j < 16; j++) hard &= hard - 1;
    }
  }
}

__device__ __forceinline__ void gsc_codes_body(
    const GridIdx g, const uint8_t* __restrict__ ax, int N, int L, int Lp, int Lw, uint32_t* __restrict__ ra,
            uint32_t* __restrict__ rb, int* __restrict__ len) {
  __shared__ int red[8];
  const int s = g.x;
  int n = 0;
  for (int w = threadIdx.x; w < Lw; w += blockDim.x) {
    uint32_t va = 0, vb = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int c = 4 * w + k;
      const int x = (c < L) ? ax[(int64_t)s * Lp + c] : 4;
      const bool res = (x < 4) || (x > 4 && x <= 15);
      n += res;
      va |= (uint32_t)(res ? x : 0xFE) << (8 * k);
      vb |= (uint32_t)(res ? x : 0xFF) << (8 * k);
    }
    ra[(int64_t)s * Lw + w] = va;
    rb[(int64_t)s * Lw + w] = vb;
  }
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = n;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += red[i];
    len[s] = t;
  }
}
__global__ void __launch_bounds__(256)
k_gsc_codes(const uint8_t* __restrict__ ax, int N, int L, int Lp, int Lw, uint32_t* __restrict__ ra,
            uint32_t* __restrict__ rb, int* __restrict__ len) {
  gsc_codes_body(native_grid(), ax, N, L, Lp, Lw, ra, rb, len);
}

// D[a][b] for the 32 x 32 tile (g.y, g.x), a < b
__device__ __forceinline__ void gsc_ident_body(
    const GridIdx g, const uint32_t* __restrict__ ra, const uint32_t* __restrict__ rb, const int* __restrict__ len,
    int N, int Lw, double* __restrict__ D) {
  __shared__ uint32_t sa[32][33], sb[32][33];
  const int A0 = g.y * 32, B0 = g.x * 32;
  if (B0 + 31 < A0) return;   // tile entirely below the diagonal
  const int tid = threadIdx.x, ty = tid >> 5, tx = tid & 31;
  int cnt[4] = {0, 0, 0, 0};
  for (int w0 = 0; w0 < Lw; w0 += 32) {
    for (int e = tid; e < 32 * 32; e += 256) {
      const int r = e >> 5, k = e & 31;
      const int a = A0 + r, b = B0 + r, w = w0 + k;
      sa[r][k] = (a < N && w < Lw) ? ra[(int64_t)a * Lw + w] : 0xFEFEFEFEu;
      sb[r][k] = (b < N && w < Lw) ? rb[(int64_t)b * Lw + w] : 0xFFFFFFFFu;
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < 32; k++) {
      const uint32_t y = sb[tx][k];
#pragma unroll
      for (int q = 0; q < 4; q++) cnt[q] += __popc(__vcmpeq4(sa[ty + 8 * q][k], y)) >> 3;
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int a = A0 + ty + 8 * q, b = B0 + tx;
    if (a < N && b < N && a < b) {
      const int mn = min(len[a], len[b]);
      const double d = (mn == 0) ? 1.0 : 1.0 - (double)cnt[q] / (double)mn;
      D[(int64_t)a * N + b] = d;
      D[(int64_t)b * N + a] = d;
    }
  }
}
__global__ void __launch_bounds__(256)
k_gsc_ident(const uint32_t* __restrict__ ra, const uint32_t* __restrict__ rb, const int* __restrict__ len, int N,
            int Lw, double* __restrict__ D) {
  gsc_ident_body(native_grid(), ra, rb, len, N, Lw, D);
}

// Order key of a distance: distances lie in [0, 1] (or +inf), and for
// non-negative doubles the IEEE bit patterns order as the values, so the
// searches compare 64-bit integers (GB300's FP64 pipe is 1/64 of FP32, its
// compares included); NaN and negative values map past every distance.
__device__ __forceinline__ unsigned long long dkey(double d) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(d);
  return (u <= 0x7FF0000000000000ull) ? u : ~0ull;
}
// A merge's distances have one divisor, so they are quotients by div_by: five
// FP64 operations against the general division's several dozen, in a part that
// issues two FP64 operations per cycle and SM.
//
// ------------------------------------------------------------------------
// UPGMA by one cluster of G CTAs, one cluster barrier per merge.
// Index i (row, column, leaf) belongs to CTA i % G.  Every CTA keeps a private
// copy of the clusters' state (size, height, weight sum) and updates it
// identically; each caches the minima of its own rows (the closest live
// column b > a, ties to the smaller b, so the best row minimum in (d, a, b)
// order is the pair a full scan finds) and rescans the ones a merge
// invalidated (their entries were written by the CTA itself or before the last
// barrier).  The merged row's new minimum is not rescanned: every CTA offers
// its best new entry of that row with its next partial, and the reduction
// after the barrier yields both the row's minimum and the next closest pair.
// The partials go straight into the other CTAs' shared memory.
//
// Each row keeps its two closest columns while they are known: a merge that
// removes the first leaves the second, and the merged cluster's distance
// (mostly between the two it replaces) takes its place where it is known to
// come before every other column, so rows are rescanned about a third as
// often.  A lane owns NR rows, columns and leaves, all their state in its
// registers.
//
// Bound by the chain of one merge: the barrier with its release of the stores,
// one round trip to L2 for the two rows (another where a row is rescanned), the
// reductions and eight dependent FP64 operations.  The first warp carries the
// merges alone: one block barrier in the chain, and FP64 work is issued once (a
// warp instruction holds the SM's FP64 pipe for 16 cycles).  The last warp
// follows it with the branch lengths and the leaves' weights; three more take
// part in rescans, whose two round trips and compares held up the whole cluster
// (3.6 ms without them at N=900).
// N=900, the 899 merges: 2.5 ms; one cooperative launch with a barrier in global
// memory per merge took 10.0 ms, 128 equal threads per CTA in a cluster 5.7.
// In a family batch each family has its own cluster: 3.0 ms for 64 ragged
// families; one CTA per family, whose FP64 pipe did every distance of a merge
// with general divisions, took 19.5.
// ------------------------------------------------------------------------
constexpr int GSC_MAXG = 16;
struct __align__(16) GscPart { unsigned long long k, ck; unsigned ab, cb; };

// lexicographic minimum over the warp of (key, tag), in every lane
__device__ __forceinline__ void gsc_warp_min(unsigned long long& k, unsigned& tag) {
  const unsigned full = 0xffffffffu;
  const unsigned hi = (unsigned)(k >> 32), lo = (unsigned)k;
  const unsigned mh = __reduce_min_sync(full, hi);
  const unsigned ml = __reduce_min_sync(full, hi == mh ? lo : full);
  tag = __reduce_min_sync(full, (hi == mh && lo == ml) ? tag : full);
  k = ((unsigned long long)mh << 32) | ml;
}

constexpr size_t GSC_SMEM_MAX = 216 * 1024;   // beside 7 KB of static arrays
// the clusters' sizes as doubles, and the weights warp's state (heights, weight
// sums and sizes, GSC_STATE bytes a sequence), which lies in global memory for
// alignments too deep to hold both (the weights are off the merges' chain)
constexpr size_t GSC_STATE = 2 * sizeof(double) + sizeof(int);
__host__ __device__ __forceinline__ size_t gsc_state_stride(int N) { return (size_t)3 * N; }   // doubles per CTA
static bool gsc_state_global(int N) { return (size_t)N * (sizeof(double) + GSC_STATE) > GSC_SMEM_MAX; }
static size_t gsc_cluster_smem(int N) {
  return (size_t)N * sizeof(double) + (gsc_state_global(N) ? 0 : (size_t)N * GSC_STATE);
}

// the last warp of a CTA: the leaves' weights.  Per merge each side's new
// branch is shared among its leaves in proportion to their weights (equally
// while those are 0); st: heights, weight sums and sizes of the clusters
template <int NR>
__device__ __forceinline__ void gsc_weights(int N, double* __restrict__ w_out, int G, int rank, double* st,
                                            const GscPart (*part)[GSC_MAXG]) {
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu;
  const int nown = (N - rank + G - 1) / G;
  double *height = st, *cw = height + N;
  int* size = reinterpret_cast<int*>(cw + N);
  for (int s = lane; s < N; s += 32) { height[s] = 0.0; cw[s] = 0.0; size[s] = 1; }
  int cl[NR];
  double w[NR];
#pragma unroll
  for (int j = 0; j < NR; j++) { cl[j] = rank + (lane + 32 * j) * G; w[j] = 0.0; }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  for (int m = 0; m < N - 1; m++) {
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    unsigned long long k = lane < G ? part[m & 1][lane].k : ~0ull;
    unsigned ab = lane < G ? part[m & 1][lane].ab : full;
    gsc_warp_min(k, ab);
    if (k == ~0ull) break;   // uniform over the cluster, as in the first warp
    const int ba = (int)(ab >> 16), bb = (int)(ab & 0xFFFFu);
    const double h = __longlong_as_double((long long)k) / 2.0;
    const double ta = cw[ba], tb = cw[bb];
    double bla = h - height[ba], blb = h - height[bb];
    if (bla < 0.0) bla = 0.0;
    if (blb < 0.0) blb = 0.0;
    const int sa = size[ba], sb = size[bb];
    double rec = lane == 0 ? ta : tb;     // both reciprocals at once
    rec = rec > 0.0 ? __drcp_rn(rec) : 0.0;
    const double ra = __shfl_sync(full, rec, 0), rb = __shfl_sync(full, rec, 1);
#pragma unroll
    for (int j = 0; j < NR; j++) {
      if (lane + 32 * j >= nown || (cl[j] != ba && cl[j] != bb)) continue;
      const bool A = cl[j] == ba;
      const double t = A ? ta : tb, bl = A ? bla : blb;
      if (t > 0.0) w[j] += div_by(__dmul_rn(bl, w[j]), t, A ? ra : rb);
      else         w[j] += bl / (double)(A ? sa : sb);
      cl[j] = ba;
    }
    __syncwarp();
    if (lane == 0) { height[ba] = h; cw[ba] = (ta + bla) + (tb + blb); size[ba] = sa + sb; }
    __syncwarp();
  }
#pragma unroll
  for (int j = 0; j < NR; j++)
    if (lane + 32 * j < nown) w_out[rank + (lane + 32 * j) * G] = w[j];
}

// Rescans: the CTA's first warp and three helpers take a quarter of the row
// each.  The two smallest of a lane's columns, then of the warp's, in
// (key, column) order.
constexpr int SCAN_WARPS = 4, SCAN_ROWS = 8;
struct __align__(16) GscTwo { unsigned long long p, q; unsigned pa, qa, pad0, pad1; };
struct GscScan {
  int n;                                   // rows to rescan, -1: the merges are over
  int rows[32 * 32];
  GscTwo res[2][SCAN_ROWS][SCAN_WARPS];
};
__device__ __forceinline__ bool gsc_less(unsigned long long k, unsigned a, unsigned long long k2, unsigned a2) {
  return k < k2 || (k == k2 && a < a2);
}
// the two smallest of two such pairs
__device__ __forceinline__ GscTwo gsc_merge2(const GscTwo& x, const GscTwo& y) {
  const bool f = gsc_less(x.p, x.pa, y.p, y.pa);
  GscTwo r;
  r.p = f ? x.p : y.p; r.pa = f ? x.pa : y.pa;
  const unsigned long long a = f ? x.q : y.q, b = f ? y.p : x.p;
  const unsigned aa = f ? x.qa : y.qa, ba = f ? y.pa : x.pa;
  const bool g = gsc_less(a, aa, b, ba);
  r.q = g ? a : b; r.qa = g ? aa : ba;
  r.pad0 = r.pad1 = 0;
  return r;
}
__device__ __forceinline__ bool gsc_alive(const double* dsz, int s) {
  return reinterpret_cast<const int*>(dsz + s)[1] != 0;
}
// row a's live columns past it by warp k of SCAN_WARPS
__device__ __forceinline__ GscTwo gsc_scan_part(const double* __restrict__ D, int N, int a, const double* dsz, int k,
                                                int lane) {
  const unsigned long long NONE = ~0ull;
  GscTwo r{NONE, NONE, 0xFFFFu, 0xFFFFu, 0, 0};
  const double* row = D + (int64_t)a * N;
  for (int b0 = a + 1 + k * 32 + lane; b0 - lane < N; b0 += 32 * SCAN_WARPS * 8) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; u++)
      v[u] = (b0 + 32 * SCAN_WARPS * u < N) ? __ldcg(row + b0 + 32 * SCAN_WARPS * u) : 0.0;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int b = b0 + 32 * SCAN_WARPS * u;
      const unsigned long long d = dkey(v[u]), key = (b < N && gsc_alive(dsz, b)) ? d : NONE;
      const bool l1 = key < r.p, l2 = key < r.q;   // b ascends: ties keep the smaller first
      r.q = l1 ? r.p : (l2 ? key : r.q);
      r.qa = l1 ? r.pa : (l2 ? (unsigned)b : r.qa);
      r.p = l1 ? key : r.p;
      r.pa = l1 ? (unsigned)b : r.pa;
    }
  }
  unsigned long long m1 = r.p, m2;
  unsigned b1 = r.pa, b2;
  gsc_warp_min(m1, b1);
  const bool won = r.p == m1 && r.pa == b1;
  m2 = won ? r.q : r.p;
  b2 = won ? r.qa : r.pa;
  gsc_warp_min(m2, b2);
  return GscTwo{m1, m2, b1, b2, 0, 0};
}
__device__ __forceinline__ void gsc_scan_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * SCAN_WARPS) : "memory"); }
// one round of up to SCAN_ROWS rows by warp k
__device__ __forceinline__ void gsc_scan_round(const double* D, int N, int G, int rank, const double* dsz, GscScan& sc,
                                               int base, int k, int lane) {
  const int n = min(sc.n - base, SCAN_ROWS);
  for (int i = 0; i < n; i++) {
    const GscTwo r = gsc_scan_part(D, N, rank + sc.rows[base + i] * G, dsz, k, lane);
    if (lane == 0) sc.res[(base / SCAN_ROWS) & 1][i][k] = r;
  }
}

template <int NR>
__device__ __forceinline__ void gsc_cluster_body(double* __restrict__ D, int N, double* __restrict__ w_out, int G,
                                                 int rank, double* state) {
  extern __shared__ __align__(16) unsigned char gsm[];
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu;
  const int nown = (N - rank + G - 1) / G;           // rows/columns/leaves rank, rank + G, ...
  double* dsz = reinterpret_cast<double*>(gsm);      // cluster sizes, 0: dead
  __shared__ GscPart part[2][GSC_MAXG];              // every CTA's partial, by the parity of the merge
  const unsigned long long NONE = ~0ull;
  const unsigned NO = 0xFFFFu, UNK = 0xFFFEu;        // no column; not known
  __shared__ GscScan sc;
  const int warp = threadIdx.x >> 5;
  if (warp == SCAN_WARPS) {   // the weights
    gsc_weights<NR>(N, w_out, G, rank, state ? state + (size_t)rank * gsc_state_stride(N) : dsz + N, part);
    return;
  }
  if (warp == 0) {            // the first scan takes every row
    for (int s = lane; s < N; s += 32) dsz[s] = 1.0;
    for (int r = lane; r < nown; r += 32) sc.rows[r] = r;
    if (lane == 0) sc.n = nown;
  }
  gsc_scan_sync();
  if (warp > 0) {             // the scan helpers
    for (int m = -1; m < N - 1; m++) {
      if (m >= 0) {
        asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        gsc_scan_sync();      // the rows to rescan
      }
      const int n = sc.n;
      if (n < 0) break;
      for (int base = 0; base < n; base += SCAN_ROWS) {
        gsc_scan_round(D, N, G, rank, dsz, sc, base, warp, lane);
        gsc_scan_sync();
      }
      if (m < 0) {
        asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
      }
    }
    return;
  }
  // own rows: the closest column (k1, a1), the second (k2, a2) or a2 = UNK
  unsigned long long k1[NR], k2[NR];
  unsigned a1[NR], a2[NR];
  bool own[NR];                                      // live rows of this lane
#pragma unroll
  for (int j = 0; j < NR; j++) {
    own[j] = lane + 32 * j < nown;
    k1[j] = k2[j] = NONE;
    a1[j] = a2[j] = NO;
  }
  // the scan of the n rows in sc.rows (helpers released already), into the
  // rows' lanes
  auto scan_rows = [&](int n) {
    for (int base = 0; base < n; base += SCAN_ROWS) {
      gsc_scan_round(D, N, G, rank, dsz, sc, base, 0, lane);
      gsc_scan_sync();
      // lane 4 i + k: warp k's part of row i
      GscTwo r = sc.res[(base / SCAN_ROWS) & 1][lane >> 2][lane & 3];
#pragma unroll
      for (int o = 1; o < SCAN_WARPS; o <<= 1) {
        GscTwo y;
        y.p = __shfl_xor_sync(full, r.p, o); y.q = __shfl_xor_sync(full, r.q, o);
        y.pa = __shfl_xor_sync(full, r.pa, o); y.qa = __shfl_xor_sync(full, r.qa, o);
        r = gsc_merge2(r, y);
      }
      const int cnt = min(n - base, SCAN_ROWS);
      for (int i = 0; i < cnt; i++) {
        const unsigned long long p = __shfl_sync(full, r.p, 4 * i), q2 = __shfl_sync(full, r.q, 4 * i);
        const unsigned pa = __shfl_sync(full, r.pa, 4 * i), qa = __shfl_sync(full, r.qa, 4 * i);
        const int row = sc.rows[base + i];
#pragma unroll
        for (int j = 0; j < NR; j++)
          if (lane + 32 * j == row) {
            k1[j] = p; a1[j] = p == NONE ? NO : pa;
            k2[j] = q2; a2[j] = q2 == NONE ? NO : qa;
          }
      }
    }
  };
  scan_rows(nown);
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");   // every CTA has started: its shared memory
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");     // can be written
  int prev = -1;                          // the last merge's row
  unsigned long long ck = NONE;           // this lane's best new entry of row prev
  unsigned cb = NO;
  for (int m = 0; m < N - 1; m++) {
    // the best cached minimum over own live rows, row prev's by the new entries
    unsigned long long qk = ck;
    unsigned qab = ((unsigned)prev << 16) | cb;
#pragma unroll
    for (int j = 0; j < NR; j++) {
      const int a = rank + (lane + 32 * j) * G;
      const unsigned ab = ((unsigned)a << 16) | a1[j];
      if (own[j] && a != prev && (k1[j] < qk || (k1[j] == qk && qk != NONE && ab < qab))) { qk = k1[j]; qab = ab; }
    }
    gsc_warp_min(qk, qab);
    gsc_warp_min(ck, cb);
    if (lane < G) {   // into CTA `lane`'s copy
      uint32_t dst;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst)
                   : "r"((uint32_t)__cvta_generic_to_shared(&part[m & 1][rank])), "r"(lane));
      asm volatile("st.shared::cluster.v2.u64 [%0], {%1, %2};" ::"r"(dst), "l"(qk), "l"(ck) : "memory");
      asm volatile("st.shared::cluster.v2.u32 [%0 + 16], {%1, %2};" ::"r"(dst), "r"(qab), "r"(cb) : "memory");
    }
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    GscPart q = lane < G ? part[m & 1][lane] : GscPart{NONE, NONE, full, NO};
    gsc_warp_min(q.k, q.ab);
    if (q.k == NONE) {         // uniform over the cluster: no pair left
      if (lane == 0) sc.n = -1;
      gsc_scan_sync();
      break;
    }
    const int ba = (int)(q.ab >> 16), bb = (int)(q.ab & 0xFFFFu);
    // the rows of the pair at own columns
    double x[NR], y[NR];
#pragma unroll
    for (int j = 0; j < NR; j++) {
      const int c = rank + (lane + 32 * j) * G;
      x[j] = own[j] ? __ldcg(D + (int64_t)ba * N + c) : 0.0;
      y[j] = own[j] ? __ldcg(D + (int64_t)bb * N + c) : 0.0;
    }
    if (prev >= 0 && prev % G == rank) {   // row prev's minimum, for its owner
      gsc_warp_min(q.ck, q.cb);
      const int r = prev / G;
#pragma unroll
      for (int j = 0; j < NR; j++)
        if (lane + 32 * j == r) { k1[j] = q.ck; a1[j] = q.ck == NONE ? NO : q.cb; a2[j] = UNK; }
    }
    const double sa = dsz[ba], sb = dsz[bb], n = sa + sb, rn = __drcp_rn(n);
    // own columns: the merged cluster's distances, the two closest of own
    // rows, and this lane's best new entry of row ba
    ck = NONE; cb = NO;
    unsigned lost = 0u;
#pragma unroll
    for (int j = 0; j < NR; j++)   // the lane's chains together; 0 for columns it does not own
      x[j] = div_by(__dadd_rn(__dmul_rn(x[j], sa), __dmul_rn(y[j], sb)), n, rn);
#pragma unroll
    for (int j = 0; j < NR; j++) {
      const int c = rank + (lane + 32 * j) * G;
      if (c == bb) own[j] = false;
      if (own[j] && c != ba) {
        __stcg(D + (int64_t)ba * N + c, x[j]);
        __stcg(D + (int64_t)c * N + ba, x[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < NR; j++) {
      const int c = rank + (lane + 32 * j) * G;
      if (!own[j] || c == ba) continue;
      const unsigned long long kd = dkey(x[j]);
      if (c > ba && kd < ck) { ck = kd; cb = (unsigned)c; }
      if (c > bb || k1[j] == NONE) continue;          // the row holds neither column
      const bool low = c < ba;                        // column ba changes as well as bb going
      const bool rem1 = a1[j] == (unsigned)bb || (low && a1[j] == (unsigned)ba);
      const bool known2 = a2[j] != UNK;
      const bool rem2 = a2[j] == (unsigned)bb || (low && a2[j] == (unsigned)ba);
      // every column not listed comes after (kb, ab)
      const unsigned long long kb = known2 ? k2[j] : k1[j];
      const unsigned ab = known2 ? a2[j] : a1[j];
      if (rem1) {
        if (known2 && !rem2) { k1[j] = k2[j]; a1[j] = a2[j]; }
        else a1[j] = UNK;
        a2[j] = UNK;
      } else if (rem2) {
        a2[j] = UNK;
      }
      if (low && (kd < kb || (kd == kb && (unsigned)ba < ab) || ab == NO)) {   // in its place among the listed
        if (a1[j] == UNK) { k1[j] = kd; a1[j] = (unsigned)ba; }
        else if (kd < k1[j] || (kd == k1[j] && (unsigned)ba < a1[j])) {
          k2[j] = k1[j]; a2[j] = a1[j]; k1[j] = kd; a1[j] = (unsigned)ba;
        } else if (a2[j] == UNK || kd < k2[j] || (kd == k2[j] && (unsigned)ba < a2[j])) {
          k2[j] = kd; a2[j] = (unsigned)ba;
        }
      }
      if (a1[j] == UNK) lost |= 1u << j;
    }
    __syncwarp();
    if (lane == 0) { dsz[ba] = n; dsz[bb] = 0.0; }
    __syncwarp();
    // rescans of own rows whose minimum was lost (their entries are this CTA's
    // own writes or older than the last barrier)
    int nl = 0;
#pragma unroll
    for (int j = 0; j < NR; j++) {
      const unsigned lm = __ballot_sync(full, (lost >> j) & 1u);
      if ((lost >> j) & 1u) sc.rows[nl + __popc(lm & ((1u << lane) - 1u))] = lane + 32 * j;
      nl += __popc(lm);
    }
    if (lane == 0) sc.n = nl;
    gsc_scan_sync();
    scan_rows(nl);
    prev = ba;
  }
}

template <int NR>
__global__ void __launch_bounds__(32 * (SCAN_WARPS + 1))
k_gsc_upgma(double* __restrict__ D, int N, double* __restrict__ w, int G, double* state) {
  gsc_cluster_body<NR>(D, N, w, G, blockIdx.x % G, state);
}

// Rows per lane at most.  R-scape's rule takes these weights up to 1,000
// sequences (two rows); 5 to 8 rows run in the kernel of 16.
constexpr int GSC_MAXR = 32;
// f(rows per lane) of the merges' kernel for N sequences
template <class F>
static cudaError_t gsc_with_nr(int nr, F f) {
  switch (nr) {
    case 1: return f(std::integral_constant<int, 1>());
    case 2: return f(std::integral_constant<int, 2>());
    case 4: return f(std::integral_constant<int, 4>());
    case 16: return f(std::integral_constant<int, 16>());
    case GSC_MAXR: return f(std::integral_constant<int, GSC_MAXR>());
  }
  return cudaErrorInvalidValue;
}

static void gsc_launch_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* la, int grid, int G, size_t sm,
                              cudaStream_t st) {
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(32 * (SCAN_WARPS + 1));
  cfg.dynamicSmemBytes = sm;
  cfg.stream = st;
  la[0].id = cudaLaunchAttributeClusterDimension;
  la[0].val.clusterDim.x = G;
  la[0].val.clusterDim.y = la[0].val.clusterDim.z = 1;
  cfg.attrs = la;
  cfg.numAttrs = 1;
}
template <class... A>
static cudaError_t gsc_cluster_launch(const void* k, int grid, int G, size_t sm, cudaStream_t st, A... a) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute la[1];
  gsc_launch_config(cfg, la, grid, G, sm, st);
  void* args[] = {(void*)&a...};
  return cudaLaunchKernelExC(&cfg, k, args);
}

// the merge kernels' limits (shared memory, clusters of 16) on the current
// device, raised once (before any stream capture), and the largest cluster
// that the device places
static cudaError_t gsc_attrs(int* max_cluster);

size_t gsc_scratch_bytes(int N, int L) {
  const size_t Lw = ((size_t)L + 3) / 4;
  return (size_t)N * N * sizeof(double) + 2 * (size_t)N * Lw * sizeof(uint32_t) + (size_t)N * sizeof(int) + 512 +
         (gsc_state_global(N) ? GSC_MAXG * gsc_state_stride(N) * sizeof(double) : 0);
}

cudaError_t launch_weights_gsc(const uint8_t* ax, int N, int L, int Lp, void* scratch, double* w, cudaStream_t st) {
  const int Lw = (L + 3) / 4;
  uint8_t* p = (uint8_t*)scratch;
  double* D = (double*)p;                 p += (size_t)N * N * sizeof(double);
  double* state = nullptr;
  if (gsc_state_global(N)) { state = (double*)p; p += GSC_MAXG * gsc_state_stride(N) * sizeof(double); }
  uint32_t* ra = (uint32_t*)p;            p += (size_t)N * Lw * sizeof(uint32_t);
  uint32_t* rb = (uint32_t*)p;            p += (size_t)N * Lw * sizeof(uint32_t);
  int* len = (int*)p;
  int maxc = 0, G = 0, nr = 0;
  const cudaError_t e = gsc_attrs(&maxc);
  if (e != cudaSuccess) return e;
  if (N < 2 || covgpu_gsc_shape(N, maxc, &G, &nr)) return cudaErrorInvalidValue;
  k_gsc_codes<<<N, 256, 0, st>>>(ax, N, L, Lp, Lw, ra, rb, len);
  const int nt = (N + 31) / 32;
  k_gsc_ident<<<dim3(nt, nt), 256, 0, st>>>(ra, rb, len, N, Lw, D);
  // all merges in one launch of one cluster
  return gsc_with_nr(nr, [&](auto rows) {
    return gsc_cluster_launch((const void*)k_gsc_upgma<decltype(rows)::value>, G, G, gsc_cluster_smem(N), st, D, N, w, G,
                              state);
  });
}

cudaError_t launch_weights_pb(const uint8_t* ax, int N, int L, int Lp, double* inv, double* w, cudaStream_t st) {
  k_pb_colinv<<<pb_blocks_of(L), 256, 0, st>>>(ax, N, L, Lp, inv);
  k_pb_rows<<<N, 256, 0, st>>>(ax, L, Lp, inv, w);
  return cudaGetLastError();
}

cudaError_t launch_gapfilter(const uint8_t* ax, const double* wgt, int N, int L, int Lp, double gapthresh, int* useme,
                             cudaStream_t st) {
  const int nb = (L + GAP_COLS - 1) / GAP_COLS, thr = 8 * GAP_SLICES;
  if (wgt) k_gapfilter<false><<<nb, thr, 0, st>>>(ax, wgt, N, L, Lp, 1.0 - gapthresh, useme);
  else     k_gapfilter<true><<<nb, thr, 0, st>>>(ax, wgt, N, L, Lp, 1.0 - gapthresh, useme);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// grouped launches over a batch of families: position-based weights of the
// families with pb set, GSC weights (a cluster per family for the merges) of
// those with gsc set
// ------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
k_pb_colinv_grp(const FamDev* __restrict__ F, int nf, const int* __restrict__ pre) {
  const int f = grp_find(pre, nf, (int)blockIdx.x);
  const FamDev& d = F[f];
  pb_colinv_body(GridIdx{(int)blockIdx.x - __ldg(pre + f), 0, pb_blocks_of(d.L)}, d.ax, d.N, d.L, d.Lp, d.pbinv);
}

__global__ void __launch_bounds__(256)
k_pb_rows_grp(const FamDev* __restrict__ F, int nf, const int* __restrict__ pre) {
  const int f = grp_find(pre, nf, (int)blockIdx.x);
  const FamDev& d = F[f];
  pb_rows_body(GridIdx{(int)blockIdx.x - __ldg(pre + f), 0, d.N}, d.ax, d.L, d.Lp, d.pbinv, d.w);
}

__global__ void __launch_bounds__(256)
k_gsc_codes_grp(const FamDev* __restrict__ F, int nf, const int* __restrict__ pre) {
  const int f = grp_find(pre, nf, (int)blockIdx.x);
  const FamDev& d = F[f];
  gsc_codes_body(GridIdx{(int)blockIdx.x - __ldg(pre + f), 0, d.N}, d.ax, d.N, d.L, d.Lp, d.Lw, d.gra, d.grb, d.glen);
}

__global__ void __launch_bounds__(256)
k_gsc_ident_grp(const FamDev* __restrict__ F, int nf, const int* __restrict__ pre) {
  const int f = grp_find(pre, nf, (int)blockIdx.x);
  const FamDev& d = F[f];
  const int nt = (d.N + 31) / 32, loc = (int)blockIdx.x - __ldg(pre + f);
  gsc_ident_body(GridIdx{loc % nt, loc / nt, nt}, d.gra, d.grb, d.glen, d.N, d.Lw, d.gD);
}

template <int NR>
__global__ void __launch_bounds__(32 * (SCAN_WARPS + 1))
k_gsc_upgma_grp(const FamDev* __restrict__ F, int nf, const int* __restrict__ pre, int G) {
  const int f = grp_find(pre, nf, (int)blockIdx.x / G);
  const FamDev& d = F[f];
  gsc_cluster_body<NR>(d.gD, d.N, d.w, G, (int)blockIdx.x % G, nullptr);
}

static cudaError_t gsc_attrs(int* max_cluster) {
  constexpr int MAXDEV = 64;
  static std::atomic<int> known[MAXDEV];   // the largest cluster, 0: not asked yet
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < MAXDEV && (*max_cluster = known[dev].load()) > 0) return cudaSuccess;
  const void* k[] = {(const void*)k_gsc_upgma<1>, (const void*)k_gsc_upgma<2>, (const void*)k_gsc_upgma<4>,
                     (const void*)k_gsc_upgma<16>, (const void*)k_gsc_upgma<32>, (const void*)k_gsc_upgma_grp<1>,
                     (const void*)k_gsc_upgma_grp<2>, (const void*)k_gsc_upgma_grp<4>,
                     (const void*)k_gsc_upgma_grp<16>, (const void*)k_gsc_upgma_grp<32>};
  int maxc = GSC_MAXG;
  for (const void* f : k) {
    if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GSC_SMEM_MAX)) != cudaSuccess)
      return e;
    if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess) return e;
    // 16 CTAs with the most shared memory that they may take in one GPC?
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute la[1];
    gsc_launch_config(cfg, la, GSC_MAXG, GSC_MAXG, GSC_SMEM_MAX, nullptr);
    if (cudaOccupancyMaxActiveClusters(&n, f, &cfg) != cudaSuccess || n < 1) {
      (void)cudaGetLastError();
      maxc = 8;
    }
  }
  if (dev < MAXDEV) known[dev].store(maxc);
  *max_cluster = maxc;
  return cudaSuccess;
}

int pb_blocks(int L) { return pb_blocks_of(L); }

cudaError_t grp_weights_pb(const FamDev* F, int nf, const int* pre_col, int nb_col, const int* pre_row, int nb_row,
                           cudaStream_t st) {
  if (nb_col > 0) k_pb_colinv_grp<<<nb_col, 256, 0, st>>>(F, nf, pre_col);
  if (nb_row > 0) k_pb_rows_grp<<<nb_row, 256, 0, st>>>(F, nf, pre_row);
  return cudaGetLastError();
}

// maxN: the largest N among the GSC families (the merges' shared memory)
cudaError_t grp_weights_gsc(const FamDev* F, int nf, const int* pre_codes, int nb_codes, const int* pre_ident,
                            int nb_ident, const int* pre_upgma, int nb_upgma, int maxN, cudaStream_t st) {
  if (nb_upgma <= 0) return cudaSuccess;
  int maxc = 0, G = 0, nr = 0;
  if (gsc_state_global(maxN) || gsc_attrs(&maxc) != cudaSuccess || covgpu_gsc_shape(maxN, maxc, &G, &nr))
    return cudaErrorInvalidValue;
  if (nb_codes > 0) k_gsc_codes_grp<<<nb_codes, 256, 0, st>>>(F, nf, pre_codes);
  if (nb_ident > 0) k_gsc_ident_grp<<<nb_ident, 256, 0, st>>>(F, nf, pre_ident);
  return gsc_with_nr(nr, [&](auto rows) {
    return gsc_cluster_launch((const void*)k_gsc_upgma_grp<decltype(rows)::value>, nb_upgma * G, G,
                              gsc_cluster_smem(maxN), st, F, nf, pre_upgma, G);
  });
}

// the device weights of each family of pre (one block each), made as the
// host makes a caller's weights: normalised to sum to N (the sum in sequence
// order), then quantised to three b-bit limbs as make_limbs does
// (cov_kernels.cu) in its general form -- normalised weights that are all
// equal are all 1.0, whose limbs give the same counts as the one-limb form.
// Writes the limbs (uint16 [3][Npad], zero-padded, and as floats [3][N]) and
// the family's limb base, scale and quantised total into F and U.
__global__ void __launch_bounds__(256)
k_weights_limbs_grp(FamDev* __restrict__ F, int nf, const int* __restrict__ pre, UmmaFam* __restrict__ U) {
  const int f = grp_find(pre, nf, (int)blockIdx.x);
  FamDev& d = F[f];
  const int N = d.N, tid = threadIdx.x;
  __shared__ double ssum, red[256];
  __shared__ unsigned long long tot;
  __shared__ int sE, sb;
  if (tid == 0) {
    double sum = 0.0;
    for (int i = 0; i < N; i++) sum = __dadd_rn(sum, d.w[i]);
    ssum = sum;
    tot = 0ull;
  }
  __syncthreads();
  const double sum = ssum;
  double wmax = 0.0;
  for (int i = tid; i < N; i += blockDim.x) {
    const double w = (sum > 0.0) ? __ddiv_rn(__dmul_rn(d.w[i], (double)N), sum) : 1.0;
    d.w[i] = w;
    wmax = fmax(wmax, w);
  }
  red[tid] = wmax;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (tid < o) red[tid] = fmax(red[tid], red[tid + o]);
    __syncthreads();
  }
  if (tid == 0) {
    int b = 11;
    while (b > 1 && (double)N * (double)((1 << b) - 1) >= 16777216.0) b--;
    int e2;
    frexp(red[0], &e2);
    sb = b;
    sE = 3 * b - e2;
  }
  __syncthreads();
  const int b = sb, E = sE;
  const double qmax = ldexp(1.0, 3 * b) - 1.0;
  const unsigned long long mask = (1ull << b) - 1ull;
  unsigned long long t = 0;
  for (int i = tid; i < d.Npad; i += blockDim.x) {
    unsigned long long q = 0;
    if (i < N) {
      double qd = rint(ldexp(d.w[i], E));
      if (qd > qmax) qd = qmax;
      q = (unsigned long long)qd;
    }
    const uint16_t l0 = (uint16_t)(q & mask), l1 = (uint16_t)((q >> b) & mask), l2 = (uint16_t)(q >> (2 * b));
    d.limbs[i] = l0;
    d.limbs[d.Npad + i] = l1;
    d.limbs[2 * d.Npad + i] = l2;
    if (i < N) {
      d.limbf[i] = (float)l0;
      d.limbf[N + i] = (float)l1;
      d.limbf[2 * N + i] = (float)l2;
    }
    t += q;
  }
  atomicAdd(&tot, t);
  __syncthreads();
  if (tid == 0) {
    const float B = (float)(1 << b), s_hi = (float)ldexp(1.0, -E);
    const double wq = ldexp((double)tot, -E);
    const float whi = (float)wq;
    d.nl = 3; d.B = B; d.s_hi = s_hi; d.s_lo = 0.f;
    d.sa.wtot = make_float2(whi, (float)(wq - (double)whi));
    U[f].B = B; U[f].s_hi = s_hi; U[f].s_lo = 0.f;
  }
}

cudaError_t grp_weights_limbs(FamDev* F, int nf, const int* pre, int nb, UmmaFam* U, cudaStream_t st) {
  if (nb > 0) k_weights_limbs_grp<<<nb, 256, 0, st>>>(F, nf, pre, U);
  return cudaGetLastError();
}

// the merges' limits, raised outside any stream capture
int grp_weights_gsc_prepare() {
  int maxc;
  return gsc_attrs(&maxc) == cudaSuccess ? 1 : 0;
}

int gsc_max_sequences() {
  int maxc = 0;
  return gsc_attrs(&maxc) == cudaSuccess ? 32 * GSC_MAXR * maxc : 0;
}

// rows of L bytes, one after the other, to a pitch of Lp: 16 bytes of a row
// per thread, from the aligned words around them (src: aligned, readable for
// 20 bytes past the last row); columns L .. Lp - 1 are left alone.  Bound by
// memory: 60 MB moved at 20000 x 1500.
__global__ void __launch_bounds__(256)
k_spread_rows(const uint8_t* __restrict__ src, int64_t N, int L, int Lp, uint8_t* __restrict__ dst) {
  const int per = Lp >> 4;
  const int64_t it = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= N * per) return;
  const int64_t r = it / per;
  const int c = (int)(it - r * per) << 4;
  if (c >= L) return;
  const int64_t o = r * L + c;
  const uint32_t* w = reinterpret_cast<const uint32_t*>(src + (o & ~(int64_t)3));
  const int sh = (int)(o & 3) * 8;
  uint32_t v[5];
#pragma unroll
  for (int k = 0; k < 5; k++) v[k] = __ldg(w + k);
#pragma unroll
  for (int k = 0; k < 4; k++) v[k] = __funnelshift_r(v[k], v[k + 1], sh);
  uint8_t* d = dst + r * Lp + c;
  if (c + 16 <= L) {
    *reinterpret_cast<uint4*>(d) = make_uint4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int k = 0; k < 16; k++)
      if (c + k < L) d[k] = (uint8_t)(v[k >> 2] >> (8 * (k & 3)));
  }
}

cudaError_t launch_spread_rows(const uint8_t* src, int N, int L, int Lp, uint8_t* dst, cudaStream_t st) {
  const int64_t items = (int64_t)N * (Lp >> 4);
  k_spread_rows<<<(unsigned)((items + 255) / 256), 256, 0, st>>>(src, N, L, Lp, dst);
  return cudaGetLastError();
}

}  // namespace covgpu

// CTAs of the merges' cluster: 16 for more than 256 sequences where the device
// places such a cluster (16 is beyond the portable size), else 8; rows per
// lane: the smallest kernel that holds N
extern "C" int covgpu_gsc_shape(int N, int max_cluster, int* ctas, int* rows) {
  if (N < 1 || max_cluster < 8 || !ctas || !rows) return 11;
  *ctas = (N <= 256 || max_cluster < covgpu::GSC_MAXG) ? 8 : covgpu::GSC_MAXG;
  const int need = (N + 32 * *ctas - 1) / (32 * *ctas);
  for (int r : {1, 2, 4, 16, covgpu::GSC_MAXR})
    if (need <= r) { *rows = r; return 0; }
  return 11;
}
