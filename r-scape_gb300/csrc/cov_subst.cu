// cov_subst.cu -- substitutions on the tree and the power of every pair.
//
// Tree_Substitutions (src/msatree.c:1423-1554) on the Fitch reconstruction
// of the alignment: for every branch (parent v -> child) and column c, bit
// s = the child's residue differs from the parent's (both canonical unless
// gaps are included) and bit u = both canonical and equal; the bits of 32
// branches pack one word, so per column
//   nsubs[c]     = sum popc(s_c)
// and per pair i < j
//   ndouble[i,j] = sum popc(s_i & s_j)                 (both change)
//   njoin[i,j]   = sum popc((s|u)_i & (s|u)_j) - popc(u_i & u_j)
//                  (both canonical, at least one changes; with gaps
//                  included: sum popc(s_i | s_j))
// computed in 32 x 32 tiles of pairs from shared-memory word tiles.
//
// power_SPAIR_Create (src/power.c:65-218): the power of a pair is the step
// curve's probability at its substitution count (nsubs_i + nsubs_j, njoin,
// ndouble): the last point whose count the pair's exceeds.
#include <cuda_runtime.h>

#include <cstdint>

#include "cov_subst.h"

namespace covgpu {

// one thread per (column, word of 32 branches), columns fastest
__global__ void __launch_bounds__(256)
k_subst_bits(const uint8_t* __restrict__ ax, const uint8_t* __restrict__ F, const int* __restrict__ left,
             const int* __restrict__ right, int N, int L, int Lp, int Wb, int includegaps, uint32_t* __restrict__ Sb,
             uint32_t* __restrict__ Ub) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)Wb * L) return;
  const int k = (int)(idx / L), c = (int)(idx % L);
  const int nb = 2 * (N - 1);
  uint32_t s = 0, u = 0;
  for (int t = 0; t < 32; t++) {
    const int e = 32 * k + t;
    if (e >= nb) break;
    const int v = e >> 1;
    const int ch = (e & 1) ? right[v] : left[v];
    const int a = F[(int64_t)v * Lp + c];
    const int b = (ch > 0) ? F[(int64_t)ch * Lp + c] : ax[(int64_t)(-ch) * Lp + c];
    if (includegaps) {
      s |= (uint32_t)(a != b) << t;
      u |= (uint32_t)(a == b) << t;
    } else {
      const bool can = a < 4 && b < 4;
      s |= (uint32_t)(can && a != b) << t;
      u |= (uint32_t)(can && a == b) << t;
    }
  }
  Sb[(int64_t)c * Wb + k] = s;
  Ub[(int64_t)c * Wb + k] = u;
}

__global__ void __launch_bounds__(256)
k_subst_nsubs(const uint32_t* __restrict__ Sb, int L, int Wb, int* __restrict__ nsubs) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= L) return;
  int n = 0;
  for (int k = 0; k < Wb; k++) n += __popc(Sb[(int64_t)c * Wb + k]);
  nsubs[c] = n;
}

// the upper triangle (i < j) of ndouble and njoin, tile (blockIdx.y, blockIdx.x)
__global__ void __launch_bounds__(256)
k_subst_pairs(const uint32_t* __restrict__ Sb, const uint32_t* __restrict__ Ub, int L, int Wb, int includegaps,
              int* __restrict__ ndouble, int* __restrict__ njoin) {
  __shared__ uint32_t si[32][33], ui[32][33], sj[32][33], uj[32][33];
  const int I0 = blockIdx.y * 32, J0 = blockIdx.x * 32;
  if (J0 + 31 <= I0) return;   // no pair i < j in this tile
  const int tid = threadIdx.x, ty = tid >> 5, tx = tid & 31;
  int dbl[4] = {0, 0, 0, 0}, cc[4] = {0, 0, 0, 0}, uu[4] = {0, 0, 0, 0};
  for (int w0 = 0; w0 < Wb; w0 += 32) {
    for (int e = tid; e < 32 * 32; e += 256) {
      const int r = e >> 5, k = e & 31, w = w0 + k;
      const int i = I0 + r, j = J0 + r;
      si[r][k] = (i < L && w < Wb) ? Sb[(int64_t)i * Wb + w] : 0u;
      ui[r][k] = (i < L && w < Wb) ? Ub[(int64_t)i * Wb + w] : 0u;
      sj[r][k] = (j < L && w < Wb) ? Sb[(int64_t)j * Wb + w] : 0u;
      uj[r][k] = (j < L && w < Wb) ? Ub[(int64_t)j * Wb + w] : 0u;
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < 32; k++) {
      const uint32_t b_s = sj[tx][k], b_u = uj[tx][k];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint32_t a_s = si[ty + 8 * q][k], a_u = ui[ty + 8 * q][k];
        dbl[q] += __popc(a_s & b_s);
        if (includegaps) {
          cc[q] += __popc(a_s | b_s);
        } else {
          cc[q] += __popc((a_s | a_u) & (b_s | b_u));
          uu[q] += __popc(a_u & b_u);
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int i = I0 + ty + 8 * q, j = J0 + tx;
    if (i < j && j < L) {
      ndouble[(int64_t)i * L + j] = dbl[q];
      njoin[(int64_t)i * L + j] = cc[q] - uu[q];
    }
  }
}

__device__ __forceinline__ double step_power(double n, const double* __restrict__ subs, const double* __restrict__ prob,
                                             int ns) {
  double p = 0.0;
  for (int s = 0; s < ns; s++) {
    if (n > subs[s]) p = prob[s];
    else break;
  }
  return p;
}

// F[k][n], n < T: curve k at n substitutions (step_power), a warp per entry:
// 32 points at a time, the first that n does not exceed found by a vote (a
// thread scanning the points one after the other: 33 us for 701 x 650 and 200
// points, 6.5 us so)
__global__ void __launch_bounds__(256)
k_power_table(int ns, const double* __restrict__ tab, int T, double* __restrict__ F) {
  const int e = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (e >= 3 * T) return;
  const int k = e / T, n = e - k * T;
  const double *subs = tab + 2 * k * ns, *prob = subs + ns;
  int last = ns;   // points that n exceeds before the first that it does not
  for (int s0 = 0; s0 < ns; s0 += 32) {
    const bool stop = s0 + lane < ns && !((double)n > subs[s0 + lane]);
    const unsigned m = __ballot_sync(0xffffffffu, stop);
    if (m) { last = s0 + __ffs(m) - 1; break; }
  }
  if (lane == 0) F[e] = last > 0 ? prob[last - 1] : 0.0;
}

// pair n = (i, j), i < j, in row-major order of the upper triangle.  The
// counts are integers, so the curves are tabled at 0 .. T - 1 substitutions
// (k_power_table; T 0: no table) and a pair takes three look-ups instead of
// three scans of FP64 comparisons; a count beyond the table is scanned.
// Bound by memory then: 701 x 650 with curves of 200 points 38 us scanned,
// 5.6 + 6.5 us tabled.
__global__ void __launch_bounds__(256)
k_power(const int* __restrict__ nsubs, const int* __restrict__ ndouble, const int* __restrict__ njoin, int L,
        int ns, const double* __restrict__ tab, int T, const double* __restrict__ F, int have_single, int have_join,
        int have_double, double* __restrict__ power, double* __restrict__ power_join,
        double* __restrict__ power_double) {
  const int i = blockIdx.y;
  const int64_t base = (int64_t)i * L - (int64_t)i * (i + 1) / 2;   // pairs before row i
  auto curve = [&](int k, int n) {
    return ((unsigned)n < (unsigned)T) ? __ldg(F + (size_t)k * T + n)
                                       : step_power((double)n, tab + 2 * k * ns, tab + (2 * k + 1) * ns, ns);
  };
  for (int j = i + 1 + blockIdx.x * blockDim.x + threadIdx.x; j < L; j += gridDim.x * blockDim.x) {
    const int64_t n = base + (j - i - 1);
    if (power) power[n] = have_single ? curve(0, nsubs[i] + nsubs[j]) : 0.0;
    if (power_join) power_join[n] = have_join ? curve(1, njoin[(int64_t)i * L + j]) : -1.0;
    if (power_double) power_double[n] = have_double ? curve(2, ndouble[(int64_t)i * L + j]) : -1.0;
  }
}

cudaError_t launch_substitutions(const uint8_t* ax, const uint8_t* F, const int* left, const int* right, int N, int L,
                                 int Lp, int includegaps, uint32_t* Sb, uint32_t* Ub, int* nsubs, int* ndouble,
                                 int* njoin, cudaStream_t st) {
  const int Wb = (2 * (N - 1) + 31) / 32;
  const int64_t items = (int64_t)Wb * L;
  k_subst_bits<<<(unsigned)((items + 255) / 256), 256, 0, st>>>(ax, F, left, right, N, L, Lp, Wb, includegaps, Sb, Ub);
  k_subst_nsubs<<<(L + 255) / 256, 256, 0, st>>>(Sb, L, Wb, nsubs);
  cudaMemsetAsync(ndouble, 0, (size_t)L * L * sizeof(int), st);
  cudaMemsetAsync(njoin, 0, (size_t)L * L * sizeof(int), st);
  const int nt = (L + 31) / 32;
  k_subst_pairs<<<dim3(nt, nt), 256, 0, st>>>(Sb, Ub, L, Wb, includegaps, ndouble, njoin);
  return cudaGetLastError();
}

// counts that the curves are tabled for: up to 4 (N - 1) (two columns'
// substitutions on 2 (N - 1) branches), where there are more pairs to look up
// than entries to fill
int power_table_size(int N, int L) {
  const int64_t T = 4 * ((int64_t)N - 1) + 1, P = (int64_t)L * (L - 1) / 2;
  return (T > 0 && T < P) ? (int)T : 0;
}

cudaError_t launch_power(const int* nsubs, const int* ndouble, const int* njoin, int L, int ns, const double* tab,
                         int T, double* F, int have_single, int have_join, int have_double, double* power,
                         double* power_join, double* power_double, cudaStream_t st) {
  if (T > 0) k_power_table<<<(3 * T + 7) / 8, 256, 0, st>>>(ns, tab, T, F);
  k_power<<<dim3((L + 255) / 256, L), 256, 0, st>>>(nsubs, ndouble, njoin, L, ns, tab, T, F, have_single, have_join,
                                                     have_double, power, power_join, power_double);
  return cudaGetLastError();
}

}  // namespace covgpu
