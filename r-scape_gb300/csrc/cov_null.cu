// cov_null.cu -- null alignments on the GPU: Fitch ancestral states and the
// shuffled-substitution replay of R-scape's default null (--nullphylo).
//
// The reconstruction depends on the columns only one by one, the replay only
// on the branches' substitution counts and the parent's current row, so the
// work goes in two parts:
//   k_fitch_cols   a CTA per (4 to 32 columns, null), the whole tree in its
//                  shared memory where it fits: the up pass of
//                  Tree_FitchAlgorithmAncenstral / tree_fitch_column
//                  (src/msatree.c:173-227, 1700-1838): intersection of the
//                  children's sets over the five states, else the union of
//                  residues only (tree_fitch_upwards :1877-1908), as
//                  byte-SIMD; the root's state; the down pass (keep the
//                  parent's state when the child's set holds it); and the
//                  substitutions of each kind on each branch, added over the
//                  columns into the branch's 25 counters.
//   the replay     the root's row with the columns shuffled
//                  (msamanip_ShuffleColumns, src/msamanip.c:1164-1233; only
//                  the root's shuffled row is ever read, every other row is
//                  replaced by its parent's row before use), then top depth
//                  first shuffle_tree_substitutions + shuffle_tree_substitute_all
//                  (src/msamanip.c:1597-1747): a branch copies the parent's
//                  current row and replays its substitutions on positions of
//                  that row holding the old state, visited in a random order (a
//                  Feistel permutation); each class's positions are ranked with
//                  warp ballots and the pass stops once every substitution is
//                  placed.  Small alignments: one launch, a cluster of CTAs per
//                  null (k_null_replay); larger ones a launch per depth.
//
// Random draws are counter-based (Philox keyed by the seed, the null index,
// the node and the column), so the result does not depend on scheduling.
//
// Buffers (per null q): F[q][Lp] the root's states; ns[q][2N][25] the
// substitutions from state a to state b on the branch above leaf s (entry s)
// or internal node v (entry N + v), at 5 a + b; SR[q][v][Lp] node v's row of
// the null alignment; leaf rows go straight to the output alignment slot.
#include "cov_dev.cuh"
#include "cov_kernels.h"
#include "cov_batch.h"
#include <algorithm>
#include <atomic>
#include <type_traits>

namespace covgpu {

__device__ __forceinline__ int choose_member(unsigned S, uint64_t seed, uint32_t null_id, uint32_t node, uint32_t col) {
  const int m = __popc(S);
  int k = 0;
  if (m > 1) k = (int)(((uint64_t)rng_u32(seed, TAG_FCHOOSE, null_id, node, col) * (uint64_t)m) >> 32);
  for (int x = 0; x < 5; x++)
    if (S & (1u << x)) { if (k == 0) return x; k--; }
  return 4;
}


// States are kept as one bit per byte (1 << state), four columns to a word,
// so the passes work on whole words; only random draws go byte by byte.
//
// word of four leaf codes: the states of codes 0-4; an ambiguity code gets a
// random state, marked with bit 7
constexpr uint32_t AMBIG = 0x80u;
__device__ __forceinline__ uint32_t leaf_word(uint32_t w, int n, int c0, uint64_t seed, uint32_t nid) {
  if ((w + 0x7B7B7B7Bu) & 0x80808080u) {   // a code above 4 (codes are below 18)
    uint32_t o = 0;
    for (int b = 0; b < 4; b++) {
      const uint32_t x = (w >> (8 * b)) & 0xFFu;
      const uint32_t s =
          x <= 4 ? 1u << x
                 : AMBIG | (1u << (int)(((uint64_t)rng_u32(seed, TAG_FLEAF, nid, (uint32_t)n, (uint32_t)(c0 + b)) * 5u) >> 32));
      o |= s << (8 * b);
    }
    return o;
  }
  const uint32_t sel = (w | (w >> 4)) & 0x00FF00FFu;   // codes to nibbles
  return __byte_perm(0x08040201u, 0x00000010u, (sel | (sel >> 8)) & 0xFFFFu);
}
// the state numbers of a word of states
__device__ __forceinline__ uint32_t state_codes(uint32_t w) {
  return ((w >> 1) & 0x0F0F0F0Fu) - ((w >> 3) & 0x01010101u) - ((w >> 2) & 0x04040404u);
}
// one state of every set of a word: the only member, or a random one; the
// bytes of pick are considered, the others kept
__device__ __forceinline__ uint32_t choose_word(uint32_t s, uint32_t pick, uint64_t seed, uint32_t nid,
                                                uint32_t node, int c0) {
  uint32_t multi = (s & (s - 0x01010101u)) & pick;   // sets are not empty: no borrow between bytes
  while (multi) {   // each lane its next byte: as many draws as the lane with the most
    const int sh = (__ffs(multi) - 1) & ~7;
    const uint32_t st = (uint32_t)choose_member((s >> sh) & 0xFFu, seed, nid, node, (uint32_t)(c0 + (sh >> 3)));
    s = (s & ~(0xFFu << sh)) | (1u << (sh + st));
    multi &= ~(0xFFu << sh);
  }
  return s;
}

// per byte: I = a & b if nonzero, else (a | b) without the gap bit
__device__ __forceinline__ uint32_t fitch_word(uint32_t a, uint32_t b) {
  const uint32_t I = a & b, U = (a | b) & 0x0F0F0F0Fu;
  const uint32_t z = __vcmpeq4(I, 0u);   // 0xFF in the bytes where I == 0
  return (I & ~z) | (U & z);
}

// The reconstruction of FW words of four columns by one CTA.  With KEEP_TREE
// the leaves, the nodes' sets (then states) and the tree lie in shared memory,
// 8 FW + 6 bytes per sequence, so a depth costs a barrier and a few shared
// accesses; KEEP_WORDS leaves the tree in global memory; KEEP_NONE takes
// everything from there (the rows from the null's buffer SR, each CTA its own
// columns).  Bound by instructions on large alignments (64% of the issue slots;
// 400 us for 20 nulls of 2,000 x 3,000), by the barriers on small ones (13 us
// for 30 x 61).
// With the reconstruction inside the replay, depth by depth, the null
// generation took (now): 30 x 61, 20 nulls 134 us (46); 400 x 300, 20 nulls
// 572 (238); 500 x 400, 200 nulls 895 (740); 2,000 x 3,000, 20 nulls 1,266
// (1,018); the reconstruction alone, 701 x 650, 300 us in 42 launches (20).
//
// The form by the number of sequences N and of columns of all nulls (us, the
// whole null generation of 20 nulls unless said):
//   {4, TREE}, {2, TREE}  while two CTAs of 512 threads fit an SM: 2,700 x
//     2,000 1,218 and 1,233, 3,500 x 2,000 1,772 and 1,617
//   {1, TREE}, {1, WORDS}  beyond, up to 4,096 columns: enough CTAs for the
//     SMs where there are few columns (20,000 x 60, one null: 370; 849 with
//     the rows in global memory)
//   {8, NONE}  the rest: full sectors and 32 warps per SM (12,000 x 1,000:
//     1,936; {1, TREE} 2,232, four words 2,191)
struct FitchCols {
  const uint8_t* ax;
  int N, L, Lp;
  const int *left, *right, *lnodes, *loff;
  int nlevels;
  uint64_t seed;
  uint32_t nid;
  uint8_t* SR;     // [N-1][Lp] (not SM: scratch)
  uint8_t* F;      // state numbers: the root's row, or every node's with all_rows
  bool all_rows;
  int* ns;         // [2N][25] branch counters, or nullptr
};
// the form of the kernel: words of a CTA and what it keeps in shared memory
enum FitchKeep { KEEP_NONE = 0, KEEP_WORDS = 1, KEEP_TREE = 2 };
static size_t fitch_smem(int N, int FW, int keep) {
  return keep == KEEP_NONE ? 0 : (size_t)N * (2 * FW * 4 + (keep == KEEP_TREE ? 3 * 2 : 0)) + 16;
}
constexpr size_t FITCH_SMEM_MAX = 224 * 1024;
static_assert(FITCH_SMEM_MAX / (2 * 4 + 3 * 2) < 32768, "the tree's node numbers fit 16 bits");
constexpr size_t FITCH_SMEM_HALF = 113 * 1024;   // two CTAs per SM
struct FitchForm { int fw, keep, threads; };
static FitchForm fitch_form(int N, int64_t cols) {
  // the widest depth of a tree of N leaves is about N / 10 nodes (coalescent)
  const int thr = N >= 512 ? 512 : (N >= 128 ? 256 : 128);
  for (int fw : {4, 2})
    if (fitch_smem(N, fw, KEEP_TREE) <= FITCH_SMEM_HALF) return {fw, KEEP_TREE, thr};
  for (int keep : {KEEP_TREE, KEEP_WORDS})
    if (cols <= 4096 && fitch_smem(N, 1, keep) <= FITCH_SMEM_MAX) return {1, keep, 1024};
  return {8, KEEP_NONE, 1024};
}
// f(FW, KEEP) of the form, as integral constants
template <class FN>
static cudaError_t with_fitch_form(FitchForm x, FN f) {
  using std::integral_constant;
  if (x.keep == KEEP_NONE) f(integral_constant<int, 8>(), integral_constant<int, KEEP_NONE>());
  else if (x.fw == 4) f(integral_constant<int, 4>(), integral_constant<int, KEEP_TREE>());
  else if (x.fw == 2) f(integral_constant<int, 2>(), integral_constant<int, KEEP_TREE>());
  else if (x.keep == KEEP_TREE) f(integral_constant<int, 1>(), integral_constant<int, KEEP_TREE>());
  else f(integral_constant<int, 1>(), integral_constant<int, KEEP_WORDS>());
  return cudaGetLastError();
}

template <int FW, int KEEP>
__device__ __forceinline__ void fitch_cols(const FitchCols& a, int grp) {
  extern __shared__ __align__(16) uint32_t fsm[];
  constexpr bool SM = KEEP != KEEP_NONE, TREE = KEEP == KEEP_TREE;
  const int N = a.N, tid = threadIdx.x, nthr = blockDim.x, c0 = grp * FW * 4;
  uint32_t* leaf = fsm;
  uint32_t* node = SM ? fsm + (size_t)N * FW : reinterpret_cast<uint32_t*>(a.SR + c0);
  const int stride = SM ? FW : a.Lp / 4;
  int16_t* lr = reinterpret_cast<int16_t*>(fsm + (size_t)2 * N * FW);   // TREE: left, right, lnodes
  if (SM) {
    for (int i = tid; i < N * FW; i += nthr) {
      const int s = i / FW, c = c0 + 4 * (i % FW);
      leaf[i] = leaf_word(*reinterpret_cast<const uint32_t*>(a.ax + (int64_t)s * a.Lp + c), s, c, a.seed, a.nid);
    }
    for (int v = tid; TREE && v < N - 1; v += nthr) {
      lr[v] = (int16_t)a.left[v]; lr[N + v] = (int16_t)a.right[v]; lr[2 * N + v] = (int16_t)a.lnodes[v];
    }
    __syncthreads();
  }
  auto left = [&](int v) { return TREE ? (int)lr[v] : a.left[v]; };
  auto right = [&](int v) { return TREE ? (int)lr[N + v] : a.right[v]; };
  auto order = [&](int k) { return TREE ? (int)lr[2 * N + k] : a.lnodes[k]; };
  auto leafw = [&](int s, int w) -> uint32_t {
    if (SM) return leaf[s * FW + w];
    const int c = c0 + 4 * w;
    return leaf_word(*reinterpret_cast<const uint32_t*>(a.ax + (int64_t)s * a.Lp + c), s, c, a.seed, a.nid);
  };
  auto sets = [&](int ch, int w) -> uint32_t {
    if (SM) return fsm[(ch > 0 ? N + ch : -ch) * FW + w] & ~(AMBIG * 0x01010101u);   // the nodes follow the leaves
    return ch > 0 ? node[(int64_t)ch * stride + w] : leafw(-ch, w) & ~(AMBIG * 0x01010101u);
  };
  for (int d = a.nlevels - 1; d >= 0; d--) {
    const int o = a.loff[d], n = (a.loff[d + 1] - o) * FW;
    for (int i = tid; i < n; i += nthr) {
      const int v = order(o + i / FW), w = i % FW;
      node[(int64_t)v * stride + w] = fitch_word(sets(left(v), w), sets(right(v), w));
    }
    __syncthreads();
  }
  for (int w = tid; w < FW; w += nthr) {   // the root's state
    const uint32_t s = choose_word(node[w], 0xFFFFFFFFu, a.seed, a.nid, 0u, c0 + 4 * w);
    node[w] = s;
    *reinterpret_cast<uint32_t*>(a.F + c0 + 4 * w) = state_codes(s);
  }
  __syncthreads();
  for (int d = 0; d < a.nlevels; d++) {
    const int o = a.loff[d], n = 2 * (a.loff[d + 1] - o) * FW;
    for (int i = tid; i < n; i += nthr) {
      const int k = i / FW, w = i % FW, v = order(o + (k >> 1)), ch = (k & 1) ? right(v) : left(v);
      const uint32_t p = node[(int64_t)v * stride + w];
      uint32_t q;
      if (ch > 0) {
        // the parent's state where the child's set holds it, else one of the set
        const uint32_t s = node[(int64_t)ch * stride + w], z = __vcmpeq4(s & p, 0u);
        q = choose_word((p & ~z) | (s & z), z, a.seed, a.nid, (uint32_t)ch, c0 + 4 * w);
        node[(int64_t)ch * stride + w] = q;
        if (a.all_rows) *reinterpret_cast<uint32_t*>(a.F + (int64_t)ch * a.Lp + c0 + 4 * w) = state_codes(q);
      } else {
        q = leafw(-ch, w);
      }
      // bytes that differ, not ambiguous (a leaf's bit 7); columns past L hold
      // gaps in every row and never differ
      const uint32_t diff = __vcmpne4(p, q) & ~__vcmpne4(q & (AMBIG * 0x01010101u), 0u);
      if (!a.ns || diff == 0u) continue;
      int* ns = a.ns + (int64_t)(ch > 0 ? N + ch : -ch) * 25;
      const uint32_t kind = 5u * state_codes(p) + state_codes(q);   // four counters' places, below 25 where diff
#pragma unroll
      for (int b = 0; b < 4; b++)
        if ((diff >> (8 * b)) & 1u) atomicAdd(ns + ((kind >> (8 * b)) & 0xFFu), 1);
    }
    __syncthreads();
  }
}

// the threads of FW words' forms (fitch_form)
constexpr int fitch_max_threads(int FW) { return FW == 4 || FW == 2 ? 512 : 1024; }
template <int FW, int KEEP>
__global__ void __launch_bounds__(fitch_max_threads(FW))
k_fitch_cols(FitchCols a, int64_t nstride, int64_t sstride) {
  a.nid += blockIdx.y;
  a.SR += blockIdx.y * sstride;
  a.F += (int64_t)blockIdx.y * a.Lp;   // the root's rows of the nulls
  if (a.ns) a.ns += blockIdx.y * nstride;
  fitch_cols<FW, KEEP>(a, blockIdx.x);
}

// the root's row of the null: its states with the columns shuffled
__device__ __forceinline__ void root_row_body(
    const GridIdx g, int L, int Lp, uint64_t seed, uint32_t first_null, int64_t stride, const uint8_t* __restrict__ F,
    uint8_t* __restrict__ SR) {
  const int c = g.x * blockDim.x + threadIdx.x, q = g.y;
  if (c >= Lp) return;
  uint32_t rk[6];
  round_keys(seed, TAG_COLPERM, first_null + q, 0, rk);
  const uint8_t* row = F + (int64_t)q * Lp;
  SR[q * stride + c] = (c < L) ? row[feistel_perm((uint32_t)c, feistel_hbits((uint32_t)L), (uint32_t)L, rk)] : (uint8_t)4;
}
__global__ void __launch_bounds__(256)
k_root_row(int L, int Lp, uint64_t seed, uint32_t first_null, int64_t stride, const uint8_t* __restrict__ F,
           uint8_t* __restrict__ SR) {
  root_row_body(native_grid(), L, Lp, seed, first_null, stride, F, SR);
}

// The replay of one (branch, null) item: the child's row starts as a copy of
// the parent's row (staged in shared memory too when srow is given, for the
// random reads that follow); then the walk goes through the slots t in order,
// maps each to position perm(t) of the parent's row and, for the state o
// there, ranks the slot among the slots of class o so far: the r-th takes
// substitution r of class o while r < need[o].  Once every class has its
// substitutions the walk stops (later slots would place nothing).  One warp
// per item walks 32 slots a step, one CTA per item as many as it has threads,
// with a prefix over the warps.
struct ReplayItem {
  int cidx;            // leaf s: s; internal node v: N + v
  uint32_t nid;
  const uint8_t* Rp;   // parent's current row
  uint8_t* Cc;         // child's row
  const int* ns;       // the branch's 25 counters
};

// this null's rows SR [N-1][Lp], alignment out [N][Lp] and counters ns [2N][25]
__device__ __forceinline__ ReplayItem replay_item(int N, int Lp, const int* left, const int* right, const int* nodes,
                                                  int item, uint32_t nid, uint8_t* SR, uint8_t* out, const int* ns) {
  ReplayItem it;
  const int v = nodes[item >> 1];
  const int ch = (item & 1) ? right[v] : left[v];
  it.cidx = (ch <= 0) ? -ch : N + ch;
  it.nid = nid;
  it.Rp = SR + (int64_t)v * Lp;
  it.Cc = (ch <= 0) ? out + (int64_t)(-ch) * Lp : SR + (int64_t)ch * Lp;
  it.ns = ns + (int64_t)it.cidx * 25;
  return it;
}

// the row copy by nthr threads (this one: tid), and cum [5][6], the running
// sums of each class's counters (rows that other SMs wrote: past L1)
__device__ __forceinline__ void replay_prepare(const ReplayItem& it, int Lp, int tid, int nthr, int (*cum)[6],
                                               uint8_t* srow) {
  if (tid < 5) {
    int s = 0;
    cum[tid][0] = 0;
#pragma unroll
    for (int d = 0; d < 5; d++) { s += it.ns[tid * 5 + d]; cum[tid][d + 1] = s; }
  }
  for (int c0 = tid * 16; c0 < Lp; c0 += nthr * 16) {   // Lp is a multiple of 32
    const uint4 v4 = __ldcg(reinterpret_cast<const uint4*>(it.Rp + c0));
    *reinterpret_cast<uint4*>(it.Cc + c0) = v4;
    if (srow) *reinterpret_cast<uint4*>(srow + c0) = v4;
  }
}

__device__ __forceinline__ unsigned pick5(const unsigned (&m)[5], int k) {
  return k == 0 ? m[0] : k == 1 ? m[1] : k == 2 ? m[2] : k == 3 ? m[3] : m[4];
}

// one item by one warp; srow (nullptr or Lp bytes) and cum [5][6] in shared
// memory, the warp's own
__device__ __forceinline__ void replay_item_warp(const ReplayItem& it, int L, int Lp, uint64_t seed, int lane,
                                                 int (*cum)[6], uint8_t* srow) {
  replay_prepare(it, Lp, lane, 32, cum, srow);
  __syncwarp();
  int need[5], total = 0;
#pragma unroll
  for (int o = 0; o < 5; o++) { need[o] = cum[o][5]; total += need[o]; }
  if (total == 0) return;
  uint32_t rk[6];
  round_keys(seed, TAG_SUBST, it.nid, (uint32_t)it.cidx, rk);
  const uint8_t* R = srow ? srow : it.Rp;
  const uint32_t hb = feistel_hbits((uint32_t)L);
  const unsigned lt = (1u << lane) - 1u;
  int run[5] = {0, 0, 0, 0, 0};
  for (int t0 = 0; t0 < L; t0 += 32) {
    const int t = t0 + lane;
    uint32_t p = 0;
    int o = 5;
    if (t < L) {
      p = feistel_perm((uint32_t)t, hb, (uint32_t)L, rk);
      o = srow ? R[p] : __ldcg(R + p);
    }
    bool done = true;
#pragma unroll
    for (int oc = 0; oc < 5; oc++) {
      const unsigned m = __ballot_sync(0xffffffffu, o == oc);
      if (o == oc) {
        const int r = run[oc] + __popc(m & lt);
        if (r < need[oc]) {
          int d = 0;
          while (r >= cum[oc][d + 1]) d++;
          it.Cc[p] = (uint8_t)d;
        }
      }
      run[oc] += __popc(m);
      done = done && (run[oc] >= need[oc]);
    }
    if (done) break;
  }
}

// one warp per item, eight items per CTA (SROW: Lp bytes of row per warp)
template <bool SROW>
__device__ __forceinline__ void replay_warp_body(
    const GridIdx g, int N, int L, int Lp, const int* __restrict__ left, const int* __restrict__ right,
    const int* __restrict__ nodes, int nn, uint64_t seed, uint32_t first_null, const int* __restrict__ ns, uint8_t* SR,
    uint8_t* out_ax, int64_t out_slot_stride) {
  extern __shared__ __align__(16) uint8_t rowbuf[];
  __shared__ int cum_s[8][5][6];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int item = g.x * 8 + warp;
  if (item >= 2 * nn) return;
  const ReplayItem it = replay_item(N, Lp, left, right, nodes, item, first_null + g.y,
                                    SR + (int64_t)g.y * (N - 1) * Lp, out_ax + g.y * out_slot_stride,
                                    ns + (int64_t)g.y * 2 * N * 25);
  replay_item_warp(it, L, Lp, seed, lane, cum_s[warp], SROW ? rowbuf + (size_t)warp * Lp : nullptr);
}
template <bool SROW>
__global__ void __launch_bounds__(256)
k_replay_warp(int N, int L, int Lp, const int* __restrict__ left, const int* __restrict__ right,
              const int* __restrict__ nodes, int nn, uint64_t seed, uint32_t first_null, const int* __restrict__ ns,
              uint8_t* SR, uint8_t* out_ax, int64_t out_slot_stride) {
  replay_warp_body<SROW>(native_grid(), N, L, Lp, left, right, nodes, nn, seed, first_null, ns, SR, out_ax,
                         out_slot_stride);
}

// one item by a CTA of NW warps; srow as above; cum [5][6], gcnt [NW][5]
// (slots per class in each warp's group of the chunk) and base [5] (slots per
// class before it) in shared memory
template <int NW>
__device__ __forceinline__ void replay_item_cta(const ReplayItem& it, int L, int Lp, uint64_t seed, int (*cum)[6],
                                                int (*gcnt)[5], int* base, uint8_t* srow) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < 5) base[tid] = 0;
  replay_prepare(it, Lp, tid, NW * 32, cum, srow);
  __syncthreads();
  int need[5], total = 0;
#pragma unroll
  for (int o = 0; o < 5; o++) { need[o] = cum[o][5]; total += need[o]; }
  if (total == 0) return;   // the same in every thread
  uint32_t rk[6];
  round_keys(seed, TAG_SUBST, it.nid, (uint32_t)it.cidx, rk);
  const uint32_t hb = feistel_hbits((uint32_t)L);
  const unsigned lt = (1u << lane) - 1u;
  const uint8_t* R = srow ? srow : it.Rp;
  for (int t0 = 0; t0 < L; t0 += NW * 32) {
    const int t = t0 + tid;
    uint32_t p = 0;
    int o = 5;
    if (t < L) {
      p = feistel_perm((uint32_t)t, hb, (uint32_t)L, rk);
      o = srow ? R[p] : __ldcg(R + p);
    }
    unsigned m[5];
#pragma unroll
    for (int oc = 0; oc < 5; oc++) m[oc] = __ballot_sync(0xffffffffu, o == oc);
    if (lane < 5) gcnt[warp][lane] = __popc(pick5(m, lane));
    __syncthreads();
    if (o < 5) {
      int r = base[o] + __popc(pick5(m, o) & lt);
      for (int w = 0; w < warp; w++) r += gcnt[w][o];
      if (r < cum[o][5]) {   // need[o], read from shared memory (o varies by lane)
        int d = 0;
        while (r >= cum[o][d + 1]) d++;
        it.Cc[p] = (uint8_t)d;
      }
    }
    __syncthreads();   // base and gcnt read
    if (tid < 5) {
      int s2 = base[tid];
      for (int w = 0; w < NW; w++) s2 += gcnt[w][tid];
      base[tid] = s2;
    }
    __syncthreads();
    bool all = true;
#pragma unroll
    for (int oc = 0; oc < 5; oc++) all = all && (base[oc] >= need[oc]);
    if (all) break;   // the same in every thread
  }
}

// one CTA per item (SROW: Lp bytes of row)
template <bool SROW>
__device__ __forceinline__ void replay_cta_body(
    const GridIdx g, int N, int L, int Lp, const int* __restrict__ left, const int* __restrict__ right,
    const int* __restrict__ nodes, int nn, uint64_t seed, uint32_t first_null, const int* __restrict__ ns, uint8_t* SR,
    uint8_t* out_ax, int64_t out_slot_stride) {
  extern __shared__ __align__(16) uint8_t rowbuf[];
  __shared__ int cum[5][6], gcnt[8][5], base[5];
  if (g.x >= 2 * nn) return;
  const ReplayItem it = replay_item(N, Lp, left, right, nodes, g.x, first_null + g.y,
                                    SR + (int64_t)g.y * (N - 1) * Lp, out_ax + g.y * out_slot_stride,
                                    ns + (int64_t)g.y * 2 * N * 25);
  replay_item_cta<8>(it, L, Lp, seed, cum, gcnt, base, SROW ? rowbuf : nullptr);
}
template <bool SROW>
__global__ void __launch_bounds__(256)
k_replay_cta(int N, int L, int Lp, const int* __restrict__ left, const int* __restrict__ right,
             const int* __restrict__ nodes, int nn, uint64_t seed, uint32_t first_null, const int* __restrict__ ns,
             uint8_t* SR, uint8_t* out_ax, int64_t out_slot_stride) {
  replay_cta_body<SROW>(native_grid(), N, L, Lp, left, right, nodes, nn, seed, first_null, ns, SR, out_ax,
                        out_slot_stride);
}

// The replay of one null by one cluster of CTAs, every depth in one launch: a
// cluster barrier between depths (the levels of one null depend on each
// other, the nulls do not).  A depth with at most one item per CTA takes a CTA
// per item, the others a warp per item.
struct NullOne {
  int N, L, Lp;
  const int *left, *right, *lnodes, *loff;   // loff [nlevels + 1]: depth offsets in lnodes
  int nlevels;
  const uint8_t* F;                          // the root's states
  const int* ns;
  uint8_t *SR, *out;                         // this null's rows and alignment
  uint64_t seed;
  uint32_t nid;
};

constexpr int NULL_WARPS = 16;

__device__ __forceinline__ void null_sync(int csize) {
  if (csize == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  }
}

__device__ __forceinline__ void null_replay(const NullOne& a, int crank, int csize) {
  extern __shared__ __align__(16) uint8_t rowbuf[];
  __shared__ int cum_s[NULL_WARPS][5][6];
  __shared__ int gcnt[NULL_WARPS][5], base[5];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  {
    uint32_t rk[6];
    round_keys(a.seed, TAG_COLPERM, a.nid, 0, rk);
    const uint32_t hb = feistel_hbits((uint32_t)a.L);
    for (int c = crank * (NULL_WARPS * 32) + tid; c < a.Lp; c += csize * (NULL_WARPS * 32))
      a.SR[c] = (c < a.L) ? a.F[feistel_perm((uint32_t)c, hb, (uint32_t)a.L, rk)] : (uint8_t)4;
  }
  null_sync(csize);
  for (int d = 0; d < a.nlevels; d++) {
    const int o = a.loff[d], n = 2 * (a.loff[d + 1] - o);
    if (n <= csize) {
      if (crank < n) {
        const ReplayItem it = replay_item(a.N, a.Lp, a.left, a.right, a.lnodes + o, crank, a.nid, a.SR, a.out, a.ns);
        replay_item_cta<NULL_WARPS>(it, a.L, a.Lp, a.seed, cum_s[0], gcnt, base, rowbuf);
      }
    } else {
      for (int item = warp * csize + crank; item < n; item += NULL_WARPS * csize) {
        const ReplayItem it = replay_item(a.N, a.Lp, a.left, a.right, a.lnodes + o, item, a.nid, a.SR, a.out, a.ns);
        replay_item_warp(it, a.L, a.Lp, a.seed, lane, cum_s[warp], rowbuf + (size_t)warp * a.Lp);
        __syncwarp();
      }
    }
    if (d + 1 < a.nlevels) null_sync(csize);
  }
}

__global__ void __launch_bounds__(NULL_WARPS * 32, 2)
k_null_replay(int N, int L, int Lp, const int* left, const int* right, const int* lnodes, const int* loff,
              int nlevels, uint64_t seed, uint32_t first_null, const uint8_t* F, const int* ns, uint8_t* SR,
              uint8_t* out, int64_t out_stride, int csize) {
  const int q = blockIdx.x / csize;
  const int64_t off = (int64_t)q * (N - 1) * Lp;
  const NullOne a{N, L, Lp, left, right, lnodes, loff, nlevels, F + (int64_t)q * Lp, ns + (int64_t)q * 2 * N * 25, SR + off,
                  out + q * out_stride, seed, first_null + q};
  null_replay(a, blockIdx.x % csize, csize);
}

// items of a launch up to which the replay goes one CTA per item: measured on
// N=2000 x L=3000 with 20 nulls, one CTA per item is faster up to about 3,000
// items (long branches near the root), one warp per item beyond.  In a family
// batch the items of all families count: 64 ragged families 84 ms a call, 96
// with the rule taken family by family.
constexpr int64_t kReplayCtaItems = 3000;

bool replay_uses_cta(int64_t items) { return items <= kReplayCtaItems; }

constexpr int NULL_MAXL = 1024;   // columns up to which one launch may replay a null
static_assert(NULL_WARPS * NULL_MAXL <= 48 * 1024, "a row per warp within the shared memory that needs no opt-in");
// CTAs of the cluster that replays one null in one launch, 0: a launch per
// depth.  One launch wins where the depths are short: up to 13M columns x
// sequences x nulls in all and rows of 1,024 columns (a warp's walk along a
// longer row takes longer than the launches), and while a null's cells are few
// for the 128 warps of its cluster: the launches spread a depth over all SMs,
// so the fewer the nulls, the sooner they win.  Measured against the launches
// (us, the whole null generation): 30 x 61, 20 nulls 46 / 77 (C = 1); 100 x 120
// 112 / 151; 400 x 300 238 / 375; 700 x 900 289 / 336; 2,000 x 300 530 / 545;
// but 500 x 400 with 200 nulls 803 / 762, 100 x 3,000 263 / 205, 8,000 x 64
// with 20 nulls 485 / 448, 4,000 x 300 with nine 710 / 636, 2,000 x 1,000 with
// five 365 / 281; with one null 2,000 x 64 172 / 189 and 3,000 x 64 218 / 222,
// 1,000 x 300 321 / 280 and 20,000 x 600 1,760 / 490.
static int null_cluster(int N, int L, int nnull) {
  if (L > NULL_MAXL || (double)N * L * nnull > 13e6 || (double)N * L > (nnull < 4 ? 0.2e6 : 0.7e6)) return 0;
  if ((int64_t)N * L < 8192) return 1;
  int dev = 0, nsm = 152, C = 8;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  while (C > 1 && (int64_t)C * nnull > 2 * nsm) C >>= 1;
  return C;
}

// the replay's shared-memory row buffers: the launch limit of both kernels
// is raised once to the device's opt-in maximum; rows that do not fit are
// read from global memory instead
static int replay_smem_limit() {
  static const int lim = [] {
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
      return 48 * 1024;
    const int dyn = optin - 4096;   // room for the kernels' static arrays
    if (dyn <= 48 * 1024 ||
        cudaFuncSetAttribute(k_replay_warp<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess ||
        cudaFuncSetAttribute(k_replay_cta<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess)
      return 48 * 1024;
    return dyn;
  }();
  return lim;
}

template <int FW, int KEEP>
__global__ void __launch_bounds__(fitch_max_threads(FW))
k_fitch_cols_grp(const FamDev* __restrict__ F, int nf, const int* __restrict__ pre, uint64_t seed) {
  const int f = grp_find(pre, nf, (int)blockIdx.x);
  const FamDev& d = F[f];
  const int gx = d.Lp / (FW * 4), loc = (int)blockIdx.x - __ldg(pre + f), q = loc / gx;
  const FitchCols a{d.ax, d.N, d.L, d.Lp, d.left, d.right, d.lnodes, d.lnodes + (d.N - 1), d.nlevels, seed,
                    (uint32_t)q, d.scratch + (int64_t)q * (d.N - 1) * d.Lp, d.fitch + (int64_t)q * d.Lp, false,
                    d.ns + (int64_t)q * 2 * d.N * 25};
  fitch_cols<FW, KEEP>(a, loc % gx);
}

// raises the shared-memory limits of this file's kernels on the current
// device, once (before any stream capture)
static cudaError_t null_attrs() {
  constexpr int MAXDEV = 64;
  static std::atomic<int> done[MAXDEV];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < MAXDEV && done[dev].load()) return cudaSuccess;
  const void* fit[] = {(const void*)k_fitch_cols<4, KEEP_TREE>,     (const void*)k_fitch_cols<2, KEEP_TREE>,
                       (const void*)k_fitch_cols<1, KEEP_TREE>,     (const void*)k_fitch_cols<1, KEEP_WORDS>,
                       (const void*)k_fitch_cols_grp<4, KEEP_TREE>, (const void*)k_fitch_cols_grp<2, KEEP_TREE>,
                       (const void*)k_fitch_cols_grp<1, KEEP_TREE>, (const void*)k_fitch_cols_grp<1, KEEP_WORDS>};
  for (const void* f : fit)
    if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FITCH_SMEM_MAX)) != cudaSuccess)
      return e;
  if (dev < MAXDEV) done[dev].store(1);
  return cudaSuccess;
}

static cudaError_t launch_fitch_cols(const FitchCols& a, int nnull, int64_t nstride, int64_t sstride,
                                     cudaStream_t st) {
  const FitchForm x = fitch_form(a.N, (int64_t)a.Lp * nnull);
  return with_fitch_form(x, [&](auto fw, auto keep) {
    k_fitch_cols<decltype(fw)::value, decltype(keep)::value>
        <<<dim3(a.Lp / (x.fw * 4), nnull), x.threads, fitch_smem(a.N, x.fw, x.keep), st>>>(a, nstride, sstride);
  });
}

cudaError_t launch_fitch_recon(const uint8_t* ax, int N, int L, int Lp, const NullTree& T, const int* level_nodes,
                               int nlevels, uint64_t seed, uint32_t nid, uint8_t* F, uint8_t* S, cudaStream_t st) {
  cudaError_t e = null_attrs();
  if (e != cudaSuccess) return e;
  const FitchCols a{ax, N, L, Lp, T.left, T.right, level_nodes, level_nodes + (N - 1), nlevels, seed, nid, S, F, true,
                    nullptr};
  return launch_fitch_cols(a, 1, 0, 0, st);
}

cudaError_t launch_nullgen(const uint8_t* ax, int N, int L, int Lp, const NullTree& T, const int* level_nodes,
                           const int* level_off, int nlevels, uint64_t seed, uint32_t first_null, int nnull,
                           uint8_t* fitch, uint8_t* rows, int* ns, uint8_t* out_ax, int64_t out_slot_stride,
                           cudaStream_t st, int* nlaunch) {
  cudaError_t e = null_attrs();
  if (e != cudaSuccess) return e;
  const int64_t stride = (int64_t)(N - 1) * Lp, nstride = (int64_t)2 * N * 25;
  const int* d_off = level_nodes + (N - 1);
  if ((e = cudaMemsetAsync(ns, 0, (size_t)nstride * nnull * sizeof(int), st)) != cudaSuccess) return e;
  const FitchCols a{ax, N, L, Lp, T.left, T.right, level_nodes, d_off, nlevels, seed, first_null, rows, fitch, false,
                    ns};
  if ((e = launch_fitch_cols(a, nnull, nstride, stride, st)) != cudaSuccess) return e;
  const int C = null_cluster(N, L, nnull);
  if (C) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C * nnull);
    cfg.blockDim = dim3(NULL_WARPS * 32);
    cfg.dynamicSmemBytes = (size_t)NULL_WARPS * Lp;
    cfg.stream = st;
    cudaLaunchAttribute la[1];
    la[0].id = cudaLaunchAttributeClusterDimension;
    la[0].val.clusterDim.x = C;
    la[0].val.clusterDim.y = la[0].val.clusterDim.z = 1;
    cfg.attrs = la;
    cfg.numAttrs = 1;
    *nlaunch += 2;
    return cudaLaunchKernelEx(&cfg, k_null_replay, N, L, Lp, T.left, T.right, level_nodes, d_off, nlevels, seed,
                              first_null, (const uint8_t*)fitch, (const int*)ns, rows, out_ax, out_slot_stride, C);
  }
  k_root_row<<<dim3((Lp + 255) / 256, nnull), 256, 0, st>>>(L, Lp, seed, first_null, stride, fitch, rows);
  *nlaunch += 2;
  // levels with few items (near the root and the leaves) go one CTA per
  // item; the others one warp per item
  const int lim = replay_smem_limit();
  const bool srow_cta = (size_t)Lp <= (size_t)lim, srow_warp = (size_t)8 * Lp <= (size_t)lim;
  for (int d = 0; d < nlevels; d++) {
    const int nn = level_off[d + 1] - level_off[d];
    if (nn <= 0) continue;
    const int* lv = level_nodes + level_off[d];
    *nlaunch += 1;
    if (replay_uses_cta((int64_t)2 * nn * nnull)) {
      const dim3 g(2 * nn, nnull);
      if (srow_cta)
        k_replay_cta<true><<<g, 256, (size_t)Lp, st>>>(N, L, Lp, T.left, T.right, lv, nn, seed, first_null, ns, rows,
                                                      out_ax, out_slot_stride);
      else
        k_replay_cta<false><<<g, 256, 0, st>>>(N, L, Lp, T.left, T.right, lv, nn, seed, first_null, ns, rows, out_ax,
                                               out_slot_stride);
    } else {
      const dim3 g((2 * nn + 7) / 8, nnull);
      if (srow_warp)
        k_replay_warp<true><<<g, 256, (size_t)8 * Lp, st>>>(N, L, Lp, T.left, T.right, lv, nn, seed, first_null, ns,
                                                            rows, out_ax, out_slot_stride);
      else
        k_replay_warp<false><<<g, 256, 0, st>>>(N, L, Lp, T.left, T.right, lv, nn, seed, first_null, ns, rows, out_ax,
                                                out_slot_stride);
    }
  }
  return cudaGetLastError();
}

// ------------------------------------------------------------------------
// grouped launches over a batch of families: one tree depth of every
// family per launch (lv[f] = {offset of the depth in lnodes, nodes at it});
// every family's nulls use the single-family streams (null ids 0..ns-1)
// ------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
k_root_row_grp(const FamDev* __restrict__ F, int nf, const int* __restrict__ pre, uint64_t seed) {
  const int f = grp_find(pre, nf, (int)blockIdx.x);
  const FamDev& d = F[f];
  const int gx = (d.Lp + 255) / 256, loc = (int)blockIdx.x - __ldg(pre + f);
  root_row_body(GridIdx{loc % gx, loc / gx, gx}, d.L, d.Lp, seed, 0u, (int64_t)(d.N - 1) * d.Lp, d.fitch,
                d.scratch);
}

template <bool SROW>
__global__ void __launch_bounds__(256)
k_replay_warp_grp(const FamDev* __restrict__ F, int nf, const int2* __restrict__ lv, const int* __restrict__ pre,
                  uint64_t seed) {
  const int f = grp_find(pre, nf, (int)blockIdx.x);
  const FamDev& d = F[f];
  const int2 v = lv[f];
  const int gx = (2 * v.y + 7) / 8, loc = (int)blockIdx.x - __ldg(pre + f);
  const int64_t ss = (int64_t)d.N * d.Lp;
  replay_warp_body<SROW>(GridIdx{loc % gx, loc / gx, gx}, d.N, d.L, d.Lp, d.left, d.right, d.lnodes + v.x, v.y, seed,
                         0u, d.ns, d.scratch, d.ax + ss, ss);
}

template <bool SROW>
__global__ void __launch_bounds__(256)
k_replay_cta_grp(const FamDev* __restrict__ F, int nf, const int2* __restrict__ lv, const int* __restrict__ pre,
                 uint64_t seed) {
  const int f = grp_find(pre, nf, (int)blockIdx.x);
  const FamDev& d = F[f];
  const int2 v = lv[f];
  const int gx = 2 * v.y, loc = (int)blockIdx.x - __ldg(pre + f);
  const int64_t ss = (int64_t)d.N * d.Lp;
  replay_cta_body<SROW>(GridIdx{loc % gx, loc / gx, gx}, d.N, d.L, d.Lp, d.left, d.right, d.lnodes + v.x, v.y, seed,
                        0u, d.ns, d.scratch, d.ax + ss, ss);
}

int replay_smem_max() {
  static const int lim = [] {
    const int l = replay_smem_limit();
    if (l > 48 * 1024 &&
        (cudaFuncSetAttribute(k_replay_warp_grp<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, l) != cudaSuccess ||
         cudaFuncSetAttribute(k_replay_cta_grp<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, l) != cudaSuccess))
      return 48 * 1024;
    return l;
  }();
  return lim;
}

cudaError_t grp_fitch(const FamDev* F, int nf, const int* pre_cols, int nb_cols, int maxN, int64_t cols,
                      const int* pre_row, int nb_row, uint64_t seed, cudaStream_t st) {
  const FitchForm x = fitch_form(maxN, cols);
  if (nb_cols > 0) {
    const cudaError_t e = with_fitch_form(x, [&](auto fw, auto keep) {
      k_fitch_cols_grp<decltype(fw)::value, decltype(keep)::value>
          <<<nb_cols, x.threads, fitch_smem(maxN, x.fw, x.keep), st>>>(F, nf, pre_cols, seed);
    });
    if (e != cudaSuccess) return e;
  }
  if (nb_row > 0) k_root_row_grp<<<nb_row, 256, 0, st>>>(F, nf, pre_row, seed);
  return cudaGetLastError();
}
// Lp is a multiple of 32
int fitch_blocks(int Lp, int maxN, int64_t cols) { return Lp / (fitch_form(maxN, cols).fw * 4); }
int grp_null_prepare() { return null_attrs() == cudaSuccess ? 1 : 0; }

// srow: every family of the launch has its rows staged in shared memory
// (maxLp bytes per item)
cudaError_t grp_replay(const FamDev* F, int nf, const int2* lv, const int* pre, int nb, bool cta, bool srow,
                       int maxLp, uint64_t seed, cudaStream_t st) {
  if (nb <= 0) return cudaSuccess;
  if (cta) {
    if (srow) k_replay_cta_grp<true><<<nb, 256, (size_t)maxLp, st>>>(F, nf, lv, pre, seed);
    else      k_replay_cta_grp<false><<<nb, 256, 0, st>>>(F, nf, lv, pre, seed);
  } else {
    if (srow) k_replay_warp_grp<true><<<nb, 256, (size_t)8 * maxLp, st>>>(F, nf, lv, pre, seed);
    else      k_replay_warp_grp<false><<<nb, 256, 0, st>>>(F, nf, lv, pre, seed);
  }
  return cudaGetLastError();
}

}  // namespace covgpu
