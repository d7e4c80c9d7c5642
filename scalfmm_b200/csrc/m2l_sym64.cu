// FP64 M2L (parity form) as FP64 tensor-core GEMMs over every level of the tree at once.
//
// Symmetric Chebyshev operators: FChebSymKernel::M2L (Src/Kernels/Chebyshev/FChebSymKernel.hpp:210-328) applies,
// for each target and each of its <= 189 far neighbours at transfer vector t, the compressed operator of t's
// symmetry class through t's permutation: L += scale * P_t^T U_c V_c^T P_t M.  With the permutation folded into
// per-slot factors U_t = P_t^T U_c, V_t = P_t^T V_c (precompute.cu), the product splits into
//   Y_t(s) = V_t^T M_s        -- depends on the source cell s and the slot only,
//   L(c)  += scale * sum_t U_t Y_t(c + d_t).
//   * phase 1, per source parity sp: every slot that cells of parity sp feed (as sources of some target) is
//     stacked into one operator Vs_sp = [V_t^T]_t (sum of ranks ~ 4,200 rows at order 7, K = p^3); one GEMM
//     Y = Vs_sp * [M_s]_s over all cells of that parity gives every Y_t(s) the levels need;
//   * phase 2, per child type ct (the target parity, which fixes the 189 transfer vectors and their order): the
//     U_t of the transfer vectors that occur one after the other (K ~ 4,200), against Y gathered through the
//     interaction list (a missing source contributes zero).
// Dense operators (CHEB_DENSE, LAGRANGE): L[m] += scale * sum_n K_t(X_m, Y_n) M[n] (FChebDenseKernel::M2L,
// FChebDenseKernel.hpp:116-127; FUnifKernel applies the same Toeplitz operator through FFTs), in two forms:
//   * by pairs: the tree's (target, source) pairs are grouped by transfer vector once per tree, D = K_t [M_s] is
//     one GEMM over each vector's pairs, and a second kernel adds each target's rows of D in the order of its list.
//     No column of a tile is missing, where a tile of neighbouring targets misses most of a surface's sources;
//     D costs 16 bytes of traffic per value, against p^3 multiply-adds;
//   * by target tiles: phase 2 with K_t in the place of U_t and the multipoles in the place of Y; for orders 3 and 4,
//     where D's traffic is most of the time, and where the pair tables would be too large.
//
// The GEMM kernel (gemm64_kernel): mma.sync m8n8k4 with FP64 operands (tcgen05 has no FP64 kind; measured on this
// B200: 36.9 TFLOP/s from 8 warps per SM, the DFMA pipe's rate, at a quarter of its operand traffic).  A tile is
// 16 * MB operator rows x 64 cells, so that both the operator panel and the gathered cells come from L2 at about
// 15 bytes per clock and SM; MB is chosen so that the tiles cover p^3 rows closely (order 7: 2 tiles of 22 blocks of
// 8 rows for 43).  8 warps as 2 (rows) x 4 (cells), each MB x 2 blocks of 8 x 8, the accumulators in registers; two
// CTAs per SM.  K advances in stages of 16 = 4 groups of 4, loaded by cp.async (zero-filled past an operator's
// rows and where a source is missing) three deep.  A transfer vector that no cell of the tile has is left out of
// the K loop, and a block of 8 cells skips the groups of transfer vectors that none of its cells has: the cells of
// a parity are in Morton order, so that on surfaces neighbours share their missing ones.
// Where the tiles are too few for the GPU, the K range of each is split over up to 8 CTAs; the last one to finish
// adds the partial sums in the order of the ranges.  Each output element is summed in a fixed order, so results do
// not depend on the work order.  The reference sums the same products in a different order; the tests hold the
// two to 1e-12 relative.
//
// Measured, all levels, before (DFMA tiles of 128 x 128, one launch per level and phase; dense: one CTA per target
// cell) and after: 1M uniform, order 7, height 6: 23.1 -> 9.25 ms (phase 1 26 TFLOP/s of operator work; phase 2, with
// the missing sources at the box faces and the padding counted, 31); 20,000 points, order 7, height 5: 6.2 -> 1.4 ms;
// 65,537 points, dense order 5, height 5: 7.6 -> 0.94 ms; 500,009 points on a surface, Lagrange order 6, height 7:
// 19.1 -> 1.7 ms by pairs (7.0 ms by target tiles: 64 neighbouring targets of a surface share 4.1 times the sources
// that each has).
#include "common.cuh"

#include <algorithm>
#include <cmath>

namespace b200 {

constexpr int G_THREADS = 256;
constexpr int G_BN = 64;        // cells per tile
constexpr int G_BK = 16;        // K per stage: 4 groups of 4
constexpr int G_STAGES = 3;
constexpr int G_LDB = G_BK + 4; // shared-memory row of a cell: 20 doubles, conflict-free fragment loads
constexpr int G_Y_MB = 8;       // phase 1: 128 rows of Vs per tile
constexpr int kMaxSplit = 8;

// 8-row blocks per warp so that ceil(nblk / (2 MB)) tiles of 2 MB blocks cover the p^3 rows with little padding
__host__ __device__ constexpr int g_mb(int p) {
  return p == 3 ? 2 : p == 4 ? 4 : p == 5 ? 8 : p == 6 ? 7 : 11;
}

struct Sym64 {
  bool dense = false;
  int lda = 0;                       // row length of the phase-2 operators: p^3 rounded up to 8
  int ysum[8] = {0};                 // rows of Vs_sp: the ranks of the slots parity sp feeds, each rounded up to 2
  int yrank[8] = {0};                // the same without the rounding (the algorithmic count)
  int ldv[8] = {0};                  // row length of Vs_sp: ysum rounded up to 8
  long long vs_off[8] = {0};         // element offset of Vs_sp in d_vs
  int ystride = 0;                   // max ysum (row stride of Y)
  int max_groups = 0;                // most K groups of 4 of any child type
  double *d_vs = nullptr;            // [sp][p^3][ldv]: Vs_sp transposed
  double *d_a = nullptr;             // phase-2 operators, row k of slot t at (arow[t] + k) * lda; dense: d_dense
  int4 *d_ent = nullptr;             // [8][189]: (first operator row, first row of Y, K, 0) of entry e of child type ct
  // pairs grouped by transfer vector (dense operators), per tree
  bool pairs = false;                // the current tree takes the pair form
  long long pair_serial = -1;        // the tree whose tables are there
  int *d_pairtab = nullptr;          // [344] first pair, [344] first tile, [343] counts / cursors of each slot
  int h_first[344] = {0};            // host copy of the first pair of each slot
  int *d_psrc = nullptr;             // [pairs] level << 27 | source cell
  int *d_ppos = nullptr;             // [cells of levels 2..][189]: the pair of a list entry, -1 if none
  double *d_d = nullptr;             // [rhs][pairs of a chunk of slots][p^3]
  size_t cap_psrc = 0, cap_ppos = 0, cap_d = 0;
  // per tree
  long long room_serial = -1;        // the tree that d_plist, d_pblk and d_y have been settled for (tree_room)
  long long list_serial = -1;
  int *d_plist = nullptr;            // cells of every level grouped by parity, in Morton order
  int *d_ptab = nullptr;             // [kMaxHeight * 8] counts, list starts, then [kMaxHeight * 8 + 1] first tiles
  int *d_pblk = nullptr;             // [blocks of 1024 cells][8]: counts, then list positions
  size_t cap_list = 0, cap_pblk = 0;
  double *d_y = nullptr;             // [rhs][ncells][ystride]
  size_t cap_y = 0;
  double *d_part = nullptr;          // partial sums of split tiles: part_slots of them, allocated once
  int *d_tick = nullptr;             // arrivals per split tile
};

namespace {

// ---- cells of levels l0..l1 grouped by parity (child type = key & 7), in Morton order ---------------------
constexpr int PB_THREADS = 256, PB_CELLS = 1024;  // a block's cells, 4 consecutive ones per thread

struct ListArgs {
  const long long *keys[kMaxHeight];
  long long n[kMaxHeight];
  long long loff[kMaxHeight];
  int blk0[kMaxHeight + 1];  // first block of each level
  int l0, l1;
};

// 8 counters of 16 bits: parities 0..3 in x, 4..7 in y
__device__ __forceinline__ ulonglong2 parity_one(int p) {
  const unsigned long long v = 1ull << (16 * (p & 3));
  return p < 4 ? make_ulonglong2(v, 0ull) : make_ulonglong2(0ull, v);
}
__device__ __forceinline__ int parity_get(ulonglong2 c, int p) {
  return (int)(((p < 4 ? c.x : c.y) >> (16 * (p & 3))) & 0xffffull);
}

// this thread's 4 cells' parities (-1 past the end) and the block's exclusive prefix of the counts
__device__ __forceinline__ ulonglong2 parity_block_scan(const ListArgs &a, int &level, long long &cell0, int (&par)[4],
                                                        ulonglong2 &total) {
  __shared__ ulonglong2 ws[PB_THREADS / 32];
  level = a.l0;
  while (level < a.l1 && (int)blockIdx.x >= a.blk0[level + 1]) ++level;
  cell0 = (long long)((int)blockIdx.x - a.blk0[level]) * PB_CELLS + threadIdx.x * 4;
  ulonglong2 own = make_ulonglong2(0ull, 0ull);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    par[u] = cell0 + u < a.n[level] ? (int)(a.keys[level][cell0 + u] & 7) : -1;
    if (par[u] >= 0) {
      const ulonglong2 o = parity_one(par[u]);
      own.x += o.x;
      own.y += o.y;
    }
  }
  ulonglong2 inc = own;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long vx = __shfl_up_sync(0xffffffffu, inc.x, o), vy = __shfl_up_sync(0xffffffffu, inc.y, o);
    if (lane >= o) {
      inc.x += vx;
      inc.y += vy;
    }
  }
  if (lane == 31) ws[w] = inc;
  __syncthreads();
  ulonglong2 pre = make_ulonglong2(0ull, 0ull);
  total = pre;
#pragma unroll
  for (int q = 0; q < PB_THREADS / 32; ++q) {
    if (q < w) {
      pre.x += ws[q].x;
      pre.y += ws[q].y;
    }
    total.x += ws[q].x;
    total.y += ws[q].y;
  }
  return make_ulonglong2(pre.x + inc.x - own.x, pre.y + inc.y - own.y);
}

__global__ void __launch_bounds__(PB_THREADS) parity_count_kernel(const __grid_constant__ ListArgs a,
                                                                  int *__restrict__ blk) {
  int level, par[4];
  long long cell0;
  ulonglong2 total;
  parity_block_scan(a, level, cell0, par, total);
  if (threadIdx.x < 8) blk[blockIdx.x * 8 + threadIdx.x] = parity_get(total, threadIdx.x);
}

// One CTA, warp p for parity p: the blocks' counts become positions within (level, parity); then the list starts
// and the first tile of every (level, parity), deepest level first (the full tiles are started before the rest).
__global__ void __launch_bounds__(256) parity_scan_kernel(const __grid_constant__ ListArgs a, int *__restrict__ blk,
                                                          int *__restrict__ tab) {
  __shared__ int cnt[kMaxHeight * 8];
  const int p = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < kMaxHeight * 8) cnt[threadIdx.x] = 0;
  __syncthreads();
  for (int l = a.l0; l <= a.l1; ++l) {
    int carry = 0;
    for (int b0 = a.blk0[l]; b0 < a.blk0[l + 1]; b0 += 32) {
      const int b = b0 + lane;
      const int v = b < a.blk0[l + 1] ? blk[b * 8 + p] : 0;
      int x = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (b < a.blk0[l + 1]) blk[b * 8 + p] = carry + x - v;
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) cnt[l * 8 + p] = carry;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int tile = 0;
    for (int l = a.l1; l >= a.l0; --l) {
      int s = (int)a.loff[l];
      for (int q = 0; q < 8; ++q) {
        const int k = l * 8 + q;
        tab[k] = cnt[k];
        tab[kMaxHeight * 8 + k] = s;
        tab[2 * kMaxHeight * 8 + (kMaxHeight - 1 - l) * 8 + q] = tile;  // index of (level, parity) in tile order
        s += cnt[k];
        tile += (cnt[k] + G_BN - 1) / G_BN;
      }
    }
    for (int k = (kMaxHeight - a.l0) * 8; k <= kMaxHeight * 8; ++k) tab[2 * kMaxHeight * 8 + k] = tile;
  }
}

__global__ void __launch_bounds__(PB_THREADS) parity_place_kernel(const __grid_constant__ ListArgs a,
                                                                  const int *__restrict__ blk,
                                                                  const int *__restrict__ tab, int *__restrict__ list) {
  int level, par[4];
  long long cell0;
  ulonglong2 total;
  ulonglong2 pos = parity_block_scan(a, level, cell0, par, total);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (par[u] < 0) continue;
    list[tab[kMaxHeight * 8 + level * 8 + par[u]] + blk[blockIdx.x * 8 + par[u]] + parity_get(pos, par[u])] =
        (int)(cell0 + u);
    const ulonglong2 o = parity_one(par[u]);
    pos.x += o.x;
    pos.y += o.y;
  }
}

// ---- pairs grouped by transfer vector ----------------------------------------------------------------------
struct PairArgs {
  const long long *keys[kMaxHeight];
  const int *ilist[kMaxHeight];
  long long start[kMaxHeight + 1];  // first cell of each level in the concatenation of levels l0..l1
  int l0, l1;
};
constexpr int PAIR_CELLS = 32, PAIR_THREADS = 256;  // cells per block

__device__ __forceinline__ int pair_level(const PairArgs &a, long long g) {
  int l = a.l0;
  while (l < a.l1 && g >= a.start[l + 1]) ++l;
  return l;
}

// PLACE false: pairs per slot.  PLACE true: each block reserves room in every slot's list and writes its pairs there
// (their order within a slot is free: each pair's row of D is summed by itself).
template <bool PLACE>
__global__ void __launch_bounds__(PAIR_THREADS) pair_kernel(const __grid_constant__ PairArgs a,
                                                            const IListTable *__restrict__ tab, int *__restrict__ cnt,
                                                            int *__restrict__ psrc, int *__restrict__ ppos) {
  __shared__ int h[343], base[343];
  __shared__ short slot[8][189];
  for (int t = threadIdx.x; t < 343; t += PAIR_THREADS) h[t] = 0;
  for (int t = threadIdx.x; t < 8 * 189; t += PAIR_THREADS) slot[t / 189][t % 189] = tab->slot[t / 189][t % 189];
  __syncthreads();
  const long long g0 = (long long)blockIdx.x * PAIR_CELLS, g1 = min(g0 + PAIR_CELLS, a.start[a.l1 + 1]);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int pass = 0; pass < (PLACE ? 2 : 1); ++pass) {
    for (long long g = g0 + w; g < g1; g += PAIR_THREADS / 32) {
      const int l = pair_level(a, g);
      const long long c = g - a.start[l];
      const int ct = (int)(a.keys[l][c] & 7);
      for (int e = lane; e < 189; e += 32) {
        const int src = a.ilist[l][c * 189 + e];
        if (pass == 0) {
          if (src >= 0) atomicAdd(&h[slot[ct][e]], 1);
        } else {
          int pos = -1;
          if (src >= 0) {
            const int t = slot[ct][e];
            pos = base[t] + atomicAdd(&h[t], 1);
            psrc[pos] = (l << 27) | src;
          }
          ppos[g * 189 + e] = pos;
        }
      }
    }
    __syncthreads();
    if (pass == 0) {
      for (int t = threadIdx.x; t < 343; t += PAIR_THREADS) {
        const int v = h[t];
        if (v) base[t] = atomicAdd(cnt + t, v);
        h[t] = 0;
      }
      __syncthreads();
    }
  }
}

// Counts to first pairs and first tiles of each slot; the counts become the slots' cursors.
__global__ void __launch_bounds__(384) pair_scan_kernel(int *__restrict__ tab) {
  __shared__ long long ws[12];
  int *first = tab, *tile = tab + 344, *cnt = tab + 688;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int v = t < 343 ? cnt[t] : 0;
  long long x = ((long long)((v + G_BN - 1) / G_BN) << 32) | (unsigned)v;  // tiles and pairs in one scan
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[w] = x;
  __syncthreads();
  for (int q = 0; q < w; ++q) x += ws[q];
  if (t < 343) {
    first[t + 1] = (int)(x & 0xffffffffll);
    tile[t + 1] = (int)(x >> 32);
    cnt[t] = (int)(x & 0xffffffffll) - v;
    if (t == 0) first[0] = tile[0] = 0;
  }
}

// L[c][rhs][m] += scale * the sum of c's rows of D whose slots lie in [s0, s1), in the order of c's list.
struct PairSumArgs {
  PairArgs tree;
  const IListTable *itab;
  const int *ppos;
  const double *D;
  long long drhs;
  int first;  // first pair of the chunk
  int s0, s1, nn, R;
  double scale[kMaxHeight];
  double *L[kMaxHeight];
};
__global__ void __launch_bounds__(128) pair_sum_kernel(const __grid_constant__ PairSumArgs a) {
  __shared__ int row[192];
  __shared__ int wcnt[6];
  const long long g = blockIdx.x;
  const int l = pair_level(a.tree, g);
  const long long c = g - a.tree.start[l];
  const int ct = (int)(a.tree.keys[l][c] & 7);
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  // the present entries, compacted in order: entries t and t + 128
  int pos[2];
  unsigned act[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int e = t + u * 128;
    pos[u] = -1;
    if (e < 189) {
      const int s = a.itab->slot[ct][e];
      if (s >= a.s0 && s < a.s1) pos[u] = a.ppos[g * 189 + e];
    }
    act[u] = __ballot_sync(0xffffffffu, pos[u] >= 0);
    if (lane == 0 && u * 4 + w < 6) wcnt[u * 4 + w] = __popc(act[u]);
  }
  __syncthreads();
  int n = 0;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    if (k == w && pos[0] >= 0) row[n + __popc(act[0] & ((1u << lane) - 1u))] = pos[0] - a.first;
    if (k == w + 4 && pos[1] >= 0) row[n + __popc(act[1] & ((1u << lane) - 1u))] = pos[1] - a.first;
    n += wcnt[k];
  }
  __syncthreads();
  const double *D = a.D + (long long)blockIdx.y * a.drhs;
  double *Lc = a.L[l] + (c * a.R + blockIdx.y) * a.nn;
  for (int m = t; m < a.nn; m += 128) {
    double s = 0.0;
#pragma unroll 8
    for (int k = 0; k < n; ++k) s += __ldcs(D + (long long)row[k] * a.nn + m);
    Lc[m] += a.scale[l] * s;
  }
}

// ---- the GEMM ------------------------------------------------------------------------------------------
struct GemmArgs {
  int nn, lda;
  int l0, l1;              // Y, TILES: levels of this launch
  int mtiles, split;       // row tiles (Y: of the parity with most rows), K ranges per tile
  int ng;                  // TILES: K groups of every operator, where they all have the same number, else 0
  unsigned ng_inv;         // 2^32 / ng, rounded up
  const int *list;         // cells grouped by parity; PAIRS: source cells grouped by slot
  const int *tab;          // counts, list starts, first tiles (parity_scan_kernel, pair_scan_kernel)
  int s0, s1, first;       // PAIRS: slots of this launch and their first pair
  double scale[kMaxHeight];
  const double *X[kMaxHeight];   // the cells' vectors: multipoles; TILES of the symmetric form: Y
  long long xstride, xrhs;       // from cell to cell, from right-hand side to right-hand side
  double *out[kMaxHeight];       // Y; TILES: locals; PAIRS: [0] is D
  long long ostride, orhs;
  const int *ilist[kMaxHeight];  // [ncells][189]
  const double *A;
  const int4 *ent;               // TILES: [8][189]
  long long a_off[8];            // Y
  int a_ld[8], rows[8];
  double *part;
  int *tick;
};

__device__ __forceinline__ void cp16(void *dst, const void *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp8(void *dst, const void *src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

template <int MB>
constexpr size_t gemm64_stage_bytes() {
  return sizeof(double) * (G_BK * (16 * MB + 4) + G_BN * G_LDB);
}

// Y:     out[cell][row]  = sum_k Vs[row][k] X[cell][k], cells of one parity
// PAIRS: out[pair][row]  = sum_k K_t[row][k] X[source][k], pairs of one slot t
// TILES: out[cell][row] += scale * sum over the transfer vectors e of child type ct of
//        sum_k A_e[row][k] X[ilist[cell][e]][xoff_e + k]
// V16: a cell's vector starts on a 16-byte boundary (Y, and multipoles of even p^3).
enum GemmMode { G_Y, G_PAIRS, G_TILES };

template <int MB, int MODE, bool V16>
__global__ void __launch_bounds__(G_THREADS, 2) gemm64_kernel(const __grid_constant__ GemmArgs a) {
  constexpr int LDA = 16 * MB + 4;  // shared-memory row of a K row: conflict-free fragment loads
  constexpr int ROWP = 8 * MB;      // 16-byte pieces of a K row
  constexpr int NU = V16 ? 2 : 4;   // copies per thread of a stage of B (16 or 8 bytes each)
  constexpr int NS = MODE == G_TILES ? 189 : 1;
  extern __shared__ __align__(16) double sh[];
  double *As = sh;                                     // [stage][16][LDA]
  double *Bs = sh + G_STAGES * G_BK * LDA;             // [stage][64][G_LDB]
  unsigned short *grp = (unsigned short *)(Bs + G_STAGES * G_BN * G_LDB);  // TILES: entry and group of each K group
  __shared__ int cells[G_BN];
  __shared__ int e_row[NS], e_x[NS], e_k[NS];          // the transfer vectors that occur in this tile
  __shared__ unsigned char e_id[NS], e_mask[NS], e_any[8][NS];  // e_mask: the tile's blocks of 8 cells that have it
  __shared__ int s_groups, s_last;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;

  // the tile: 64 cells of one (level, parity) or 64 pairs of one slot, its rows and its K range
  const int *first = MODE == G_PAIRS ? a.tab + 344 : a.tab + 2 * kMaxHeight * 8;
  int k0 = MODE == G_PAIRS ? a.s0 : (kMaxHeight - 1 - a.l1) * 8;
  int k1 = MODE == G_PAIRS ? a.s1 : (kMaxHeight - a.l0) * 8;
  const int split = blockIdx.x % a.split, item = blockIdx.x / a.split, mt = item % a.mtiles;
  const int tile = first[k0] + item / a.mtiles;
  if (tile >= first[k1]) return;
  while (k1 - k0 > 1) {  // the last list whose first tile is <= tile
    const int mid = (k0 + k1) >> 1;
    if (first[mid] <= tile)
      k0 = mid;
    else
      k1 = mid;
  }
  const int level = MODE == G_PAIRS ? 0 : kMaxHeight - 1 - (k0 >> 3), ct = MODE == G_PAIRS ? 0 : k0 & 7;
  if (MODE == G_Y && mt * 16 * MB >= a.rows[ct]) return;
  const int n0 = (tile - first[k0]) * G_BN;
  const int l_start = MODE == G_PAIRS ? a.tab[k0] : a.tab[kMaxHeight * 8 + level * 8 + ct];
  const int l_count = MODE == G_PAIRS ? a.tab[k0 + 1] - l_start : a.tab[level * 8 + ct];
  const int ntile = min(G_BN, l_count - n0);
  if (tid < G_BN) cells[tid] = tid < ntile ? a.list[l_start + n0 + tid] : -1;
  __syncthreads();

  // K groups of 4: of the one operator, or of the transfer vectors that some cell of the tile has
  int groups;
  const int *il = nullptr;
  if (MODE == G_TILES) {
    il = a.ilist[level];
    // e_any[b][e]: some cell of block b (8 cells, one warp each) has a source at entry e
    const int nb = min(8, ntile - w * 8);
    for (int e = lane; e < 189; e += 32) {
      bool any = false;
      for (int u = 0; u < nb; ++u) any |= il[(long long)cells[w * 8 + u] * 189 + e] >= 0;
      e_any[w][e] = any ? 1 : 0;
    }
    __syncthreads();
    if (w == 0) {
      int ne = 0, ng = 0;
      for (int e0 = 0; e0 < 189; e0 += 32) {
        const int e = e0 + lane;
        unsigned m = 0;
        if (e < 189)
#pragma unroll
          for (int b = 0; b < 8; ++b) m |= (unsigned)e_any[b][e] << b;
        const int4 en = e < 189 ? a.ent[ct * 189 + e] : make_int4(0, 0, 0, 0);
        const int gk = m ? (en.z + 3) >> 2 : 0;
        const unsigned act = __ballot_sync(0xffffffffu, gk > 0);
        int x = gk;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        const int ei = ne + __popc(act & ((1u << lane) - 1u)), g0 = ng + x - gk;
        if (gk > 0) {
          e_row[ei] = en.x;
          e_x[ei] = en.y;
          e_k[ei] = en.z;
          e_id[ei] = (unsigned char)e;
          e_mask[ei] = (unsigned char)m;
          if (!a.ng)
            for (int g = 0; g < gk; ++g) grp[g0 + g] = (unsigned short)(ei | (g << 8));
        }
        ne += __popc(act);
        ng += __shfl_sync(0xffffffffu, x, 31);
      }
      if (lane == 0) s_groups = ng;
    }
    __syncthreads();
    groups = s_groups;
  } else {
    groups = (a.nn + 3) >> 2;
  }
  const int nst = (groups + 3) >> 2;
  const int st0 = (int)((long long)nst * split / a.split), st1 = (int)((long long)nst * (split + 1) / a.split);

  // TILES: entry (of the tile's list) and group within it of K group q: from the table, or by division where every
  // operator has the same number of groups (dense operators)
  auto locate = [&](int q, int &ei, int &gi) {
    if (a.ng) {
      ei = (int)__umulhi((unsigned)q, a.ng_inv);
      gi = q - ei * a.ng;
    } else {
      const unsigned v = grp[q];
      ei = (int)(v & 255u);
      gi = (int)(v >> 8);
    }
  };
  // loaders.  A: warp w copies K rows 2w, 2w + 1 of a stage (group w / 2).  B: the 16 values of a stage of one cell
  // by 8 (16) consecutive threads, so that a warp's copies fall on whole 128-byte lines.
  const int lda = MODE == G_Y ? a.a_ld[ct] : a.lda;
  const double *A = a.A + (MODE == G_Y ? a.a_off[ct] : MODE == G_PAIRS ? (long long)k0 * a.nn * lda : 0) + mt * 16 * MB;
  const int pieces = min(ROWP, (lda - mt * 16 * MB) >> 1);
  const int bc = V16 ? tid >> 3 : tid >> 4;             // cells bc, bc + 256 / (8 or 16), ...
  const int bk = V16 ? 2 * (tid & 7) : tid & 15;        // K position within the stage
  const double *X = a.X[MODE == G_PAIRS ? a.l0 : level] + (long long)blockIdx.y * a.xrhs;
  const double *bp[MODE == G_TILES ? 1 : NU];           // Y, PAIRS: the cells' vectors at this thread's K position
  int src[MODE == G_TILES ? NU : 1];                    // TILES: sources of the next stage to copy (read ahead)
  if (MODE != G_TILES) {
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      const int c = cells[bc + u * (G_BN / NU)];
      const double *base = MODE == G_PAIRS && c >= 0 ? a.X[c >> 27] + (long long)blockIdx.y * a.xrhs : X;
      bp[u] = c < 0 ? nullptr : base + (long long)(MODE == G_PAIRS ? c & 0x7ffffff : c) * a.xstride + bk;
    }
  }
  auto sources = [&](int st) {
    if (MODE == G_TILES) {
      const int q = st * 4 + (bk >> 2);
      int e = -1;
      if (st < st1 && q < groups) {
        int ei, gi;
        locate(q, ei, gi);
        e = e_id[ei];
      }
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const int c = cells[bc + u * (G_BN / NU)];
        src[u] = e >= 0 && c >= 0 ? il[(long long)c * 189 + e] : -1;
      }
    }
  };
  auto load = [&](int st) {
    const int s = st % G_STAGES;
    {
      const int q = st * 4 + (w >> 1);
      if (q < groups) {
        int ei = 0, gi = q;
        if (MODE == G_TILES) locate(q, ei, gi);
        const int K = MODE == G_TILES ? e_k[ei] : a.nn;
        const long long r0 = MODE == G_TILES ? e_row[ei] : 0;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int k = gi * 4 + ((2 * w + u) & 3);
          const double *g = A + (r0 + (k < K ? k : 0)) * lda;
          double *d = As + (s * G_BK + 2 * w + u) * LDA;
          for (int c = lane; c < pieces; c += 32) cp16(d + 2 * c, g + 2 * c, k < K ? 16 : 0);
        }
      }
    }
    double *d = Bs + (s * G_BN + bc) * G_LDB + bk;
    if (MODE == G_TILES) {
      const int q = st * 4 + (bk >> 2);
      if (q < groups) {
        int ei, gi;
        locate(q, ei, gi);
        const int k = gi * 4 + (bk & 3), left = e_k[ei] - k;  // valid values from this position on
        const int bytes = left <= 0 ? 0 : V16 && left > 1 ? 16 : 8;
#pragma unroll
        for (int u = 0; u < NU; ++u) {
          const double *g = src[u] >= 0 && left > 0 ? X + (long long)src[u] * a.xstride + e_x[ei] + k : X;
          if (V16)
            cp16(d + u * (G_BN / NU) * G_LDB, g, src[u] >= 0 ? bytes : 0);
          else
            cp8(d + u * (G_BN / NU) * G_LDB, g, src[u] >= 0 ? bytes : 0);
        }
      }
    } else {
      const bool in = st * G_BK + bk < a.nn;
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const bool ok = in && bp[u];
        const double *g = ok ? bp[u] + st * G_BK : X;
        if (V16)
          cp16(d + u * (G_BN / NU) * G_LDB, g, ok ? 16 : 0);
        else
          cp8(d + u * (G_BN / NU) * G_LDB, g, ok ? 8 : 0);
      }
    }
    cp_commit();
  };

  const int wm = w & 1, wn = w >> 1;  // rows wm * MB blocks, cells wn * 2 blocks
  double acc[MB][2][2];
#pragma unroll
  for (int i = 0; i < MB; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  sources(st0);
#pragma unroll
  for (int u = 0; u < G_STAGES - 1; ++u) {
    if (st0 + u < st1)
      load(st0 + u);
    else
      cp_commit();
    sources(st0 + u + 1);
  }
  const bool own = wn * 16 < ntile;  // Y, PAIRS: the tile has cells of this warp's
  const int ar = (lane & 3) * LDA + wm * MB * 8 + (lane >> 2);
  const int br = (wn * 16 + (lane >> 2)) * G_LDB + (lane & 3);
  for (int st = st0; st < st1; ++st) {
    cp_wait<G_STAGES - 2>();
    __syncthreads();
    if (st + G_STAGES - 1 < st1)
      load(st + G_STAGES - 1);
    else
      cp_commit();
    sources(st + G_STAGES);
    const double *as = As + (st % G_STAGES) * G_BK * LDA + ar;
    const double *bs = Bs + (st % G_STAGES) * G_BN * G_LDB + br;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int q = st * 4 + g;
      if (q >= groups) break;
      unsigned m = 3u;
      if (MODE != G_TILES && !own) break;
      if (MODE == G_TILES) {
        int ei, gi;
        locate(q, ei, gi);
        m = (e_mask[ei] >> (2 * wn)) & 3u;
      }
      if (!m) continue;
      double av[MB];
#pragma unroll
      for (int i = 0; i < MB; ++i) av[i] = as[g * 4 * LDA + i * 8];
      if (m & 1u) {
        const double b = bs[g * 4];
#pragma unroll
        for (int i = 0; i < MB; ++i) dmma(acc[i][0], av[i], b);
      }
      if (m & 2u) {
        const double b = bs[g * 4 + 8 * G_LDB];
#pragma unroll
        for (int i = 0; i < MB; ++i) dmma(acc[i][1], av[i], b);
      }
    }
  }
  cp_wait<0>();

  // lane holds rows lane / 4 (+ 8 i) of cells 2 (lane % 4), + 1 (+ 8 j)
  const int row0 = mt * 16 * MB + wm * MB * 8 + (lane >> 2);
  const int rows = MODE == G_Y ? a.rows[ct] : a.nn;
  double *out = a.out[level] + (long long)blockIdx.y * a.orhs;
  if (MODE != G_TILES) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int n = wn * 16 + j * 8 + 2 * (lane & 3) + u;
        if (n >= ntile) continue;
        double *o = out + (MODE == G_PAIRS ? (long long)(l_start - a.first + n0 + n) : (long long)cells[n]) * a.ostride;
#pragma unroll
        for (int i = 0; i < MB; ++i)
          if (row0 + 8 * i < rows) o[row0 + 8 * i] = acc[i][j][u];
      }
    return;
  }
  const double scale = a.scale[level];
  if (a.split > 1) {
    // partial sums [split][thread's values][thread]; the last CTA of the tile adds them in the order of the ranges
    const long long slot = (long long)blockIdx.y * (gridDim.x / a.split) + item;
    double *part = a.part + slot * a.split * (MB * 4 * G_THREADS) + tid;
#pragma unroll
    for (int i = 0; i < MB; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int u = 0; u < 2; ++u)
          part[((long long)split * MB * 4 + i * 4 + j * 2 + u) * G_THREADS] = acc[i][j][u];
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(a.tick + slot, 1) == a.split - 1;
    __syncthreads();
    if (!s_last) return;
    if (tid == 0) a.tick[slot] = 0;  // ready for the next launch
    __threadfence();
#pragma unroll
    for (int i = 0; i < MB; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          double s = 0.0;
          for (int k = 0; k < a.split; ++k)
            s += __ldcg(part + ((long long)k * MB * 4 + i * 4 + j * 2 + u) * G_THREADS);
          acc[i][j][u] = s;
        }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int n = wn * 16 + j * 8 + 2 * (lane & 3) + u;
      if (n >= ntile) continue;
      double *o = out + (long long)cells[n] * a.ostride;
#pragma unroll
      for (int i = 0; i < MB; ++i)
        if (row0 + 8 * i < rows) o[row0 + 8 * i] += scale * acc[i][j][u];
    }
}

// out[m][row] = Vt[foff + m * rank + q] for the row's (foff, rank, q); rank 0: a padding row
__global__ void gather_vs_kernel(int ld, int nn, const int3 *__restrict__ rows, const double *__restrict__ Vt,
                                 double *__restrict__ out) {
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (g >= (long long)ld * nn) return;
  const int3 r = rows[g % ld];
  out[g] = r.y > 0 ? Vt[r.x + (g / ld) * r.y + r.z] : 0.0;
}
// out[k][m] = Ut[foff + m * rank + q] for operator row k's (foff, rank, q), zero for m >= nn
__global__ void gather_a_kernel(long long nrows, int nn, int lda, const int3 *__restrict__ rows,
                                const double *__restrict__ Ut, double *__restrict__ out) {
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (g >= nrows * lda) return;
  const int m = (int)(g % lda);
  const int3 r = rows[g / lda];
  out[g] = m < nn ? Ut[r.x + (long long)m * r.y + r.z] : 0.0;
}

int sm_count(const Context &c) {
  int v = 148;
  cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, c.device);
  return v > 0 ? v : 148;
}

int source_parity(const IListTable &t, int ct, int e) {
  const int px = (((ct >> 2) & 1) + t.off[ct][e][0]) & 1, py = (((ct >> 1) & 1) + t.off[ct][e][1]) & 1,
            pz = ((ct & 1) + t.off[ct][e][2]) & 1;
  return (px << 2) | (py << 1) | pz;
}

b200fmm_status upload_entries(Context &c, Sym64 *s, const std::vector<int4> &ent) {
  for (int ct = 0; ct < 8; ++ct) {
    int g = 0;
    for (int e = 0; e < 189; ++e) g += (ent[ct * 189 + e].z + 3) / 4;
    s->max_groups = std::max(s->max_groups, g);
  }
  B200_CUDA(cudaMalloc(&s->d_ent, sizeof(int4) * ent.size()));
  B200_CUDA(cudaMemcpy(s->d_ent, ent.data(), sizeof(int4) * ent.size(), cudaMemcpyHostToDevice));
  B200_CUDA(cudaMalloc(&s->d_ptab, sizeof(int) * (3 * kMaxHeight * 8 + 1)));
  return B200FMM_OK;
}

}  // namespace

void sym64_free(Context &c) {
  Sym64 *s = c.s64;
  if (!s) return;
  for (void *p : {(void *)s->d_vs, (void *)(s->dense ? nullptr : s->d_a), (void *)s->d_ent, (void *)s->d_plist,
                  (void *)s->d_ptab, (void *)s->d_pblk, (void *)s->d_y, (void *)s->d_part, (void *)s->d_tick,
                  (void *)s->d_pairtab, (void *)s->d_psrc, (void *)s->d_ppos, (void *)s->d_d})
    if (p) cudaFree(p);
  delete s;
  c.s64 = nullptr;
}

// The operators of both phases, gathered on the device from the per-slot factors (d_Ut, d_Vt: row-major p^3 x r
// each, at the slot's offset toff).
b200fmm_status sym64_prepare(Context &c, const double *d_Ut, const double *d_Vt, const std::vector<long long> &toff,
                             const std::vector<int> &trank) {
  sym64_free(c);
  Sym64 *s = new Sym64();
  c.s64 = s;
  const int nn = c.nn;
  s->lda = (nn + 7) & ~7;
  // the slots each source parity feeds: entry e of child type ct reads the cell at offset itab.off[ct][e], whose
  // parity is ct's parity plus that offset, per axis.  Each slot's rows of Y start at a multiple of 2, so that 16-byte
  // copies are aligned.
  std::vector<int> ybase(8 * 343, -1);
  std::vector<int3> vrows;
  std::vector<long long> vfirst(8);
  long long vs_total = 0;
  for (int sp = 0; sp < 8; ++sp) {
    std::vector<char> fed(343, 0);
    for (int ct = 0; ct < 8; ++ct)
      for (int e = 0; e < c.itab.n[ct]; ++e)
        if (source_parity(c.itab, ct, e) == sp) fed[c.itab.slot[ct][e]] = 1;
    vfirst[sp] = (long long)vrows.size();
    for (int t = 0; t < 343; ++t)
      if (fed[t]) {
        if (toff[t] < 0) return fail(B200FMM_ERR_INVALID, "symmetric operators: a far slot has no factor");
        ybase[sp * 343 + t] = (int)(vrows.size() - vfirst[sp]);
        for (int q = 0; q < ((trank[t] + 1) & ~1); ++q)
          vrows.push_back(q < trank[t] ? make_int3((int)toff[t], trank[t], q) : make_int3(0, 0, 0));
        s->yrank[sp] += trank[t];
      }
    s->ysum[sp] = (int)(vrows.size() - vfirst[sp]);
    while ((vrows.size() - vfirst[sp]) & 7) vrows.push_back(make_int3(0, 0, 0));
    s->ldv[sp] = (int)(vrows.size() - vfirst[sp]);
    s->vs_off[sp] = vs_total;
    vs_total += (long long)s->ldv[sp] * nn;
    s->ystride = std::max(s->ystride, s->ysum[sp]);
  }
  std::vector<int3> arows;
  std::vector<int> afirst(343, 0);
  for (int t = 0; t < 343; ++t) {
    afirst[t] = (int)arows.size();
    if (toff[t] >= 0)
      for (int q = 0; q < trank[t]; ++q) arows.push_back(make_int3((int)toff[t], trank[t], q));
  }
  std::vector<int4> ent(8 * 189, make_int4(0, 0, 0, 0));
  for (int ct = 0; ct < 8; ++ct)
    for (int e = 0; e < c.itab.n[ct]; ++e) {
      const int t = c.itab.slot[ct][e];
      ent[ct * 189 + e] = make_int4(afirst[t], ybase[source_parity(c.itab, ct, e) * 343 + t], trank[t], 0);
    }
  int3 *d_vrows = nullptr, *d_arows = nullptr;
  const long long na = (long long)arows.size();
  B200_CUDA(cudaMalloc(&s->d_vs, sizeof(double) * std::max<long long>(vs_total, 1)));
  B200_CUDA(cudaMalloc(&s->d_a, sizeof(double) * std::max<long long>(na * s->lda, 1)));
  B200_CHECK(upload_entries(c, s, ent));
  B200_CUDA(cudaMalloc(&d_vrows, sizeof(int3) * std::max<size_t>(vrows.size(), 1)));
  B200_CUDA(cudaMalloc(&d_arows, sizeof(int3) * std::max<size_t>(arows.size(), 1)));
  B200_CUDA(cudaMemcpy(d_vrows, vrows.data(), sizeof(int3) * vrows.size(), cudaMemcpyHostToDevice));
  B200_CUDA(cudaMemcpy(d_arows, arows.data(), sizeof(int3) * arows.size(), cudaMemcpyHostToDevice));
  for (int sp = 0; sp < 8; ++sp)
    if (s->ldv[sp] > 0)
      gather_vs_kernel<<<grid_for((long long)s->ldv[sp] * nn, 256), 256>>>(s->ldv[sp], nn, d_vrows + vfirst[sp], d_Vt,
                                                                          s->d_vs + s->vs_off[sp]);
  if (na > 0) gather_a_kernel<<<grid_for(na * s->lda, 256), 256>>>(na, nn, s->lda, d_arows, d_Ut, s->d_a);
  B200_CUDA(cudaGetLastError());
  B200_CUDA(cudaDeviceSynchronize());
  cudaFree(d_vrows);
  cudaFree(d_arows);
  return B200FMM_OK;
}

// The dense operators d_dense [343][n][m] as phase-2 operators, in place (their rows are a multiple of 8 values).
b200fmm_status dense64_prepare(Context &c) {
  sym64_free(c);
  Sym64 *s = new Sym64();
  c.s64 = s;
  s->dense = true;
  const int nn = c.nn;
  s->lda = (nn + 7) & ~7;
  std::vector<int4> ent(8 * 189, make_int4(0, 0, 0, 0));
  for (int ct = 0; ct < 8; ++ct)
    for (int e = 0; e < c.itab.n[ct]; ++e) ent[ct * 189 + e] = make_int4(c.itab.slot[ct][e] * nn, 0, nn, 0);
  B200_CHECK(upload_entries(c, s, ent));
  B200_CUDA(cudaMalloc(&s->d_pairtab, sizeof(int) * (2 * 344 + 343)));
  s->d_a = c.d_dense;
  return B200FMM_OK;
}

bool sym64_fed_ranks(const Context &c, double *fed) {
  if (!c.s64 || c.s64->dense) return false;
  for (int p = 0; p < 8; ++p) fed[p] = c.s64->yrank[p];
  return true;
}

namespace {

constexpr size_t kYCap = (size_t)16 << 30;    // most bytes of Y for one right-hand side
constexpr size_t kYBatch = (size_t)2 << 30;   // several right-hand sides share a launch up to this

template <class T>
b200fmm_status grow64(T *&p, size_t &cap, size_t n) {
  if (p && n <= cap) return B200FMM_OK;
  if (p) B200_CUDA(cudaFree(p));
  p = nullptr;
  cap = 0;
  B200_CUDA(cudaMalloc((void **)&p, sizeof(T) * std::max<size_t>(n, 1)));
  cap = n;
  return B200FMM_OK;
}

// CTAs that share the K ranges of split tiles: about four per resident slot (two per SM).  tiles * split stays at or
// below this, so that partial sums for so many serve every call and never move.
long long part_slots(const Context &c) { return 4LL * 2 * sm_count(c); }

// The buffers of the current tree's M2L: settled by its first call, for all levels and for each alone, and kept until
// the next tree, so that none that a captured evaluation holds moves.  Nothing is allocated inside a capture: there
// the buffers of an earlier tree serve where they are large enough, else B200FMM_ERR_UNSUPPORTED.
b200fmm_status tree_room(Context &c) {
  Sym64 &s = *c.s64;
  if (s.room_serial == c.tree_serial) return B200FMM_OK;
  const size_t per = sizeof(double) * (size_t)s.ystride;
  size_t total = 0, blocks = 0, largest = 0;  // largest: cells of the largest level within the cap
  for (int l = 2; l < c.H; ++l) {
    const size_t n = (size_t)c.lv[l].n;
    total += n;
    blocks += (n + PB_CELLS - 1) / PB_CELLS;
    if (per * n <= kYCap) largest = std::max(largest, n);
  }
  if (stream_captured(c)) {
    if (s.cap_list < total || s.cap_pblk < blocks * 8 || (!s.dense && s.cap_y < largest * s.ystride))
      return fail(B200FMM_ERR_UNSUPPORTED, "FP64 M2L: its buffers are allocated by an evaluation that is not captured");
  } else {
    B200_CHECK(grow64(s.d_plist, s.cap_list, total));
    B200_CHECK(grow64(s.d_pblk, s.cap_pblk, blocks * 8));
    if (!s.dense) {
      // Y of every level, of as many right-hand sides as share a launch; fewer where there is no room for that
      b200fmm_status st = B200FMM_ERR_OOM;
      if (per * total <= kYCap)
        for (size_t rb = std::min<size_t>(c.R, std::max<size_t>(1, kYBatch / std::max<size_t>(1, per * total)));
             rb > 0 && st != B200FMM_OK; rb /= 2) {
          st = grow64(s.d_y, s.cap_y, rb * total * s.ystride);
          if (st != B200FMM_OK) cudaGetLastError();
        }
      if (st != B200FMM_OK) B200_CHECK(grow64(s.d_y, s.cap_y, largest * s.ystride));
    }
  }
  s.room_serial = c.tree_serial;
  return B200FMM_OK;
}

// Parity lists of the current tree, once per tree (a graph builds its own).
b200fmm_status parity_lists(Context &c) {
  Sym64 &s = *c.s64;
  if (s.list_serial == c.tree_serial) return B200FMM_OK;
  const int LL = c.H - 1;
  long long total = 0;
  int blocks = 0;
  ListArgs la{};
  la.l0 = 2;
  la.l1 = LL;
  for (int l = 2; l <= LL; ++l) {
    la.keys[l] = c.lv[l].keys;
    la.n[l] = c.lv[l].n;
    la.loff[l] = total;
    la.blk0[l] = blocks;
    total += c.lv[l].n;
    blocks += (int)((c.lv[l].n + PB_CELLS - 1) / PB_CELLS);
  }
  la.blk0[LL + 1] = blocks;
  parity_count_kernel<<<blocks, PB_THREADS, 0, c.stream>>>(la, s.d_pblk);
  parity_scan_kernel<<<1, 256, 0, c.stream>>>(la, s.d_pblk, s.d_ptab);
  parity_place_kernel<<<blocks, PB_THREADS, 0, c.stream>>>(la, s.d_pblk, s.d_ptab, s.d_plist);
  c.launches += 3;
  B200_CUDA(cudaGetLastError());
  if (!stream_captured(c)) s.list_serial = c.tree_serial;
  return B200FMM_OK;
}

// Room for D: the pairs of as many slots as fit kDBytes (at least the largest slot), all right-hand sides of a share.
constexpr size_t kDBytes = (size_t)1 << 30;
constexpr size_t kPairTables = (size_t)8 << 30;  // most bytes of the pair tables
constexpr int kPairOrder = 5;                    // lowest order of the pair form

PairArgs pair_args(const Context &c) {
  PairArgs a{};
  a.l0 = 2;
  a.l1 = c.H - 1;
  a.start[2] = 0;
  for (int l = 2; l <= a.l1; ++l) {
    a.keys[l] = c.lv[l].keys;
    a.ilist[l] = c.lv[l].ilist;
    a.start[l + 1] = a.start[l] + c.lv[l].n;
  }
  return a;
}

template <int MB, int MODE, bool V16>
b200fmm_status launch_gemm64(const GemmArgs &a, dim3 grid, size_t sh, cudaStream_t st) {
  B200_CUDA(cudaFuncSetAttribute(gemm64_kernel<MB, MODE, V16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh));
  gemm64_kernel<MB, MODE, V16><<<grid, G_THREADS, sh, st>>>(a);
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

// Levels l0..l1.  Y (symmetric form) holds the levels of the call, one after the other.
b200fmm_status gemm64_levels(Context &c, int l0, int l1) {
  Sym64 &s = *c.s64;
  GemmArgs a{};
  long long cells = 0, tiles = 0, yoff[kMaxHeight] = {0};
  for (int l = l0; l <= l1; ++l) {
    yoff[l] = cells;
    cells += c.lv[l].n;
    if (c.lv[l].n) tiles += (c.lv[l].n + G_BN - 1) / G_BN + 8;  // bounds the tiles of the level's 8 parities
    a.scale[l] = 2.0 / (c.cfg.box_width / (double)(1LL << l));
    a.ilist[l] = c.lv[l].ilist;
  }
  if (cells == 0) return B200FMM_OK;
  a.nn = c.nn;
  a.l0 = l0;
  a.l1 = l1;
  a.list = s.d_plist;
  a.tab = s.d_ptab;
  // right-hand sides that share a launch: as many as Y's room holds (tree_room)
  int rb = c.R;
  const size_t ycells = (size_t)cells * s.ystride;
  if (!s.dense) {
    const size_t share = std::min(s.cap_y / ycells, std::max<size_t>(1, kYBatch / (sizeof(double) * ycells)));
    if (share == 0) return fail(B200FMM_ERR_STATE, "FP64 M2L: no room for Y");
    rb = (int)std::min<size_t>(c.R, share);
  }
  const int mb = g_mb(c.p), nblk = (c.nn + 7) / 8;
  const int mtiles = (nblk + 2 * mb - 1) / (2 * mb);
  for (int r0 = 0; r0 < c.R; r0 += rb) {
    const int nr = std::min(rb, c.R - r0);
    if (!s.dense) {
      GemmArgs b = a;
      for (int l = l0; l <= l1; ++l) {
        b.X[l] = c.lv[l].M + (size_t)r0 * c.nn;
        b.out[l] = s.d_y + (size_t)yoff[l] * s.ystride;
      }
      b.xstride = (long long)c.R * c.nn;
      b.xrhs = c.nn;
      b.ostride = s.ystride;
      b.orhs = (long long)ycells;
      b.A = s.d_vs;
      int rows = 0;
      for (int p = 0; p < 8; ++p) {
        b.a_off[p] = s.vs_off[p];
        b.a_ld[p] = s.ldv[p];
        b.rows[p] = s.ysum[p];
        rows = std::max(rows, s.ysum[p]);
      }
      b.mtiles = (rows + 16 * G_Y_MB - 1) / (16 * G_Y_MB);
      b.split = 1;
      const dim3 grid((unsigned)(tiles * b.mtiles), nr);
      const size_t sh = G_STAGES * gemm64_stage_bytes<G_Y_MB>();
      if (c.nn % 2 == 0)
        B200_CHECK((launch_gemm64<G_Y_MB, G_Y, true>(b, grid, sh, c.stream)));
      else
        B200_CHECK((launch_gemm64<G_Y_MB, G_Y, false>(b, grid, sh, c.stream)));
      ++c.launches;
    }
    GemmArgs b = a;
    for (int l = l0; l <= l1; ++l) {
      b.X[l] = s.dense ? c.lv[l].M + (size_t)r0 * c.nn : s.d_y + (size_t)yoff[l] * s.ystride;
      b.out[l] = c.lv[l].L + (size_t)r0 * c.nn;
    }
    b.xstride = s.dense ? (long long)c.R * c.nn : s.ystride;
    b.xrhs = s.dense ? c.nn : (long long)ycells;
    b.ostride = (long long)c.R * c.nn;
    b.orhs = c.nn;
    b.A = s.d_a;
    b.lda = s.lda;
    b.ent = s.d_ent;
    b.mtiles = mtiles;
    if (s.dense) {
      b.ng = (c.nn + 3) / 4;
      b.ng_inv = (unsigned)(((1ull << 32) + b.ng - 1) / b.ng);
    }
    // K ranges per tile where the tiles alone are fewer than part_slots
    const long long items = tiles * mtiles * nr, slots = part_slots(c);
    b.split = (int)std::max<long long>(1, std::min<long long>(kMaxSplit, slots / items));
    if (b.split > 1 && !s.d_part) {
      const size_t part = sizeof(double) * (size_t)slots * mb * 4 * G_THREADS;
      // nothing is allocated inside a capture; unsplit tiles also where there is no room
      if (stream_captured(c)) {
        b.split = 1;
      } else if ((!s.d_tick && cudaMalloc(&s.d_tick, sizeof(int) * slots) != cudaSuccess) ||
                 cudaMalloc(&s.d_part, part) != cudaSuccess) {
        cudaGetLastError();
        s.d_part = nullptr;
        b.split = 1;
      } else {
        B200_CUDA(cudaMemsetAsync(s.d_tick, 0, sizeof(int) * slots, c.stream));
      }
    }
    b.part = s.d_part;
    b.tick = s.d_tick;
    const dim3 grid((unsigned)(tiles * mtiles * b.split), nr);
    const size_t groups = s.dense ? 0 : (size_t)s.max_groups * sizeof(unsigned short);
#define B200_G64(P)                                                                \
  case P: {                                                                        \
    constexpr int MB = g_mb(P);                                                    \
    const size_t sh = G_STAGES * gemm64_stage_bytes<MB>() + groups;                \
    if (s.dense)                                                                   \
      B200_CHECK((launch_gemm64<MB, G_TILES, P % 2 == 0>(b, grid, sh, c.stream))); \
    else                                                                           \
      B200_CHECK((launch_gemm64<MB, G_TILES, true>(b, grid, sh, c.stream)));       \
    break;                                                                         \
  }
    switch (c.p) {
      B200_G64(3) B200_G64(4) B200_G64(5) B200_G64(6) B200_G64(7) B200_G64(8)
      default: return fail(B200FMM_ERR_UNSUPPORTED, "order not built");
    }
#undef B200_G64
    ++c.launches;
  }
  return B200FMM_OK;
}

// Every level of a tree with pair tables, chunk by chunk of slots.
b200fmm_status pairs_levels(Context &c) {
  Sym64 &s = *c.s64;
  const int LL = c.H - 1;
  const int mb = g_mb(c.p), nblk = (c.nn + 7) / 8;
  GemmArgs a{};
  PairSumArgs ps{};
  ps.tree = pair_args(c);
  ps.itab = c.d_itab;
  ps.ppos = s.d_ppos;
  ps.nn = c.nn;
  ps.R = c.R;
  a.nn = c.nn;
  a.lda = s.lda;
  a.l0 = 2;
  a.l1 = LL;
  a.mtiles = (nblk + 2 * mb - 1) / (2 * mb);
  a.split = 1;
  a.list = s.d_psrc;
  a.tab = s.d_pairtab;
  a.xstride = (long long)c.R * c.nn;
  a.xrhs = c.nn;
  a.ostride = c.nn;
  a.A = s.d_a;
  const long long cells = ps.tree.start[LL + 1];
  const long long room = (long long)(s.cap_d / c.nn);  // rows of D
  for (int s0 = 0; s0 < 343;) {
    int s1 = s0 + 1;
    while (s1 < 343 && s.h_first[s1 + 1] - (long long)s.h_first[s0] <= room) ++s1;
    const long long np = s.h_first[s1] - (long long)s.h_first[s0];
    if (np > 0) {
      const int rb = (int)std::max<long long>(1, std::min<long long>(c.R, room / np));
      for (int r0 = 0; r0 < c.R; r0 += rb) {
        const int nr = std::min(rb, c.R - r0);
        a.s0 = s0;
        a.s1 = s1;
        a.first = ps.first = s.h_first[s0];
        ps.s0 = s0;
        ps.s1 = s1;
        a.out[0] = s.d_d;
        a.orhs = ps.drhs = np * c.nn;
        ps.D = s.d_d;
        for (int l = 2; l <= LL; ++l) {
          a.X[l] = c.lv[l].M + (size_t)r0 * c.nn;
          ps.L[l] = c.lv[l].L + (size_t)r0 * c.nn;
          ps.scale[l] = 2.0 / (c.cfg.box_width / (double)(1LL << l));
        }
        const long long tiles = (np + G_BN - 1) / G_BN + (s1 - s0);  // bounds the tiles of these slots
        const dim3 grid((unsigned)(tiles * a.mtiles), nr);
#define B200_G64(P)                                                                       \
  case P: {                                                                               \
    static_assert(P >= kPairOrder, "the pair form is built for the orders that take it"); \
    constexpr int MB = g_mb(P);                                                           \
    const size_t sh = G_STAGES * gemm64_stage_bytes<MB>();                                \
    B200_CHECK((launch_gemm64<MB, G_PAIRS, P % 2 == 0>(a, grid, sh, c.stream)));          \
    break;                                                                                \
  }
        switch (c.p) {
          B200_G64(5) B200_G64(6) B200_G64(7) B200_G64(8)
          default: return fail(B200FMM_ERR_UNSUPPORTED, "order not built");
        }
#undef B200_G64
        pair_sum_kernel<<<dim3((unsigned)cells, nr), 128, 0, c.stream>>>(ps);
        c.launches += 2;
      }
    }
    s0 = s1;
  }
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

}  // namespace

// What set_particles does for the dense forms: it queues the pair counts and their copy to the host, and once it has
// waited for them, the buffers of the tile form are sized, so that a first evaluation may be captured.
b200fmm_status dense64_tree_counts(Context &c, int *host_first) {
  Sym64 &s = *c.s64;
  s.pairs = false;
  const PairArgs pa = pair_args(c);
  const long long cells = pa.start[c.H];
  // pair positions are int, source cells 27 bits: above, and where the tables would be too large, the tile form
  if (c.p < kPairOrder || cells * 189 >= 2147483647LL || cells >= (1LL << 27) ||
      sizeof(int) * 2 * 189 * (size_t)cells > kPairTables)
    return B200FMM_OK;
  int *cnt = s.d_pairtab + 688;
  B200_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * 343, c.stream));
  const unsigned blocks = grid_for(cells, PAIR_CELLS);
  pair_kernel<false><<<blocks, PAIR_THREADS, 0, c.stream>>>(pa, c.d_itab, cnt, nullptr, nullptr);
  pair_scan_kernel<<<1, 384, 0, c.stream>>>(s.d_pairtab);
  B200_CUDA(cudaGetLastError());
  B200_CUDA(cudaMemcpyAsync(host_first, s.d_pairtab, sizeof(int) * 344, cudaMemcpyDeviceToHost, c.stream));
  c.tree_launches += 2;
  s.pairs = true;
  return B200FMM_OK;
}

b200fmm_status dense64_tree(Context &c, const int *host_first) {
  Sym64 &s = *c.s64;
  if (s.pairs)
    for (int t = 0; t < 344; ++t) s.h_first[t] = host_first[t];
  return tree_room(c);
}

// The pair form's tables and D, by the first evaluation of a tree that wants the M2L of all its levels (before P2M,
// beside the near field).  Inside a capture nothing is allocated: an evaluation that finds no tables takes the tile
// form, as do near-field or single-level calls, which need none.
b200fmm_status dense64_pairs(Context &c) {
  Sym64 &s = *c.s64;
  if (!s.pairs || s.pair_serial == c.tree_serial || stream_captured(c)) return B200FMM_OK;
  const PairArgs pa = pair_args(c);
  const long long cells = pa.start[c.H], np = s.h_first[343];
  long long largest = 1;
  for (int t = 0; t < 343; ++t) largest = std::max<long long>(largest, s.h_first[t + 1] - s.h_first[t]);
  const size_t row = sizeof(double) * c.nn;
  size_t rows = std::max<size_t>((size_t)largest, std::min<size_t>((size_t)np * c.R, kDBytes / row));
  // an eighth of the device stays free for what an evaluation cannot do without (a batch keeps many handles)
  size_t avail = 0, device = 0;
  const size_t nsrc = (size_t)std::max<long long>(np, 1), npos = (size_t)cells * 189;
  auto more = [](size_t cap, size_t n, size_t bytes) { return n > cap ? (n - cap) * bytes : (size_t)0; };
  const size_t tables = more(s.cap_psrc, nsrc, sizeof(int)) + more(s.cap_ppos, npos, sizeof(int));
  auto fits = [&] {
    const size_t need = tables + more(s.cap_d, rows * c.nn, sizeof(double));
    if (need > 0 && device == 0) {
      B200_CUDA(cudaMemGetInfo(&avail, &device));
      avail -= std::min(avail, device / 8);
    }
    return need <= avail ? B200FMM_OK : B200FMM_ERR_OOM;
  };
  while (rows > (size_t)largest && fits() != B200FMM_OK) rows = std::max<size_t>((size_t)largest, rows / 2);
  bool ok = fits() == B200FMM_OK && grow64(s.d_psrc, s.cap_psrc, nsrc) == B200FMM_OK &&
            grow64(s.d_ppos, s.cap_ppos, npos) == B200FMM_OK;
  while (ok && s.cap_d < rows * c.nn && grow64(s.d_d, s.cap_d, rows * c.nn) != B200FMM_OK) {
    cudaGetLastError();
    if (rows == (size_t)largest) ok = false;
    rows = std::max<size_t>((size_t)largest, rows / 2);
  }
  if (!ok) {
    cudaGetLastError();
    s.pairs = false;  // no room: the tile form
    return B200FMM_OK;
  }
  pair_kernel<true><<<grid_for(cells, PAIR_CELLS), PAIR_THREADS, 0, c.stream>>>(pa, c.d_itab, s.d_pairtab + 688,
                                                                               s.d_psrc, s.d_ppos);
  ++c.launches;
  B200_CUDA(cudaGetLastError());
  s.pair_serial = c.tree_serial;
  return B200FMM_OK;
}

// One level, or every level with level < 0.  Returns B200FMM_ERR_UNSUPPORTED before any launch when Y of the
// largest level of the call would exceed the cap, or when a capture finds no buffers for this tree, so that the
// caller keeps the per-target kernel.
b200fmm_status run_m2l_gemm64(Context &c, int level) {
  Sym64 &s = *c.s64;
  const int LL = c.H - 1;
  const int l0 = level < 0 ? 2 : level, l1 = level < 0 ? LL : level;
  long long total = 0, nmax = 0;
  for (int l = l0; l <= l1; ++l) {
    total += c.lv[l].n;
    nmax = std::max(nmax, c.lv[l].n);
  }
  const size_t per = sizeof(double) * (size_t)s.ystride;
  if (!s.dense && per * nmax > kYCap)
    return fail(B200FMM_ERR_UNSUPPORTED, "FP64 M2L: Y of the largest level exceeds 16 GiB");
  if (s.dense && level < 0) {
    B200_CHECK(dense64_pairs(c));
    if (s.pairs && s.pair_serial == c.tree_serial) return pairs_levels(c);
  }
  B200_CHECK(tree_room(c));
  B200_CHECK(parity_lists(c));
  // Y of every level at once, or level by level where there is no room for that
  if (s.dense || l0 == l1 || s.cap_y >= (size_t)total * s.ystride) return gemm64_levels(c, l0, l1);
  for (int l = l0; l <= l1; ++l) B200_CHECK(gemm64_levels(c, l, l));
  return B200FMM_OK;
}

}  // namespace b200
