// Tree construction on the GPU -- integer work, bit-exact with the reference's rules:
//   leaf coordinate  FCoordinateComputer::GetTreeCoordinate (Src/Containers/FCoordinateComputer.hpp:16-40)
//   Morton key       FTreeCoordinate::getMortonIndex (Src/Containers/FTreeCoordinate.hpp:91-113)
//   leaf order       FOctree::insert appends in input order -> a stable sort by key
//   leaf neighbours  FTreeCoordinate::getNeighborsIndexes (FTreeCoordinate.hpp:189-216)
//   interaction list FTreeCoordinate::getInteractionNeighbors (FTreeCoordinate.hpp:219-264)
//
// The sorts (particles by leaf key, leaves by column) are stable LSD radix sorts with 8-bit digits: a histogram per
// tile, its prefix over the tiles, a scatter with ranks within a warp by __match_any_sync; particle keys have
// 3*(height-1) significant bits, two passes at height 6.
//
// A tree of a few thousand particles is bound by the number of dependent launches (2-4 us each), not by their work,
// so what can share a launch does: the first histogram with the keys, the prefix over few tiles with the scatter, all
// clears of a tree in one kernel, and the compactions of leaves, levels and records take their blocks' offsets from
// the earlier blocks' counts instead of a scan of their own (at most 2,048 blocks).  Together with the interaction
// lists of full levels by key instead of search: set_particles of 1M points 0.31 -> 0.24 ms; a whole evaluation of
// 2,003 points from host arrays 0.505 -> 0.415 ms, of 20,000 points in FP64 0.74 -> 0.66 ms.
#include "common.cuh"

#include <algorithm>
#include <cstring>

namespace b200 {

namespace {

constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 8;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS8_BINS = 256;  // 8-bit digits: each warp of a tile owns 256 consecutive items (8 rounds of 32)
static_assert(RS_THREADS == RS8_BINS && RS_ITEMS == 8, "one thread per digit; 8 rounds of 32 items per warp");

// --------------------------------------------------------------------------------------------------
// keys, with the histogram of their first digit
// --------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(RS_THREADS) keys_kernel(
    long long n, const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ z, double cx,
    double cy, double cz, double box_width, double leaf_width, int height, unsigned long long *__restrict__ keys,
    int *__restrict__ vals, int *__restrict__ err, unsigned *__restrict__ counts, unsigned *__restrict__ total) {
  __shared__ unsigned h[RS8_BINS];
  h[threadIdx.x] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * RS_TILE;
  const int last = (1 << (height - 1)) - 1;
#pragma unroll 2
  for (int k = 0; k < RS_ITEMS; ++k) {
    const long long i = base + k * RS_THREADS + threadIdx.x;
    if (i >= n) break;
    const double r[3] = {x[i] - cx, y[i] - cy, z[i] - cz};
    int c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (!(r[d] >= 0.0 && r[d] <= box_width)) {  // also rejects NaN
        atomicExch(err, 1);
        c[d] = 0;
      } else if (r[d] == box_width) {
        c[d] = last;
      } else {
        c[d] = (int)(r[d] / leaf_width);
        if (c[d] > last) c[d] = last;  // unreachable for in-box input; keeps the key in range
      }
    }
    const unsigned long long key = (unsigned long long)morton_encode3(c[0], c[1], c[2]);
    keys[i] = key;
    vals[i] = (int)i;
    atomicAdd(&h[key & (RS8_BINS - 1)], 1u);
  }
  __syncthreads();
  counts[(long long)blockIdx.x * RS8_BINS + threadIdx.x] = h[threadIdx.x];
  if (h[threadIdx.x]) atomicAdd(total + threadIdx.x, h[threadIdx.x]);
}

// --------------------------------------------------------------------------------------------------
// radix sort
// --------------------------------------------------------------------------------------------------
// Histogram of one tile: counts[block][digit], and the digits' totals.
__global__ void rs8_hist(const unsigned long long *__restrict__ keys, long long n, int shift,
                         unsigned *__restrict__ counts, unsigned *__restrict__ total) {
  __shared__ unsigned h[RS8_BINS];
  h[threadIdx.x] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * RS_TILE;
#pragma unroll
  for (int k = 0; k < RS_ITEMS; ++k) {
    const long long i = base + k * RS_THREADS + threadIdx.x;
    if (i < n) atomicAdd(&h[(keys[i] >> shift) & (RS8_BINS - 1)], 1u);
  }
  __syncthreads();
  counts[(long long)blockIdx.x * RS8_BINS + threadIdx.x] = h[threadIdx.x];
  if (h[threadIdx.x]) atomicAdd(total + threadIdx.x, h[threadIdx.x]);
}

// counts[block][digit] to the counts of the blocks before, in place: a CTA per 32 digits, its 32 warps each a range
// of blocks.
__global__ void __launch_bounds__(1024) rs8_prefix(unsigned *__restrict__ counts, long long nblocks) {
  __shared__ unsigned part[32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned *c = counts + blockIdx.x * 32 + lane;
  const long long b0 = nblocks * w / 32, b1 = nblocks * (w + 1) / 32;
  unsigned s = 0;
#pragma unroll 8
  for (long long b = b0; b < b1; ++b) s += c[b * RS8_BINS];
  part[w][lane] = s;
  __syncthreads();
  unsigned run = 0;
  for (int q = 0; q < w; ++q) run += part[q][lane];
#pragma unroll 8
  for (long long b = b0; b < b1; ++b) {
    const unsigned v = c[b * RS8_BINS];
    c[b * RS8_BINS] = run;
    run += v;
  }
}

// Exclusive prefix over the block's threads; total is the sum.  ws: 33 words of shared memory.
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned *ws, unsigned &total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[w] = x;
  __syncthreads();
  if (w == 0) {
    unsigned t = lane < (int)(blockDim.x >> 5) ? ws[lane] : 0u, u = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, u, o);
      if (lane >= o) u += y;
    }
    ws[lane] = u - t;
    if (lane == 31) ws[32] = u;
  }
  __syncthreads();
  const unsigned r = ws[w] + x - v;
  total = ws[32];
  __syncthreads();
  return r;
}

// Stable scatter of one tile.  Warp w owns the tile's items [256 w, 256 w + 256), taken in 8 rounds of 32
// consecutive items; within a round the lanes with the same digit find each other (__match_any_sync) and
// rank by lane, and per-warp running counts carry the ranks across rounds.  An item's position is the
// tile's global offset for its digit (the totals of the smaller digits and the counts of the tiles before: PREFIX
// says that counts holds those, else they are added up here), plus the items of that digit in the tile's earlier
// warps, plus its rank in its own warp: input order is kept within every digit.
template <bool PREFIX>
__global__ void __launch_bounds__(RS_THREADS) rs8_scatter(const unsigned long long *__restrict__ kin,
                                                          const int *__restrict__ vin,
                                                          unsigned long long *__restrict__ kout,
                                                          int *__restrict__ vout, long long n, int shift,
                                                          const unsigned *__restrict__ counts,
                                                          const unsigned *__restrict__ total) {
  constexpr int W = RS_THREADS / 32;
  __shared__ unsigned ws[33];
  __shared__ unsigned wc[W][RS8_BINS];  // per-warp counts, then the counts of the warps before
  __shared__ unsigned boff[RS8_BINS];
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
#pragma unroll
  for (int k = 0; k < W; ++k) wc[k][t] = 0;
  unsigned before = 0, all;
  if (PREFIX) {
    before = counts[(long long)blockIdx.x * RS8_BINS + t];
  } else {
#pragma unroll 8
    for (int b = 0; b < (int)blockIdx.x; ++b) before += counts[b * RS8_BINS + t];
  }
  boff[t] = before + block_exclusive_scan(total[t], ws, all);
  __syncthreads();
  const long long base = (long long)blockIdx.x * RS_TILE + (long long)w * (32 * RS_ITEMS);
  const unsigned lt = (1u << lane) - 1u;
  unsigned long long k[RS_ITEMS];
  int v[RS_ITEMS], dg[RS_ITEMS];
  unsigned rank[RS_ITEMS];
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    const long long i = base + j * 32 + lane;
    const bool ok = i < n;
    k[j] = ok ? kin[i] : 0ull;
    v[j] = ok ? vin[i] : 0;
    dg[j] = ok ? (int)((k[j] >> shift) & (RS8_BINS - 1)) : RS8_BINS;
    const unsigned peers = __match_any_sync(0xffffffffu, dg[j]);
    const unsigned before = ok ? wc[w][dg[j]] : 0u;
    rank[j] = before + __popc(peers & lt);
    __syncwarp();
    if (ok && (peers & lt) == 0) wc[w][dg[j]] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  {
    // thread t: digit t, exclusive prefix over the warps
    unsigned run = 0;
#pragma unroll
    for (int q = 0; q < W; ++q) {
      const unsigned c = wc[q][t];
      wc[q][t] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < RS_ITEMS; ++j) {
    if (dg[j] >= RS8_BINS) continue;
    const unsigned pos = boff[dg[j]] + wc[w][dg[j]] + rank[j];
    kout[pos] = k[j];
    vout[pos] = v[j];
  }
}

// --------------------------------------------------------------------------------------------------
// tree arrays
// --------------------------------------------------------------------------------------------------
__global__ void gather_particles(long long n, int R, const int *__restrict__ perm, const double *__restrict__ x,
                                 const double *__restrict__ y, const double *__restrict__ z,
                                 const double *__restrict__ q, double *__restrict__ xs, double *__restrict__ ys,
                                 double *__restrict__ zs, double *__restrict__ qs, long long *__restrict__ perm64,
                                 int *__restrict__ iperm) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long j = perm[i];
  xs[i] = x[j];
  ys[i] = y[j];
  zs[i] = z[j];
  for (int r = 0; r < R; ++r) qs[(long long)r * n + i] = q[(long long)r * n + j];
  perm64[i] = j;
  iperm[j] = (int)i;
}

__global__ void gather_charges(long long n, int R, const long long *__restrict__ perm, const double *__restrict__ q,
                               double *__restrict__ qs) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long j = perm[i];
  for (int r = 0; r < R; ++r) qs[(long long)r * n + i] = q[(long long)r * n + j];
}

// Blocks of the passes below take `chunk` consecutive items each, at most kMaxBlocks blocks, so that a block can add
// up the counts of all blocks before it.
constexpr int kMaxBlocks = 2048, CB_T = 1024;
__host__ __device__ inline long long chunk_of(long long n) {
  const long long c = (n + kMaxBlocks - 1) / kMaxBlocks;
  return (c + CB_T - 1) / CB_T * CB_T;
}
// sum of v[0 .. blockIdx.x) (every thread of a CB_T-thread block gets it)
__device__ __forceinline__ long long sum_before(const long long *__restrict__ v, long long *ws) {
  long long s = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += CB_T) s += v[b];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  s = 0;
#pragma unroll
  for (int k = 0; k < CB_T / 32; ++k) s += ws[k];
  __syncthreads();
  return s;
}

// cells of every level 0..LL: one per change of the sorted particle key above that level's bits, counted per warp
// (ballot), then per block in shared memory, then one atomic per block and level; the leaves of each block go to heads
__global__ void __launch_bounds__(CB_T) level_counts_kernel(long long n, long long chunk,
                                                            const unsigned long long *__restrict__ keys, int LL,
                                                            long long *__restrict__ heads,
                                                            unsigned long long *__restrict__ counts) {
  __shared__ unsigned bc[kMaxHeight];
  if (threadIdx.x < kMaxHeight) bc[threadIdx.x] = 0;
  __syncthreads();
  const long long end = min(n, (blockIdx.x + 1) * chunk);
  const int lane = threadIdx.x & 31;
  for (long long i0 = blockIdx.x * chunk; i0 < end; i0 += CB_T) {
    const long long i = i0 + threadIdx.x;
    const unsigned long long k = i < n ? keys[i] : 0ull, kp = (i > 0 && i < n) ? keys[i - 1] : 0ull;
    for (int l = 0; l <= LL; ++l) {
      const int shift = 3 * (LL - l);
      const bool head = i < n && (i == 0 || (k >> shift) != (kp >> shift));
      const unsigned m = __ballot_sync(0xffffffffu, head);
      if (lane == 0 && m) atomicAdd(&bc[l], (unsigned)__popc(m));
    }
  }
  __syncthreads();
  if (threadIdx.x <= LL && bc[threadIdx.x]) atomicAdd(counts + threadIdx.x, (unsigned long long)bc[threadIdx.x]);
  if (threadIdx.x == 0) heads[blockIdx.x] = bc[LL];
}

__global__ void __launch_bounds__(CB_T) compact_leaves(long long n, long long chunk,
                                                       const unsigned long long *__restrict__ keys,
                                                       const long long *__restrict__ heads,
                                                       long long *__restrict__ leaf_keys,
                                                       long long *__restrict__ leaf_start) {
  __shared__ long long wl[CB_T / 32];
  __shared__ unsigned ws[33];
  long long idx = sum_before(heads, wl);
  const long long end = min(n, (blockIdx.x + 1) * chunk);
  for (long long i0 = blockIdx.x * chunk; i0 < end; i0 += CB_T) {
    const long long i = i0 + threadIdx.x;
    const unsigned long long k = i < n ? keys[i] : 0ull;
    const bool head = i < n && (i == 0 || k != keys[i - 1]);
    unsigned total;
    const unsigned ex = block_exclusive_scan(head ? 1u : 0u, ws, total);
    if (head) {
      leaf_keys[idx + ex] = (long long)k;
      leaf_start[idx + ex] = i;
    }
    idx += total;
  }
  if (end == n && threadIdx.x == 0) leaf_start[idx] = n;
}

constexpr int CL_WORDS = 4096;  // 8-byte words per block
__global__ void __launch_bounds__(256) clear_kernel(const __grid_constant__ ClearArgs a) {
  int k = 0;
  while (k + 1 < a.count && blockIdx.x >= a.first[k + 1]) ++k;
  const unsigned long long v = a.ones[k] ? ~0ull : 0ull;
  const long long w0 = (long long)(blockIdx.x - a.first[k]) * CL_WORDS, w1 = min(a.n[k], w0 + CL_WORDS);
  unsigned long long *p = a.p[k];
  for (long long i = w0 + 2 * threadIdx.x; i < w1; i += 512) {
    if (i + 1 < w1)
      *reinterpret_cast<ulonglong2 *>(p + i) = make_ulonglong2(v, v);
    else
      p[i] = v;
  }
}
void add_state(ClearList &cl, Context &c) {
  for (int l = 2; l < c.H; ++l) {
    const size_t bytes = sizeof(double) * (size_t)c.lv[l].n * c.R * c.nn;
    cl.add(c.lv[l].M, bytes, false);
    cl.add(c.lv[l].L, bytes, false);
  }
  cl.add(c.d_res, sizeof(double4) * (size_t)c.N * c.R, false);
}

// ---- upper levels of the tree, all at once from the sorted leaf keys ---------------------------------
// Cell c of level l < LL starts at the first leaf whose key >> 3(LL - l) differs from its predecessor's;
// a leaf's cell index at level l is the number of such starts up to it, minus one.  At most three launches for
// all levels: per-block start counts, their exclusive scans, then keys and parent/child links; up to ML_SUM blocks
// the last one adds up the earlier blocks' counts itself, and one block needs none.
constexpr int ML_T = 1024, ML_SUM = 256;
struct LevelLinks {
  long long *keys[kMaxHeight];
  int *parent[kMaxHeight];
  int *child[kMaxHeight];
};

__global__ void ml_count_kernel(long long nl, const long long *__restrict__ K, int LL, unsigned *__restrict__ bcount,
                                int nblk) {
  __shared__ unsigned ws[33];
  const long long i = (long long)blockIdx.x * ML_T + threadIdx.x;
  const long long k = i < nl ? K[i] : 0, kp = (i > 0 && i < nl) ? K[i - 1] : 0;
  for (int l = 0; l < LL; ++l) {
    const int sh = 3 * (LL - l);
    const bool head = i < nl && (i == 0 || (k >> sh) != (kp >> sh));
    unsigned total;
    block_exclusive_scan(head ? 1u : 0u, ws, total);
    if (threadIdx.x == 0) bcount[(long long)l * nblk + blockIdx.x] = total;
  }
}

__global__ void ml_scan_kernel(unsigned *__restrict__ bcount, int nblk) {
  __shared__ unsigned ws[33];
  unsigned *b = bcount + (long long)blockIdx.x * nblk;
  unsigned carry = 0;
  for (int base = 0; base < nblk; base += ML_T) {
    const int j = base + threadIdx.x;
    const unsigned v = j < nblk ? b[j] : 0u;
    unsigned total;
    const unsigned ex = block_exclusive_scan(v, ws, total);
    if (j < nblk) b[j] = carry + ex;
    carry += total;
  }
}

__global__ void ml_build_kernel(long long nl, const long long *__restrict__ K, int LL,
                                const unsigned *__restrict__ boff, int nblk, LevelLinks P) {
  __shared__ unsigned ws[33];
  __shared__ unsigned before[kMaxHeight];  // starts of the earlier blocks, by level
  if (nblk <= ML_SUM) {
    const int l = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (l < LL) {
      unsigned s = 0;
      for (int b = lane; b < (int)blockIdx.x; b += 32) s += boff[(long long)l * nblk + b];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) before[l] = s;
    }
  } else if (threadIdx.x < LL) {
    before[threadIdx.x] = boff[(long long)threadIdx.x * nblk + blockIdx.x];
  }
  __syncthreads();
  const long long i = (long long)blockIdx.x * ML_T + threadIdx.x;
  const long long k = i < nl ? K[i] : 0, kp = (i > 0 && i < nl) ? K[i - 1] : 0;
  int idx_next = (int)i;  // this leaf's cell at level l + 1 (at LL: the leaf itself)
  bool head_next = true;  // the leaf starts that cell
  for (int l = LL - 1; l >= 0; --l) {
    const int sh = 3 * (LL - l);
    const bool head = i < nl && (i == 0 || (k >> sh) != (kp >> sh));
    unsigned total;
    const unsigned ex = block_exclusive_scan(head ? 1u : 0u, ws, total);
    const int idx = (int)(before[l] + ex) + (head ? 1 : 0) - 1;
    if (i < nl) {
      if (head) P.keys[l][idx] = k >> sh;
      if (head_next) {
        P.parent[l + 1][idx_next] = idx;
        P.child[l][(long long)idx * 8 + ((k >> (sh - 3)) & 7)] = idx_next;
      }
    }
    idx_next = idx;
    head_next = head;
  }
}

// interaction lists and dense grids of every level in one launch each: block b serves cell b of the
// concatenated levels 2..LL
struct LevelCellsT {
  const long long *keys[kMaxHeight];
  int *ilist[kMaxHeight];
  int *grid[kMaxHeight];
  long long start[kMaxHeight + 1];
  int l0, l1;
};

__device__ __forceinline__ int level_at(const LevelCellsT &C, long long g) {
  int l = C.l0;
  while (l < C.l1 && g >= C.start[l + 1]) ++l;
  return l;
}

// One thread per (leaf, neighbour position).  In a full leaf level (every cell a leaf) leaf i has Morton key
// i, so the neighbour's index is its key; otherwise it is found by binary search.
__global__ void leaf_neighbors_kernel(long long nleaves, const long long *__restrict__ keys, int height, int full,
                                      int *__restrict__ nbr) {
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (g >= nleaves * 27) return;
  const long long c = g / 27;
  const int p = (int)(g % 27);
  int ix, iy, iz;
  morton_decode3(keys[c], ix, iy, iz);
  const int lim = 1 << (height - 1);
  const int dx = p / 9 - 1, dy = (p / 3) % 3 - 1, dz = p % 3 - 1;
  int v = -1;
  if (p == 13) {
    v = (int)c;
  } else if (ix + dx >= 0 && ix + dx < lim && iy + dy >= 0 && iy + dy < lim && iz + dz >= 0 && iz + dz < lim) {
    const long long key = morton_encode3(ix + dx, iy + dy, iz + dz);
    v = full ? (int)key : find_key(keys, nleaves, key);
  }
  nbr[g] = v;
}

__global__ void ilist_kernel(const __grid_constant__ LevelCellsT C, const IListTable *__restrict__ tab) {
  const int level = level_at(C, blockIdx.x);
  const long long c = blockIdx.x - C.start[level];
  const long long ncells = C.start[level + 1] - C.start[level];
  const long long *__restrict__ keys = C.keys[level];
  int *__restrict__ ilist = C.ilist[level];
  int ix, iy, iz;
  const long long key = keys[c];
  morton_decode3(key, ix, iy, iz);
  const int ct = (int)(key & 7);
  const int lim = 1 << level;
  const bool full = ncells == 1LL << (3 * level);  // every cell present: a cell's index is its key
  for (int e = threadIdx.x; e < 189; e += blockDim.x) {
    const int sx = ix + tab->off[ct][e][0], sy = iy + tab->off[ct][e][1], sz = iz + tab->off[ct][e][2];
    int v = -1;
    if (sx >= 0 && sx < lim && sy >= 0 && sy < lim && sz >= 0 && sz < lim)
      v = full ? (int)morton_encode3(sx, sy, sz) : find_key(keys, ncells, morton_encode3(sx, sy, sz));
    ilist[c * 189 + e] = v;
  }
}

__global__ void grid_index_kernel(const __grid_constant__ LevelCellsT C) {
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (g >= C.start[C.l1 + 1]) return;
  const int level = level_at(C, g);
  const long long c = g - C.start[level];
  const long long *__restrict__ keys = C.keys[level];
  int *__restrict__ grid = C.grid[level];
  int ix, iy, iz;
  morton_decode3(keys[c], ix, iy, iz);
  const long long side = 1LL << level;
  grid[((long long)iz * side + iy) * side + ix] = (int)c;
}

// column key of a leaf: (x, y) of its cell; a stable sort by it from Morton order (monotone in z inside a
// column) puts the three z-neighbours of every column next to each other
__global__ void leaf_column_keys(long long nleaves, const long long *__restrict__ keys, int LL,
                                 unsigned long long *__restrict__ k, int *__restrict__ v) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= nleaves) return;
  int ix, iy, iz;
  morton_decode3(keys[i], ix, iy, iz);
  k[i] = ((unsigned long long)ix << LL) | (unsigned long long)iy;
  v[i] = (int)i;
}

// Column order, source records and work items of the near field, chunk by chunk of leaves (chunk_of).  COLUMNS: the
// leaf at position r of the column order is order[r]; without order, in a full leaf level (every cell a leaf, so leaf
// i has Morton key i), the leaf at r = (x * side + y) * side + z is the cell (x, y, z).  The work items
// (p2p_leaf_items) go leaf by leaf.
struct NearArgs {
  long long nl, chunk;
  int LL, whole, item;
  const int *order;
  const long long *leaf_start;
  int *rank_of;
  long long *rec_base, *chunk_base;
  long long *recs, *items;  // per block
};
__device__ __forceinline__ int column_leaf(const NearArgs &a, long long r) {
  if (a.order) return a.order[r];
  const int side = 1 << a.LL;
  return (int)morton_encode3((int)(r >> (2 * a.LL)), (int)(r >> a.LL) & (side - 1), (int)r & (side - 1));
}
template <bool COLUMNS>
__device__ __forceinline__ void near_counts(const NearArgs &a, long long r, unsigned &rec, unsigned &it, int &leaf) {
  rec = it = 0;
  leaf = 0;
  if (r >= a.nl) return;
  it = (unsigned)p2p_leaf_items(a.leaf_start[r + 1] - a.leaf_start[r], a.whole, a.item);
  if (COLUMNS) {
    leaf = column_leaf(a, r);
    rec = (unsigned)((a.leaf_start[leaf + 1] - a.leaf_start[leaf] + 1) >> 1);  // two particles per record
  }
}
template <bool COLUMNS>
__global__ void __launch_bounds__(CB_T) near_sums_kernel(const __grid_constant__ NearArgs a) {
  __shared__ unsigned long long sum[2];
  if (threadIdx.x < 2) sum[threadIdx.x] = 0;
  __syncthreads();
  unsigned long long s[2] = {0, 0};
  const long long end = min(a.nl, (blockIdx.x + 1) * a.chunk);
  for (long long r = blockIdx.x * a.chunk + threadIdx.x; r < end; r += CB_T) {
    unsigned rec, it;
    int leaf;
    near_counts<COLUMNS>(a, r, rec, it, leaf);
    s[0] += rec;
    s[1] += it;
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
    if ((threadIdx.x & 31) == 0 && s[k]) atomicAdd(&sum[k], s[k]);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a.recs[blockIdx.x] = (long long)sum[0];
    a.items[blockIdx.x] = (long long)sum[1];
  }
}
template <bool COLUMNS>
__global__ void __launch_bounds__(CB_T) near_bases_kernel(const __grid_constant__ NearArgs a) {
  __shared__ long long wl[CB_T / 32];
  __shared__ unsigned ws[33];
  long long rec0 = COLUMNS ? sum_before(a.recs, wl) : 0, it0 = sum_before(a.items, wl);
  const long long end = min(a.nl, (blockIdx.x + 1) * a.chunk);
  for (long long r0 = blockIdx.x * a.chunk; r0 < end; r0 += CB_T) {
    const long long r = r0 + threadIdx.x;
    unsigned rec, it, total;
    int leaf;
    near_counts<COLUMNS>(a, r, rec, it, leaf);
    if (COLUMNS) {
      const unsigned ex = block_exclusive_scan(rec, ws, total);
      if (r < a.nl) {
        a.rec_base[r] = rec0 + ex;
        a.rank_of[leaf] = (int)r;
      }
      rec0 += total;
    }
    const unsigned ex = block_exclusive_scan(it, ws, total);
    if (r < a.nl) a.chunk_base[r] = it0 + ex;
    it0 += total;
  }
  if (end == a.nl && threadIdx.x == 0) {
    if (COLUMNS) a.rec_base[a.nl] = rec0;
    a.chunk_base[a.nl] = it0;
  }
}

// grow-only device buffer: reallocates (and bumps the tree generation) only when n exceeds the capacity
template <class T>
b200fmm_status grow(Context &c, T *&p, size_t &cap, size_t n) {
  if (p && n <= cap) return B200FMM_OK;
  if (p) cudaFree(p);
  p = nullptr;
  const size_t nc = std::max<size_t>(n, cap + cap / 4);
  B200_CUDA(cudaMalloc((void **)&p, sizeof(T) * std::max<size_t>(nc, 1)));
  cap = nc;
  ++c.tree_gen;
  return B200FMM_OK;
}

// Stable LSD radix sort of (key, value) over `bits` bits, tile counts in d_cnt, digit totals (zeroed by the caller,
// 256 words per pass) in total; `hist` says that the first pass's histogram is there.  k0, v0 end up with the result.
constexpr int RS_SUM = 64;  // tiles up to which the scatter adds up the earlier tiles' counts itself
b200fmm_status radix_sort(Context &c, unsigned long long *&k0, unsigned long long *&k1, int *&v0, int *&v1, long long n,
                          int bits, unsigned *total, bool hist, long long &launches) {
  const long long nb = (n + RS_TILE - 1) / RS_TILE;
  unsigned *cnt = c.d_cnt;
  for (int sh = 0; sh < bits; sh += 8, total += RS8_BINS) {
    if (sh > 0 || !hist) {
      rs8_hist<<<(unsigned)nb, RS_THREADS, 0, c.stream>>>(k0, n, sh, cnt, total);
      ++launches;
    }
    if (nb > RS_SUM) {
      rs8_prefix<<<RS8_BINS / 32, 1024, 0, c.stream>>>(cnt, nb);
      rs8_scatter<true><<<(unsigned)nb, RS_THREADS, 0, c.stream>>>(k0, v0, k1, v1, n, sh, cnt, total);
      ++launches;
    } else {
      rs8_scatter<false><<<(unsigned)nb, RS_THREADS, 0, c.stream>>>(k0, v0, k1, v1, n, sh, cnt, total);
    }
    ++launches;
    std::swap(k0, k1);
    std::swap(v0, v1);
  }
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

// d_err: the domain error flag; from byte 16 the cell count of each level; then the digit totals of the sort
constexpr size_t kErrTotals = 16 + sizeof(unsigned long long) * kMaxHeight;
constexpr int kSortPasses = (3 * (kMaxHeight - 1) + 7) / 8;
constexpr size_t kErrBytes = kErrTotals + sizeof(unsigned) * RS8_BINS * kSortPasses;

template <class T>
void dfree(T *&p) {
  if (p) cudaFree(p);
  p = nullptr;
}

}  // namespace

void ClearList::add(void *p, size_t bytes, bool ones) {
  if (!bytes) return;
  const int k = a.count++;
  a.p[k] = (unsigned long long *)p;
  a.n[k] = (long long)(bytes / 8);
  a.ones[k] = ones ? 1 : 0;
  a.first[k + 1] = a.first[k] + (unsigned)((a.n[k] + CL_WORDS - 1) / CL_WORDS);
}
b200fmm_status ClearList::launch(cudaStream_t s) {
  if (a.count) clear_kernel<<<a.first[a.count], 256, 0, s>>>(a);
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

void free_tree(Context &c) {
  dfree(c.d_x);
  dfree(c.d_y);
  dfree(c.d_z);
  dfree(c.d_q);
  dfree(c.d_perm);
  dfree(c.d_leaf_start);
  dfree(c.d_leaf_nbr);
  dfree(c.d_leaf_rank);
  dfree(c.d_rec_base);
  dfree(c.d_chunk_base);
  dfree(c.d_pq32);
  dfree(c.d_res);
  dfree(c.d_iperm);
  dfree(c.d_sortk);
  dfree(c.d_sortv);
  dfree(c.d_flags);
  dfree(c.d_cnt);
  dfree(c.d_stage);
  dfree(c.d_err);
  for (int l = 0; l < kMaxHeight; ++l) {
    Level &L = c.lv[l];
    dfree(L.keys);
    dfree(L.parent);
    dfree(L.child);
    dfree(L.ilist);
    dfree(L.M);
    dfree(L.L);
    dfree(L.grid);
    L.n = 0;
    L.cap = 0;
    L.grid_ready = false;
  }
  c.cap_N = c.cap_leaf = c.cap_sort = c.cap_cnt = c.cap_stage = c.cap_flags = 0;
  c.N = 0;
  c.has_particles = false;
  c.packed32 = false;
  ++c.tree_gen;
}

b200fmm_status upload_charges(Context &c, const double *q, bool on_device) {
  const long long n = c.N;
  if (!on_device) {
    B200_CHECK(grow(c, c.d_stage, c.cap_stage, (size_t)n * (3 + c.R)));
    B200_CUDA(cudaMemcpyAsync(c.d_stage, q, sizeof(double) * n * c.R, cudaMemcpyHostToDevice, c.stream));
    q = c.d_stage;
  }
  gather_charges<<<grid_for(n, 256), 256, 0, c.stream>>>(n, c.R, c.d_perm, q, c.d_q);
  B200_CUDA(cudaGetLastError());
  B200_CUDA(cudaEventRecord(c.ev_stage_free, c.stream));  // the staging buffer's last reader
  c.packed32 = false;
  return B200FMM_OK;
}

// Level storage for n cells (grow-only; M and L are zeroed by execute / reset_expansions).
static b200fmm_status level_storage(Context &c, Level &L, long long n) {
  L.n = n;
  if (L.keys && (size_t)n <= L.cap) return B200FMM_OK;
  size_t cap = L.cap, tmp;
  B200_CHECK(grow(c, L.keys, cap, (size_t)n));
  tmp = L.cap;
  B200_CHECK(grow(c, L.parent, tmp, cap));
  tmp = 8 * L.cap;
  B200_CHECK(grow(c, L.child, tmp, 8 * cap));
  tmp = 189 * L.cap;
  B200_CHECK(grow(c, L.ilist, tmp, 189 * cap));
  tmp = (size_t)c.R * c.nn * L.cap;
  B200_CHECK(grow(c, L.M, tmp, (size_t)c.R * c.nn * cap));
  tmp = (size_t)c.R * c.nn * L.cap;
  B200_CHECK(grow(c, L.L, tmp, (size_t)c.R * c.nn * cap));
  L.cap = cap;
  return B200FMM_OK;
}

b200fmm_status build_tree(Context &c, const double *x, const double *y, const double *z, const double *q,
                          bool on_device) {
  const long long n = c.N;
  const int H = c.H, LL = H - 1;
  cudaStream_t s = c.stream;
  c.tree_launches = 0;
  c.packed32 = false;
  if (!c.h_pinned) B200_CUDA(cudaMallocHost((void **)&c.h_pinned, kPinnedCounts + 4 * sizeof(int)));
  // particle-sized buffers
  size_t cap;
  cap = c.cap_N;
  B200_CHECK(grow(c, c.d_x, cap, (size_t)n));
  cap = c.cap_N;
  B200_CHECK(grow(c, c.d_y, cap, (size_t)n));
  cap = c.cap_N;
  B200_CHECK(grow(c, c.d_z, cap, (size_t)n));
  cap = c.cap_N;
  B200_CHECK(grow(c, c.d_perm, cap, (size_t)n));
  cap = c.cap_N;
  B200_CHECK(grow(c, c.d_iperm, cap, (size_t)n));
  cap = c.cap_N * c.R;
  B200_CHECK(grow(c, c.d_q, cap, (size_t)n * c.R));
  cap = c.cap_N * c.R;
  B200_CHECK(grow(c, c.d_res, cap, (size_t)n * c.R));
  {
    // FP32 P2P copies: target hi [R][N], target lo [N], pair-packed sources [R][N+2][4]
    size_t cp = c.cap_N * (c.R + 1) + 4 * c.R * (c.cap_N + 2);
    B200_CHECK(grow(c, c.d_pq32, cp, (size_t)n * (c.R + 1) + 4 * (size_t)c.R * (n + 2)));
  }
  c.cap_N = std::max(c.cap_N, (size_t)n);
  {
    // the two sort buffers share one capacity: each compares against the old value
    size_t cs = c.cap_sort;
    B200_CHECK(grow(c, c.d_sortk, cs, (size_t)2 * (n + 1)));
    cs = c.cap_sort;
    B200_CHECK(grow(c, c.d_sortv, cs, (size_t)2 * (n + 1)));
    c.cap_sort = std::max(c.cap_sort, (size_t)(2 * (n + 1)));
  }
  const long long nb = (n + RS_TILE - 1) / RS_TILE;
  // tile counts, and the digit totals of the leaf sort
  B200_CHECK(grow(c, c.d_cnt, c.cap_cnt, (size_t)RS8_BINS * (nb + kSortPasses)));
  // block counts: leaves per chunk; cells per block of ML_T leaves and level; records and items per chunk
  B200_CHECK(grow(c, c.d_flags, c.cap_flags,
                  (size_t)std::max<long long>(2 * kMaxBlocks, ((n + ML_T - 1) / ML_T) * kMaxHeight / 2 + 1)));
  if (!c.d_err) B200_CUDA(cudaMalloc(&c.d_err, kErrBytes));
  // inputs on the device
  const double *dx = x, *dy = y, *dz = z, *dq = q;
  if (!on_device) {
    B200_CHECK(grow(c, c.d_stage, c.cap_stage, (size_t)n * (3 + c.R)));
    // The inputs travel on a copy stream of their own: in a time-stepping loop this upload runs while the
    // previous evaluation is still executing on the main stream.  The staging buffer is rewritten only after
    // its last main-stream reader (the previous build's gather, or set_charges' gather) has run.  The keys wait
    // for the coordinates; the charges, first read by the gather after the sort, arrive meanwhile.
    const size_t nb8 = sizeof(double) * (size_t)n, in_bytes = nb8 * (3 + c.R);
    const void *in[4] = {x, y, z, q};
    const bool staged = in_bytes <= kStageIn && may_stage(in, 4, in_bytes, 3 * kStageLocked);
    // the pinned buffer's last copy has ended by now (every call waits for the device), unless one failed half-way
    if (staged) B200_CUDA(cudaStreamSynchronize(c.stream_in));
    B200_CUDA(cudaStreamWaitEvent(c.stream_in, c.ev_stage_free, 0));
    if (staged && ensure_stage(c, in_bytes) == B200FMM_OK) {
      char *h = (char *)c.h_stage;
      std::memcpy(h, x, nb8);
      std::memcpy(h + nb8, y, nb8);
      std::memcpy(h + 2 * nb8, z, nb8);
      std::memcpy(h + 3 * nb8, q, nb8 * c.R);
      B200_CUDA(cudaMemcpyAsync(c.d_stage, h, in_bytes, cudaMemcpyHostToDevice, c.stream_in));
      B200_CUDA(cudaEventRecord(c.ev_in_xyz, c.stream_in));
      B200_CUDA(cudaEventRecord(c.ev_in_q, c.stream_in));
    } else {
      B200_CUDA(cudaMemcpyAsync(c.d_stage, x, sizeof(double) * n, cudaMemcpyHostToDevice, c.stream_in));
      B200_CUDA(cudaMemcpyAsync(c.d_stage + n, y, sizeof(double) * n, cudaMemcpyHostToDevice, c.stream_in));
      B200_CUDA(cudaMemcpyAsync(c.d_stage + 2 * n, z, sizeof(double) * n, cudaMemcpyHostToDevice, c.stream_in));
      B200_CUDA(cudaEventRecord(c.ev_in_xyz, c.stream_in));
      B200_CUDA(cudaMemcpyAsync(c.d_stage + 3 * n, q, sizeof(double) * n * c.R, cudaMemcpyHostToDevice, c.stream_in));
      B200_CUDA(cudaEventRecord(c.ev_in_q, c.stream_in));
    }
    B200_CUDA(cudaStreamWaitEvent(s, c.ev_in_xyz, 0));
    dx = c.d_stage;
    dy = c.d_stage + n;
    dz = c.d_stage + 2 * n;
    dq = c.d_stage + 3 * n;
  }
  unsigned long long *k0 = c.d_sortk, *k1 = c.d_sortk + n;
  int *v0 = c.d_sortv, *v1 = c.d_sortv + n;
  long long *heads = c.d_flags;
  unsigned *totals = (unsigned *)((char *)c.d_err + kErrTotals);
  B200_CUDA(cudaMemsetAsync(c.d_err, 0, kErrBytes, s));
  const double W = c.cfg.box_width;
  const double leaf_w = W / (double)(1 << LL);
  keys_kernel<<<(unsigned)nb, RS_THREADS, 0, s>>>(n, dx, dy, dz, c.cfg.center[0] - W / 2, c.cfg.center[1] - W / 2,
                                                  c.cfg.center[2] - W / 2, W, leaf_w, H, k0, v0, c.d_err, c.d_cnt,
                                                  totals);
  ++c.tree_launches;
  // stable LSD radix sort of (key, original index)
  B200_CHECK(radix_sort(c, k0, k1, v0, v1, n, 3 * LL, totals, true, c.tree_launches));
  if (!on_device) B200_CUDA(cudaStreamWaitEvent(s, c.ev_in_q, 0));
  gather_particles<<<grid_for(n, 256), 256, 0, s>>>(n, c.R, v0, dx, dy, dz, dq, c.d_x, c.d_y, c.d_z, c.d_q, c.d_perm,
                                                 c.d_iperm);
  B200_CUDA(cudaEventRecord(c.ev_stage_free, s));  // the last reader of the staging buffer
  // the cell count of every level at once (and the leaf heads), then the build's one synchronisation
  unsigned long long *counts = (unsigned long long *)(c.d_err + 4);
  const long long chunk = chunk_of(n);
  const unsigned nchunk = grid_for(n, (int)chunk);
  level_counts_kernel<<<nchunk, CB_T, 0, s>>>(n, chunk, k0, LL, heads, counts);
  c.tree_launches += 2;
  B200_CUDA(cudaMemcpyAsync(c.h_pinned, c.d_err, 16 + sizeof(long long) * (LL + 1), cudaMemcpyDeviceToHost, s));
  B200_CUDA(cudaStreamSynchronize(s));
  const long long *ncells = c.h_pinned + 2;  // per level
  if ((int)c.h_pinned[0]) return fail(B200FMM_ERR_DOMAIN, "a particle lies outside the box or has a non-finite coordinate");
  const long long nleaves = ncells[LL];
  Level &leaf = c.lv[LL];
  B200_CHECK(level_storage(c, leaf, nleaves));
  {
    size_t cl = c.cap_leaf;
    B200_CHECK(grow(c, c.d_leaf_start, cl, (size_t)nleaves + 1));
    cl = c.cap_leaf * 27;
    B200_CHECK(grow(c, c.d_leaf_nbr, cl, (size_t)(nleaves + 1) * 27));
    cl = c.cap_leaf;
    B200_CHECK(grow(c, c.d_leaf_rank, cl, (size_t)nleaves + 1));
    cl = c.cap_leaf;
    B200_CHECK(grow(c, c.d_rec_base, cl, (size_t)nleaves + 1));
    cl = c.cap_leaf;
    B200_CHECK(grow(c, c.d_chunk_base, cl, (size_t)nleaves + 1));
    c.cap_leaf = std::max(c.cap_leaf, (size_t)nleaves + 1);
  }
  compact_leaves<<<nchunk, CB_T, 0, s>>>(n, chunk, k0, heads, leaf.keys, c.d_leaf_start);
  ++c.tree_launches;
  // upper levels: storage from the counts taken before the synchronisation, then keys and links of every
  // level from the leaf keys.  Everything that starts from a cleared state is cleared in one launch: child links and
  // cell grids (-1), expansions and results.
  LevelLinks links{};
  ClearList clear;
  for (int l = LL - 1; l >= 0; --l) {
    Level &pa = c.lv[l];
    B200_CHECK(level_storage(c, pa, ncells[l]));
    clear.add(pa.child, sizeof(int) * 8 * (size_t)pa.n, true);  // -1: no child
    links.keys[l] = pa.keys;
    links.parent[l] = pa.parent;
    links.child[l] = pa.child;
  }
  links.parent[LL] = leaf.parent;
  if (c.cfg.precision == B200FMM_MIXED)
    for (int l = 2; l <= LL; ++l) {
      Level &L = c.lv[l];
      const size_t bytes = sizeof(int) << (3 * l);
      if (!L.grid) {
        B200_CUDA(cudaMalloc(&L.grid, bytes));
        ++c.tree_gen;
      }
      clear.add(L.grid, bytes, true);  // -1: empty
    }
  add_state(clear, c);
  B200_CHECK(clear.launch(s));
  ++c.tree_launches;
  if (LL > 0) {
    const int nblk = (int)((nleaves + ML_T - 1) / ML_T);
    unsigned *bcount = (unsigned *)c.d_flags;  // LL * nblk entries; the block counts of the leaves are free now
    if (nblk > 1) {
      ml_count_kernel<<<nblk, ML_T, 0, s>>>(nleaves, leaf.keys, LL, bcount, nblk);
      ++c.tree_launches;
    }
    if (nblk > ML_SUM) {
      ml_scan_kernel<<<LL, ML_T, 0, s>>>(bcount, nblk);
      ++c.tree_launches;
    }
    ml_build_kernel<<<nblk, ML_T, 0, s>>>(nleaves, leaf.keys, LL, bcount, nblk, links);
    ++c.tree_launches;
  }
  // neighbour and interaction lists, dense grids
  leaf_neighbors_kernel<<<grid_for(nleaves * 27, 256), 256, 0, s>>>(nleaves, leaf.keys, H,
                                                                    nleaves == (1LL << (3 * LL)) ? 1 : 0, c.d_leaf_nbr);
  ++c.tree_launches;
  if (LL >= 2) {
    LevelCellsT C{};
    C.l0 = 2;
    C.l1 = LL;
    C.start[2] = 0;
    for (int l = 2; l <= LL; ++l) {
      Level &L = c.lv[l];
      C.keys[l] = L.keys;
      C.ilist[l] = L.ilist;
      C.start[l + 1] = C.start[l] + L.n;
      C.grid[l] = L.grid;
    }
    const long long total = C.start[LL + 1];
    if (total > 0) {
      // the interaction lists feed the FP64 M2L; the tensor-core M2L works from the cell grids, and MIXED
      // builds the lists only when asked for work counts (build_ilists)
      if (c.cfg.precision == B200FMM_FP64) {
        ilist_kernel<<<(unsigned)total, 192, 0, s>>>(C, c.d_itab);
        ++c.tree_launches;
        c.ilist_serial = c.tree_serial;
      } else {
        grid_index_kernel<<<grid_for(total, 256), 256, 0, s>>>(C);
        ++c.tree_launches;
      }
    }
  }
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

// The target shard of execute(): leaves [lo, hi), the Morton range whose particles are those of ranks
// [rank * N / count, (rank + 1) * N / count) of the sorted order rounded to whole leaves, and at every level the
// cells [a, b) that are ancestors of those leaves (contiguous in Morton order).  One thread.
struct ShardLinks {
  const int *parent[kMaxHeight];
  int LL;
};
__global__ void shard_range_kernel(const long long *__restrict__ leaf_start, long long nleaves, long long N, int rank,
                                   int count, const __grid_constant__ ShardLinks S, long long *__restrict__ out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  // the first leaf that starts at or after particle t
  auto first_leaf = [&](long long t) {
    long long a = 0, b = nleaves;
    while (a < b) {
      const long long m = (a + b) >> 1;
      if (leaf_start[m] < t) a = m + 1; else b = m;
    }
    return a;
  };
  const long long lo = rank == 0 ? 0 : first_leaf(N * rank / count);
  const long long hi = rank == count - 1 ? nleaves : first_leaf(N * (rank + 1) / count);
  out[0] = lo;
  out[1] = hi;
  for (int l = 0; l < kMaxHeight; ++l) out[2 + 2 * l] = out[3 + 2 * l] = 0;
  if (hi <= lo) return;
  long long a = lo, b = hi - 1;
  for (int l = S.LL; l >= 0; --l) {
    out[2 + 2 * l] = a;
    out[3 + 2 * l] = b + 1;
    if (l > 0) {
      a = S.parent[l][a];
      b = S.parent[l][b];
    }
  }
}

b200fmm_status shard_ranges(Context &c) {
  const int LL = c.H - 1;
  ShardLinks S{};
  S.LL = LL;
  for (int l = 0; l <= LL; ++l) S.parent[l] = c.lv[l].parent;
  shard_range_kernel<<<1, 32, 0, c.stream>>>(c.d_leaf_start, c.lv[LL].n, c.N, c.shard_rank, c.shard_count, S,
                                             c.d_shard);
  ++c.launches;
  B200_CUDA(cudaGetLastError());
  if (!stream_captured(c)) c.shard_serial = c.tree_serial;
  return B200FMM_OK;
}

// Interaction lists of levels 2..height-1 of the current tree, if not built yet.
b200fmm_status build_ilists(Context &c) {
  const int LL = c.H - 1;
  if (LL < 2 || c.ilist_serial == c.tree_serial) return B200FMM_OK;
  LevelCellsT C{};
  C.l0 = 2;
  C.l1 = LL;
  C.start[2] = 0;
  for (int l = 2; l <= LL; ++l) {
    C.keys[l] = c.lv[l].keys;
    C.ilist[l] = c.lv[l].ilist;
    C.start[l + 1] = C.start[l] + c.lv[l].n;
  }
  const long long total = C.start[LL + 1];
  if (total > 0) ilist_kernel<<<(unsigned)total, 192, 0, c.stream>>>(C, c.d_itab);
  B200_CUDA(cudaGetLastError());
  c.ilist_serial = c.tree_serial;
  return B200FMM_OK;
}

}  // namespace b200

namespace b200 {

// Queues a zero of the expansions of every level and of the results.
b200fmm_status clear_state(Context &c) {
  ClearList clear;
  add_state(clear, c);
  return clear.launch(c.stream);
}

static NearArgs near_args(const Context &c, int whole, int item) {
  NearArgs a{};
  a.LL = c.H - 1;
  a.nl = c.lv[a.LL].n;
  a.chunk = chunk_of(a.nl);
  a.whole = whole;
  a.item = item;
  a.leaf_start = c.d_leaf_start;
  a.rank_of = c.d_leaf_rank;
  a.rec_base = c.d_rec_base;
  a.chunk_base = c.d_chunk_base;
  a.recs = c.d_flags;
  a.items = c.d_flags + kMaxBlocks;
  return a;
}

b200fmm_status leaf_column_order(Context &c) {
  NearArgs a = near_args(c, c.p2p_whole, c.p2p_item);
  cudaStream_t s = c.stream;
  if (a.nl != (1LL << (3 * a.LL))) {
    // the particle sort's buffers are free after the tree build and hold 2(N+1) >= 2 nleaves entries
    unsigned long long *k0 = c.d_sortk, *k1 = c.d_sortk + a.nl;
    int *v0 = c.d_sortv, *v1 = c.d_sortv + a.nl;
    const long long nb = (c.N + RS_TILE - 1) / RS_TILE;
    unsigned *totals = c.d_cnt + (size_t)RS8_BINS * nb;
    B200_CUDA(cudaMemsetAsync(totals, 0, sizeof(unsigned) * RS8_BINS * kSortPasses, s));
    leaf_column_keys<<<grid_for(a.nl, 256), 256, 0, s>>>(a.nl, c.lv[a.LL].keys, a.LL, k0, v0);
    ++c.launches;
    B200_CHECK(radix_sort(c, k0, k1, v0, v1, a.nl, 2 * a.LL, totals, false, c.launches));
    a.order = v0;
  }
  const unsigned blocks = grid_for(a.nl, (int)a.chunk);
  near_sums_kernel<true><<<blocks, CB_T, 0, s>>>(a);
  near_bases_kernel<true><<<blocks, CB_T, 0, s>>>(a);
  c.launches += 2;
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

b200fmm_status leaf_items(Context &c, int whole, int item) {
  const NearArgs a = near_args(c, whole, item);
  const unsigned blocks = grid_for(a.nl, (int)a.chunk);
  near_sums_kernel<false><<<blocks, CB_T, 0, c.stream>>>(a);
  near_bases_kernel<false><<<blocks, CB_T, 0, c.stream>>>(a);
  c.launches += 2;
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

}  // namespace b200
