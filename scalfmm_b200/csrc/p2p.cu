// Near field P2P for the Laplace 1/r kernel over each leaf and its <=26 neighbour leaves.
//
// Pair math (FP2PR::MutualParticles / NonMutualParticles, Src/Kernels/P2P/FP2PR.hpp:14-69):
//   phi_t += q_s / r,   F_t += -q_t q_s (x_t - x_s) / r^3.
// The reference evaluates each unordered pair once (mutual half shell, FChebSymKernel.hpp:468-478);
// the ordered pairs summed here per target are the same set.
//
//  * FP64 (parity form): one CTA per 32 targets of a leaf, the sources of the leaf and its neighbours staged through
//    shared memory, rsqrt() in FP64.
//  * FP32 (mixed form), two source particles against two targets per lane and step with Blackwell's packed FP32x2
//    instructions (add/mul/fma.f32x2): positions relative to the box corner as a float pair (hi, lo), so that per pair
//    dx = (t_hi - s_hi) + (t_lo - s_lo) with the first difference exact for nearby particles (Sterbenz),
//    which keeps the close pairs -- the ones that dominate the forces -- accurate to a few ulp.  One warp per
//    leaf or piece of a larger one; the neighbour leaves are walked as contiguous runs of records (one per neighbour
//    column) copied into shared memory by the bulk-copy engine (cp.async.bulk + mbarrier, 3-deep ring); rsqrt on the
//    SFU; per-target compensated (two-sum) accumulation of partial sums; the result is added
//    in FP64 to the far field.
#include "common.cuh"

#include <mutex>

namespace b200 {

namespace {

constexpr int P2P64_WARPS = 4, P2P64_THREADS = 32 * P2P64_WARPS;
constexpr int P2P64_TGT = 32;  // targets per work item

// The pairs of NR right-hand sides of one source with one target; SELF: the source may be the target itself.
template <int NR, bool SELF>
__device__ __forceinline__ void p2p64_pair(const double4 &s, bool self, const double *__restrict__ sq, int sq_stride,
                                           double tx, double ty, double tz, double (&pv)[NR], double (&gx)[NR],
                                           double (&gy)[NR], double (&gz)[NR]) {
  const double dx = tx - s.x, dy = ty - s.y, dz = tz - s.z;
  double inv = rsqrt(dx * dx + dy * dy + dz * dz);
  if (SELF && self) inv = 0.0;
  const double inv2 = inv * inv;
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    double p = inv * (NR == 1 ? s.w : sq[r * sq_stride]);
    if (SELF && self) p = 0.0;  // the target is left out, whatever its charge (0 times an infinite one is no number)
    const double f = p * inv2;
    pv[r] += p;
    gx[r] += dx * f;
    gy[r] += dy * f;
    gz[r] += dz * f;
  }
}

// FP64.  One CTA per work item (up to 32 targets of a leaf, c.d_chunk_base); the sources of the leaf and its
// neighbours are one sequence, staged 128 at a time, and each warp takes 32 of them against all the item's targets
// (lane = target; 16 or 8 targets are replicated over 2 or 4 lane groups with every 2nd or 4th source).  The warps'
// sums are added at the end in a fixed order.  What bounds it is the FP64 pipe: per pair 3 differences, 3 for r^2,
// the reciprocal square root (about 9 instructions of rsqrt(); the division and square root of sqrt(1 / r^2) that
// the reference writes take about 22) and 7 for the sums: 1M uniform points in leaves of 30: 3.85 -> 1.53 ms (0.51
// Tpairs/s), 500,009 on a surface 2.05 -> 0.82 ms; 60,000 clustered points, whose dense leaves one CTA each carried
// before, 9.1 -> 0.39 ms.  Against sums in extended precision the error is 0.3-0.6 of the earlier kernel's (shorter
// chains of additions).  shard (optional): [first leaf, end leaf) of the targets.
template <int NR>
__global__ void __launch_bounds__(P2P64_THREADS) p2p_fp64_kernel(
    int R, long long N, long long nleaves, const long long *__restrict__ leaf_start, const int *__restrict__ nbr,
    const long long *__restrict__ chunk_base, int variant, const double *__restrict__ x, const double *__restrict__ y,
    const double *__restrict__ z, const double *__restrict__ q, double4 *__restrict__ res,
    const long long *__restrict__ shard) {
  __shared__ __align__(32) double4 src[P2P64_THREADS];              // x, y, z, q (of the only right-hand side)
  __shared__ double srcq[NR > 1 ? NR : 1][NR > 1 ? P2P64_THREADS : 1];
  __shared__ double red[P2P64_WARPS - 1][4][32];
  __shared__ long long s_first[27];   // first particle of each neighbour present
  __shared__ int s_off[28], s_n, s_self;  // where its sources begin in the sequence; which one is the leaf itself
  const long long leaf_lo = shard ? shard[0] : 0, leaf_hi = shard ? shard[1] : nleaves;
  const long long item = chunk_base[leaf_lo] + blockIdx.x;
  if (item >= chunk_base[leaf_hi]) return;
  long long leaf = leaf_lo, hi = leaf_hi - 1;  // the last leaf whose first item is <= item
  while (leaf < hi) {
    const long long mid = (leaf + hi + 1) >> 1;
    if (chunk_base[mid] <= item)
      leaf = mid;
    else
      hi = mid - 1;
  }
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  if (w == 0) {
    int nb = lane < 27 ? nbr[leaf * 27 + lane] : -1;
    if (variant == 1 && lane == 13) nb = -1;
    const long long a = nb >= 0 ? leaf_start[nb] : 0;
    const int cnt = nb >= 0 ? (int)(leaf_start[nb + 1] - a) : 0;
    int e = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, e, o);
      if (lane >= o) e += v;
    }
    const unsigned m = __ballot_sync(0xffffffffu, cnt > 0);
    const int k = __popc(m & ((1u << lane) - 1u));
    if (cnt > 0) {
      s_first[k] = a;
      s_off[k] = e - cnt;
    }
    if (lane == 13) s_self = cnt > 0 ? k : -1;
    if (lane == 31) {
      s_n = __popc(m);
      s_off[__popc(m)] = e;
    }
  }
  __syncthreads();
  const int nn = s_n, total = s_off[nn], self = s_self;
  const long long t0 = leaf_start[leaf] + P2P64_TGT * (item - chunk_base[leaf]);
  const int m = (int)min((long long)P2P64_TGT, leaf_start[leaf + 1] - t0);
  const int T = m <= 8 ? 8 : (m <= 16 ? 16 : 32), G = 32 / T;
  const int tl = lane & (T - 1), g = lane / T;
  const bool active = tl < m;
  const double tx = active ? x[t0 + tl] : 0, ty = active ? y[t0 + tl] : 0, tz = active ? z[t0 + tl] : 0;
  // the sequence position of the target itself
  const int own = self >= 0 ? s_off[self] + (int)(t0 - s_first[self]) + tl : -1;
  const int own0 = self >= 0 ? s_off[self] : -1, own1 = self >= 0 ? s_off[self + 1] : -1;
  for (int r0 = 0; r0 < R; r0 += NR) {
    double pv[NR], gx[NR], gy[NR], gz[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) pv[r] = gx[r] = gy[r] = gz[r] = 0.0;
    for (int sb = 0; sb < total; sb += P2P64_THREADS) {
      __syncthreads();
      const int k = sb + t;
      if (k < total) {
        int a = 0, b = nn - 1;  // the last neighbour that begins at or before k
        while (a < b) {
          const int mid = (a + b + 1) >> 1;
          if (s_off[mid] <= k)
            a = mid;
          else
            b = mid - 1;
        }
        const long long j = s_first[a] + (k - s_off[a]);
        src[t] = make_double4(x[j], y[j], z[j], NR == 1 ? q[(long long)r0 * N + j] : 0.0);
        if (NR > 1)
#pragma unroll
          for (int r = 0; r < NR; ++r) srcq[r][t] = r0 + r < R ? q[(long long)(r0 + r) * N + j] : 0.0;
      }
      __syncthreads();
      const int i1 = min(32 * w + 32, total - sb);
      if (sb + i1 > own0 && sb + 32 * w < own1) {
        for (int i = 32 * w + g; i < i1; i += G)
          p2p64_pair<NR, true>(src[i], sb + i == own, &srcq[0][i], P2P64_THREADS, tx, ty, tz, pv, gx, gy, gz);
      } else {
#pragma unroll 4
        for (int i = 32 * w + g; i < i1; i += G)
          p2p64_pair<NR, false>(src[i], false, &srcq[0][i], P2P64_THREADS, tx, ty, tz, pv, gx, gy, gz);
      }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      if (r0 + r >= R) break;
      double v[4] = {pv[r], gx[r], gy[r], gz[r]};
#pragma unroll
      for (int c = 0; c < 4; ++c)
        for (int o = T; o < 32; o <<= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
      __syncthreads();
      if (w > 0)
#pragma unroll
        for (int c = 0; c < 4; ++c) red[w - 1][c][lane] = v[c];
      __syncthreads();
      if (w == 0 && active && g == 0) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int u = 0; u < P2P64_WARPS - 1; ++u) v[c] += red[u][c][lane];
        const long long j = (long long)(r0 + r) * N + t0 + tl;
        const double nq = -q[j];
        add_result(res + j, v[0], nq * v[1], nq * v[2], nq * v[3]);
      }
    }
  }
}

// ---- FP32 compensated ------------------------------------------------------------------------------
//
// Layout of the FP32 copies (one buffer, d_pq32):
//   tgt_hi[R][N] float4 (x_hi, y_hi, z_hi, q) and tgt_lo[N] float4 (x_lo, y_lo, z_lo, 0): the position of every
//     particle relative to the box corner as a float pair (hi = fl(x - x0), lo = fl(x - x0 - hi)), read by the
//     lane that owns the particle as a target;
//   src[R][N+2][4] float4: the same particles as sources, two per 64-byte record and pre-negated so that
//     packed FP32x2 instructions consume them directly: (-x0,-x1,-y0,-y1) (-z0,-z1,q0,q1) (-lx0,-lx1,-ly0,-ly1)
//     (-lz0,-lz1,0,0).  A leaf with an odd count is padded with a zero-charge particle far away.
// Record order: the leaves in column order (x, y, then z; rank_of[leaf], first record rec_base[rank]), so that
// the up to three z-neighbours of each of the 9 neighbour columns of a target leaf are one contiguous run of
// records.  Without rank_of/rec_base (the allocation-free entry point) the leaves stay in Morton order with
// leaf L's records starting at (leaf_start[L] + L) / 2 (gap records padded); only Morton-adjacent z-neighbours
// then share a run.
//
// Because the coordinates are relative to the box corner (>= 0) and hi carries 24 bits, for close pairs
// t_hi - s_hi is exact (Sterbenz), and dx = (t_hi - s_hi) + (t_lo - s_lo) is accurate to about one ulp of dx:
// the close pairs, which dominate the forces, keep full FP32 relative accuracy.
constexpr double P2P32_PAD = 1.0e15;

__host__ __device__ inline long long p2p_pairs_capacity(long long N) { return N + 2; }

// first source record of the leaf at position rank of the record order
__device__ __forceinline__ long long rec_begin(const long long *__restrict__ rec_base,
                                               const long long *__restrict__ leaf_start, long long rank) {
  return rec_base ? rec_base[rank] : (leaf_start[rank] + rank) >> 1;
}

__global__ void pack_records32(long long N, int R, const long long *__restrict__ leaf_start,
                               const int *__restrict__ rank_of, const long long *__restrict__ rec_base,
                               const double *__restrict__ x, const double *__restrict__ y,
                               const double *__restrict__ z, const double *__restrict__ q, double x0, double y0,
                               double z0, float4 *__restrict__ hi, float4 *__restrict__ lo,
                               float4 *__restrict__ src) {
  const long long leaf = blockIdx.x;
  const long long s0 = leaf_start[leaf], s1 = leaf_start[leaf + 1];
  const long long rank = rank_of ? rank_of[leaf] : leaf;
  const long long b0 = rec_begin(rec_base, leaf_start, rank), b1 = rec_begin(rec_base, leaf_start, rank + 1);
  for (long long i = s0 + threadIdx.x; i < s1; i += blockDim.x) {
    const double lx = x[i] - x0, ly = y[i] - y0, lz = z[i] - z0;
    const float hx = (float)lx, hy = (float)ly, hz = (float)lz;
    lo[i] = make_float4((float)(lx - (double)hx), (float)(ly - (double)hy), (float)(lz - (double)hz), 0.f);
    for (int r = 0; r < R; ++r) hi[(long long)r * N + i] = make_float4(hx, hy, hz, (float)q[(long long)r * N + i]);
  }
  const long long P = p2p_pairs_capacity(N);
  for (long long pp = threadIdx.x; pp < b1 - b0; pp += blockDim.x) {
    float h[2][3], l[2][3];
    bool real[2];
    for (int u = 0; u < 2; ++u) {
      const long long j = s0 + 2 * pp + u;
      real[u] = j < s1;
      const double d[3] = {real[u] ? x[j] - x0 : P2P32_PAD, real[u] ? y[j] - y0 : P2P32_PAD,
                           real[u] ? z[j] - z0 : P2P32_PAD};
      for (int a = 0; a < 3; ++a) {
        h[u][a] = (float)d[a];
        l[u][a] = (float)(d[a] - (double)h[u][a]);
      }
    }
    for (int r = 0; r < R; ++r) {
      const long long j0 = s0 + 2 * pp;
      const float q0 = real[0] ? (float)q[(long long)r * N + j0] : 0.f;
      const float q1 = real[1] ? (float)q[(long long)r * N + j0 + 1] : 0.f;
      float4 *rec = src + ((long long)r * P + b0 + pp) * 4;
      rec[0] = make_float4(-h[0][0], -h[1][0], -h[0][1], -h[1][1]);
      rec[1] = make_float4(-h[0][2], -h[1][2], q0, q1);
      rec[2] = make_float4(-l[0][0], -l[1][0], -l[0][1], -l[1][1]);
      rec[3] = make_float4(-l[0][2], -l[1][2], 0.f, 0.f);
    }
  }
}

// Compensated (two-sum) accumulation of two values at once, packed.
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ void two_sum2(float2 &hi, float2 &lo, float2 v) {
  const float2 s = __fadd2_rn(hi, v);
  const float2 bp = __fadd2_rn(s, neg2(hi));
  const float2 err = __fadd2_rn(__fadd2_rn(hi, neg2(__fadd2_rn(s, neg2(bp)))), __fadd2_rn(v, neg2(bp)));
  hi = s;
  lo = __fadd2_rn(lo, err);
}

constexpr int P2P32_WARPS = 2;   // work items per CTA (one warp each): few, so that a long one holds little else up
constexpr int P2P32_STAGE = 56;  // source records (112 particles) per bulk-copy stage
constexpr int P2P32_FLUSH = 24;  // records per lane whose sums enter the compensated sums together
constexpr int P2P32_TGT = 2;     // targets per lane
constexpr int P2P32_NBUF = 3;    // stages in flight per warp

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// Bounded wait on an mbarrier phase; returns false when the iteration budget runs out.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned phase) {
  for (int it = 0; it < (1 << 22); ++it) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(phase)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// The same wait taken by a whole warp: every lane polls, and the warp agrees on the outcome, so that either all
// lanes go on or all give up (a lane that left alone would break the full-mask shuffles that follow).
__device__ __forceinline__ bool mbar_wait_warp(unsigned long long *bar, unsigned phase) {
  return __all_sync(0xffffffffu, mbar_wait(bar, phase));
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}

// 1/sqrt(x) on the SFU with subnormal inputs flushed to zero (PTX rsqrt.approx.ftz.f32).  rsqrtf, which also
// serves subnormal inputs, made the near field about 8 % slower with bit-identical results on the bench tree;
// r^2 here is subnormal only for particles closer than ~1e-19 box widths, which the flush treats like
// coincident particles.
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// A lane's target: its position, each coordinate twice for the packed instructions.
struct Target32 {
  float2 hx, hy, hz, lx, ly, lz;
};
struct Sums32 {
  float2 pv, ax, ay, az;
};

// One record (two sources) against each of the lane's targets: packed FP32x2 difference, r^2, rsqrt on the SFU.
template <bool SELF>
__device__ __forceinline__ void p2p_record(const float4 *__restrict__ s, int k, const int (&self_rel)[P2P32_TGT],
                                           const Target32 (&t)[P2P32_TGT], Sums32 (&acc)[P2P32_TGT]) {
  const float4 A = s[4 * k], B = s[4 * k + 1], C = s[4 * k + 2], D = s[4 * k + 3];
#pragma unroll
  for (int u = 0; u < P2P32_TGT; ++u) {
    const float2 dx =
        __fadd2_rn(__fadd2_rn(t[u].hx, make_float2(A.x, A.y)), __fadd2_rn(t[u].lx, make_float2(C.x, C.y)));
    const float2 dy =
        __fadd2_rn(__fadd2_rn(t[u].hy, make_float2(A.z, A.w)), __fadd2_rn(t[u].ly, make_float2(C.z, C.w)));
    const float2 dz =
        __fadd2_rn(__fadd2_rn(t[u].hz, make_float2(B.x, B.y)), __fadd2_rn(t[u].lz, make_float2(D.x, D.y)));
    float2 r2 = __fmul2_rn(dx, dx);
    r2 = __ffma2_rn(dy, dy, r2);
    r2 = __ffma2_rn(dz, dz, r2);
    float2 inv;
    if (SELF) {
      inv = make_float2(2 * k == self_rel[u] ? 0.f : rsqrt_ftz(r2.x), 2 * k + 1 == self_rel[u] ? 0.f : rsqrt_ftz(r2.y));
    } else {
      inv = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
    }
    const float2 qi = __fmul2_rn(make_float2(B.z, B.w), inv);
    const float2 qi3 = __fmul2_rn(qi, __fmul2_rn(inv, inv));
    acc[u].pv = __fadd2_rn(acc[u].pv, qi);
    acc[u].ax = __ffma2_rn(dx, qi3, acc[u].ax);
    acc[u].ay = __ffma2_rn(dy, qi3, acc[u].ay);
    acc[u].az = __ffma2_rn(dz, qi3, acc[u].az);
  }
}

// One warp per work item.  A lane carries two targets, so that each record that it reads from shared memory serves
// four pairs.  What bounds the kernel is the FP32 pipe (19 packed instructions per record and target, 1.96 Tpairs/s at
// most) and the instructions around the pair loop: with one target per lane, stages of 32 records and a compensated
// sum per stage, about half of the issued instructions were not the pairs'.  Two targets alone changed nothing; with
// stages of 56 records (the three z-neighbours of a leaf of 30 are one stage), packed compensated sums of both targets
// after every 24 records of a lane (chains no longer than before: the error is 0.9-1.0 of the earlier kernel's) and
// 128 registers: 1M uniform 0.885 -> 0.81 ms, 2M on a surface 6.13 -> 5.68 ms, 200k in leaves of 49 0.347 -> 0.285
// ms.  (Five CTAs of four warps at 100 registers and stages of 44: 0.95, 5.98 and 0.31 ms.)  Sums after every 16
// records cost 4 % more, after every 64 give 2 % but a larger error.
// The targets are taken 64, 32, 16 or 8 at a time (p2p_chunk); 32 (16, 8) targets occupy 16 (8, 4) lanes and are
// replicated over 2 (4, 8) lane groups, each group walking every 2nd (4th, 8th) source record, and the groups' sums
// are combined by shuffles at the end, so that small and ragged leaves keep the lanes busy.
// The sources are walked as runs of contiguous records (one per neighbour column and z-adjacent group),
// each split into stages of <= P2P32_STAGE records copied by one bulk copy into a ring of P2P32_NBUF buffers,
// issued P2P32_NBUF - 1 stages ahead of the math.  After every P2P32_FLUSH records of a lane, and at the end of a
// stage, the partial sums enter the targets' (hi, lo) accumulators by a two-sum.
// With chunk_base, warp (CTA x, warp w) takes the work item blockIdx.x * P2P32_WARPS + w: a leaf of at most
// `whole` targets, or `isize` targets of a larger one (a dense leaf spreads over many warps; items past the count
// leave at once).  Without it (the allocation-free entry point) a warp takes a whole leaf.
__device__ __forceinline__ bool p2p_item(long long item, long long nleaves, const long long *__restrict__ leaf_start,
                                         const long long *__restrict__ chunk_base, int whole, int isize,
                                         long long &leaf, long long &c0, long long &c1) {
  if (!chunk_base) {
    if (item >= nleaves) return false;
    leaf = item;
    c0 = leaf_start[leaf];
    c1 = leaf_start[leaf + 1];
    return true;
  }
  if (item >= chunk_base[nleaves]) return false;
  long long lo = 0, hi = nleaves - 1;  // the last leaf whose first item is <= item
  while (lo < hi) {
    const long long mid = (lo + hi + 1) >> 1;
    if (chunk_base[mid] <= item)
      lo = mid;
    else
      hi = mid - 1;
  }
  leaf = lo;
  const long long s0 = leaf_start[leaf], s1 = leaf_start[leaf + 1];
  if (s1 - s0 <= whole) {
    c0 = s0;
    c1 = s1;
  } else {
    c0 = s0 + (long long)isize * (item - chunk_base[leaf]);
    c1 = min(c0 + isize, s1);
  }
  return true;
}

// Targets of the next pass over the sources, of `left` that remain: a power of two with at least half of the 2 x 32
// slots in use, and 33..48 as 32 and the rest.
__device__ __forceinline__ int p2p_chunk(long long left) { return left > 48 ? 64 : left > 16 ? 32 : left > 8 ? 16 : 8; }

// Where the results go: the handle's records, or a caller's four arrays (the allocation-free entry point).
struct OutRecords {
  double4 *res;
  __device__ __forceinline__ void add(long long j, double p, double x, double y, double z) const {
    add_result(res + j, p, x, y, z);
  }
};
struct OutArrays {
  double *phi, *fx, *fy, *fz;
  __device__ __forceinline__ void add(long long j, double p, double x, double y, double z) const {
    phi[j] += p;
    fx[j] += x;
    fy[j] += y;
    fz[j] += z;
  }
};

template <class Out>
__global__ void __launch_bounds__(P2P32_WARPS * 32, 8) p2p_fp32_kernel(
    int R, long long N, long long nleaves, const long long *__restrict__ leaf_start, const int *__restrict__ nbr,
    int variant, const int *__restrict__ rank_of, const long long *__restrict__ rec_base,
    const long long *__restrict__ chunk_base, int whole, int isize, const long long *__restrict__ shard,
    const float4 *__restrict__ pq,
    const float4 *__restrict__ plo, const float4 *__restrict__ src, const Out out, int *__restrict__ status) {
  __shared__ __align__(128) float4 buf[P2P32_WARPS][P2P32_NBUF][4 * P2P32_STAGE];
  __shared__ __align__(8) unsigned long long bar[P2P32_WARPS][P2P32_NBUF];
  __shared__ long long rbase[P2P32_WARPS][27];
  __shared__ int rcount[P2P32_WARPS][27];
  __shared__ unsigned char rself[P2P32_WARPS][27];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    for (int b = 0; b < P2P32_NBUF; ++b) mbar_init(&bar[w][b], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  // the work items of the targets' leaves: all, or the shard's [shard[0], shard[1])
  const long long leaf_lo = shard ? shard[0] : 0, leaf_hi = shard ? shard[1] : nleaves;
  const long long item0 = chunk_base ? chunk_base[leaf_lo] : leaf_lo;
  const long long item1 = chunk_base ? chunk_base[leaf_hi] : leaf_hi;
  const long long item = item0 + (long long)blockIdx.x * P2P32_WARPS + w;
  long long leaf, c0, c1;
  if (item >= item1 || !p2p_item(item, nleaves, leaf_start, chunk_base, whole, isize, leaf, c0, c1)) return;
  const long long P = p2p_pairs_capacity(N);
  const long long t0 = leaf_start[leaf];
  const int my_rank = rank_of ? rank_of[leaf] : (int)leaf;
  const long long self_rec = rec_begin(rec_base, leaf_start, my_rank);
  // the runs of this leaf: lane e < 27 looks at neighbour position e = ((dx+1)*3 + dy+1)*3 + dz+1
  int nr = 0;
  {
    const int e = lane < 27 ? lane : 26;
    int nb = lane < 27 ? nbr[leaf * 27 + e] : -1;
    if (variant == 1 && e == 13) nb = -1;
    const int rk = nb >= 0 ? (rank_of ? rank_of[nb] : nb) : -1;
    const int dz = e % 3;
    const int rk_prev = __shfl_up_sync(0xffffffffu, rk, 1);
    const int rk_next = __shfl_down_sync(0xffffffffu, rk, 1);
    const int rk_next2 = __shfl_down_sync(0xffffffffu, rk, 2);
    const bool start = lane < 27 && rk >= 0 && !(dz > 0 && rk_prev >= 0 && rk_prev + 1 == rk);
    int last = rk;
    if (dz < 2 && rk_next >= 0 && rk_next == last + 1) {
      last = rk_next;
      if (dz == 0 && rk_next2 >= 0 && rk_next2 == last + 1) last = rk_next2;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, start);
    if (start) {
      const int k = __popc(mask & ((1u << lane) - 1u));
      const long long b0 = rec_begin(rec_base, leaf_start, rk), b1 = rec_begin(rec_base, leaf_start, last + 1);
      rbase[w][k] = b0;
      rcount[w][k] = (int)(b1 - b0);
      rself[w][k] = (variant == 0 && e / 3 == 4 && rk <= my_rank && my_rank <= last) ? 1 : 0;
    }
    nr = __popc(mask);
    __syncwarp();
  }
  unsigned phase_bits = 0;  // one parity bit per buffer
  for (int r = 0; r < R; ++r) {
    const float4 *pr = pq + (long long)r * N;
    const float4 *sr = src + (long long)r * P * 4;
    for (long long tb = c0; tb < c1;) {
      const int chunk = p2p_chunk(c1 - tb);
      const int m = (int)min((long long)chunk, c1 - tb);
      const int T = chunk / P2P32_TGT;  // lanes per group
      const int G = 32 / T;             // lane groups, each on every G-th record
      const int tl = lane & (T - 1), g = lane / T;
      Target32 tg[P2P32_TGT];
      float tq[P2P32_TGT];
      float2 hi[4], lo[4];  // compensated potential and force sums of both targets (.x, .y)
#pragma unroll
      for (int c = 0; c < 4; ++c) hi[c] = lo[c] = make_float2(0.f, 0.f);
#pragma unroll
      for (int u = 0; u < P2P32_TGT; ++u) {
        const bool on = tl + u * T < m;
        const float4 me = on ? pr[tb + tl + u * T] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 mel = on ? plo[tb + tl + u * T] : make_float4(0.f, 0.f, 0.f, 0.f);
        tg[u] = {make_float2(me.x, me.x),   make_float2(me.y, me.y),   make_float2(me.z, me.z),
                 make_float2(mel.x, mel.x), make_float2(mel.y, mel.y), make_float2(mel.z, mel.z)};
        tq[u] = me.w;
      }
      const long long self_slot = 2 * self_rec + (tb + tl - t0);  // target 0's own slot in the record numbering
      // stage sequence: (run e, first record p, record count n); issue up to NBUF-1 stages ahead
      int ie = 0, ip = 0;  // next stage to issue
      int ce = 0, cp = 0;  // stage being computed
      int issued = 0, done = 0;
      auto next_stage = [&](int &e, int &p0, int &n) -> bool {
        while (e < nr && p0 >= rcount[w][e]) {
          ++e;
          p0 = 0;
        }
        if (e >= nr) return false;
        n = min(P2P32_STAGE, rcount[w][e] - p0);
        return true;
      };
      auto issue = [&]() {
        int n;
        if (!next_stage(ie, ip, n)) return false;
        const int b = issued % P2P32_NBUF;
        if (lane == 0) {
          mbar_expect_tx(&bar[w][b], n * 64);
          bulk_g2s(&buf[w][b][0], sr + (rbase[w][ie] + ip) * 4, n * 64, &bar[w][b]);
        }
        ip += n;
        ++issued;
        return true;
      };
      for (int k = 0; k < P2P32_NBUF - 1; ++k)
        if (!issue()) break;
      while (done < issued) {
        int cn;
        next_stage(ce, cp, cn);
        const int b = done % P2P32_NBUF;
        if (!mbar_wait_warp(&bar[w][b], (phase_bits >> b) & 1u)) {
          // give up: flag it, and let the copies still in flight land (bounded) before the CTA leaves
          if (lane == 0) {
            atomicExch(status, 1);
            for (int k = done; k < issued; ++k) {
              const int bk = k % P2P32_NBUF;
              mbar_wait(&bar[w][bk], (phase_bits >> bk) & 1u);
            }
          }
          __syncwarp();
          return;
        }
        phase_bits ^= 1u << b;
        const float4 *s = buf[w][b];
        const bool own = rself[w][ce];
        int self_rel[P2P32_TGT];
#pragma unroll
        for (int u = 0; u < P2P32_TGT; ++u)  // the target's slot in this stage
          self_rel[u] = (int)(self_slot - 2 * (rbase[w][ce] + cp)) + u * T;
        for (int k0 = g; k0 < cn; k0 += P2P32_FLUSH * G) {
          const int k1 = min(cn, k0 + P2P32_FLUSH * G);
          Sums32 acc[P2P32_TGT];
#pragma unroll
          for (int u = 0; u < P2P32_TGT; ++u) acc[u].pv = acc[u].ax = acc[u].ay = acc[u].az = make_float2(0.f, 0.f);
          if (own) {
#pragma unroll 2
            for (int k = k0; k < k1; k += G) p2p_record<true>(s, k, self_rel, tg, acc);
          } else {
#pragma unroll 2
            for (int k = k0; k < k1; k += G) p2p_record<false>(s, k, self_rel, tg, acc);
          }
          two_sum2(hi[0], lo[0], make_float2(acc[0].pv.x + acc[0].pv.y, acc[1].pv.x + acc[1].pv.y));
          two_sum2(hi[1], lo[1], make_float2(acc[0].ax.x + acc[0].ax.y, acc[1].ax.x + acc[1].ax.y));
          two_sum2(hi[2], lo[2], make_float2(acc[0].ay.x + acc[0].ay.y, acc[1].ay.x + acc[1].ay.y));
          two_sum2(hi[3], lo[3], make_float2(acc[0].az.x + acc[0].az.y, acc[1].az.x + acc[1].az.y));
        }
        cp += cn;
        ++done;
        __syncwarp();  // every lane is done with buffer b before it is refilled
        issue();
      }
      // combine the lane groups that shared this chunk's targets
#pragma unroll
      for (int c = 0; c < 4; ++c)
        for (int off = T; off < 32; off <<= 1) {
          const float2 oh = make_float2(__shfl_xor_sync(0xffffffffu, hi[c].x, off),
                                        __shfl_xor_sync(0xffffffffu, hi[c].y, off));
          const float2 ol = make_float2(__shfl_xor_sync(0xffffffffu, lo[c].x, off),
                                        __shfl_xor_sync(0xffffffffu, lo[c].y, off));
          two_sum2(hi[c], lo[c], oh);
          lo[c] = __fadd2_rn(lo[c], ol);
        }
      if (g == 0) {
#pragma unroll
        for (int u = 0; u < P2P32_TGT; ++u) {
          if (tl + u * T >= m) continue;
          const long long j = (long long)r * N + tb + tl + u * T;
          const double nq = -(double)tq[u];
          double v[4];
#pragma unroll
          for (int c = 0; c < 4; ++c)
            v[c] = u == 0 ? (double)hi[c].x + (double)lo[c].x : (double)hi[c].y + (double)lo[c].y;
          out.add(j, v[0], nq * v[1], nq * v[2], nq * v[3]);
        }
      }
      tb += m;
    }
  }
}

// ---- several right-hand sides ------------------------------------------------------------------------
//
// With nrhs > 1 the charge vectors share the positions, so the geometry of a pair (differences, r^2, rsqrt,
// 1/r^3) is formed once for MR_G right-hand sides at a time, as the reference's multi-RHS near field forms it
// once for all NVALS vectors (FP2P::FullMutualMultiRhs, Src/Kernels/P2P/FP2PMultiRhs.hpp:10-189).  Layout:
//   tgt_hi[N] float4 (x_hi, y_hi, z_hi, 0), tgt_lo[N] float4 (x_lo, y_lo, z_lo, 0), tgt_q[R][N] float;
//   src[G][N+2][5] float4 for each group of MR_G right-hand sides, two sources per 80-byte record:
//     (-x0,-x1,-y0,-y1) (-z0,-z1,-lz0,-lz1) (-lx0,-lx1,-ly0,-ly1) (q0,q1 of rhs 0; q0,q1 of rhs 1) (rhs 2; rhs 3),
//   charges of right-hand sides past R are zero.  Record order and runs are those of the single-RHS kernel.
constexpr int MR_G = 4;
constexpr int MR_REC = 5;  // float4 per record
constexpr int MR_STAGE = 48;  // records per bulk-copy stage
constexpr int MR_FLUSH = 24;  // records of a stage whose sums enter the compensated sums together

__global__ void pack_records32_mrhs(long long N, int R, const long long *__restrict__ leaf_start,
                                    const int *__restrict__ rank_of, const long long *__restrict__ rec_base,
                                    const double *__restrict__ x, const double *__restrict__ y,
                                    const double *__restrict__ z, const double *__restrict__ q, double x0, double y0,
                                    double z0, float4 *__restrict__ hi, float4 *__restrict__ lo, float *__restrict__ qt,
                                    float4 *__restrict__ src) {
  const long long leaf = blockIdx.x;
  const long long s0 = leaf_start[leaf], s1 = leaf_start[leaf + 1];
  const long long rank = rank_of ? rank_of[leaf] : leaf;
  const long long b0 = rec_begin(rec_base, leaf_start, rank), b1 = rec_begin(rec_base, leaf_start, rank + 1);
  for (long long i = s0 + threadIdx.x; i < s1; i += blockDim.x) {
    const double lx = x[i] - x0, ly = y[i] - y0, lz = z[i] - z0;
    const float hx = (float)lx, hy = (float)ly, hz = (float)lz;
    hi[i] = make_float4(hx, hy, hz, 0.f);
    lo[i] = make_float4((float)(lx - (double)hx), (float)(ly - (double)hy), (float)(lz - (double)hz), 0.f);
    for (int r = 0; r < R; ++r) qt[(long long)r * N + i] = (float)q[(long long)r * N + i];
  }
  const long long P = p2p_pairs_capacity(N);
  const int G = (R + MR_G - 1) / MR_G;
  for (long long pp = threadIdx.x; pp < b1 - b0; pp += blockDim.x) {
    float h[2][3], l[2][3];
    bool real[2];
    for (int u = 0; u < 2; ++u) {
      const long long j = s0 + 2 * pp + u;
      real[u] = j < s1;
      const double d[3] = {real[u] ? x[j] - x0 : P2P32_PAD, real[u] ? y[j] - y0 : P2P32_PAD,
                           real[u] ? z[j] - z0 : P2P32_PAD};
      for (int a = 0; a < 3; ++a) {
        h[u][a] = (float)d[a];
        l[u][a] = (float)(d[a] - (double)h[u][a]);
      }
    }
    const long long j0 = s0 + 2 * pp;
    auto charge = [&](int r, int u) -> float {
      return (r < R && real[u]) ? (float)q[(long long)r * N + j0 + u] : 0.f;
    };
    for (int g = 0; g < G; ++g) {
      float4 *rec = src + ((long long)g * P + b0 + pp) * MR_REC;
      rec[0] = make_float4(-h[0][0], -h[1][0], -h[0][1], -h[1][1]);
      rec[1] = make_float4(-h[0][2], -h[1][2], -l[0][2], -l[1][2]);
      rec[2] = make_float4(-l[0][0], -l[1][0], -l[0][1], -l[1][1]);
      const int r0 = MR_G * g;
      rec[3] = make_float4(charge(r0, 0), charge(r0, 1), charge(r0 + 1, 0), charge(r0 + 1, 1));
      rec[4] = make_float4(charge(r0 + 2, 0), charge(r0 + 2, 1), charge(r0 + 3, 0), charge(r0 + 3, 1));
    }
  }
}

// One record (two sources) against the lane's target for MR_G right-hand sides: the geometry once, then per
// right-hand side phi += q / r and the force sums q d / r^3.
template <bool SELF>
__device__ __forceinline__ void p2p_record_mrhs(const float4 *__restrict__ s, int k, int self_rel, float2 th_x,
                                                float2 th_y, float2 th_z, float2 tl_x, float2 tl_y, float2 tl_z,
                                                float2 (&pv)[MR_G], float2 (&ax)[MR_G], float2 (&ay)[MR_G],
                                                float2 (&az)[MR_G]) {
  const float4 A = s[MR_REC * k], B = s[MR_REC * k + 1], C = s[MR_REC * k + 2], Q0 = s[MR_REC * k + 3],
               Q1 = s[MR_REC * k + 4];
  const float2 dx = __fadd2_rn(__fadd2_rn(th_x, make_float2(A.x, A.y)), __fadd2_rn(tl_x, make_float2(C.x, C.y)));
  const float2 dy = __fadd2_rn(__fadd2_rn(th_y, make_float2(A.z, A.w)), __fadd2_rn(tl_y, make_float2(C.z, C.w)));
  const float2 dz = __fadd2_rn(__fadd2_rn(th_z, make_float2(B.x, B.y)), __fadd2_rn(tl_z, make_float2(B.z, B.w)));
  float2 r2 = __fmul2_rn(dx, dx);
  r2 = __ffma2_rn(dy, dy, r2);
  r2 = __ffma2_rn(dz, dz, r2);
  float2 inv;
  if (SELF) {
    inv = make_float2(2 * k == self_rel ? 0.f : rsqrt_ftz(r2.x), 2 * k + 1 == self_rel ? 0.f : rsqrt_ftz(r2.y));
  } else {
    inv = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
  }
  const float2 inv2 = __fmul2_rn(inv, inv);
  const float2 q[MR_G] = {make_float2(Q0.x, Q0.y), make_float2(Q0.z, Q0.w), make_float2(Q1.x, Q1.y),
                          make_float2(Q1.z, Q1.w)};
#pragma unroll
  for (int g = 0; g < MR_G; ++g) {
    const float2 qi = __fmul2_rn(q[g], inv);
    const float2 qi3 = __fmul2_rn(qi, inv2);
    pv[g] = __fadd2_rn(pv[g], qi);
    ax[g] = __ffma2_rn(dx, qi3, ax[g]);
    ay[g] = __ffma2_rn(dy, qi3, ay[g]);
    az[g] = __ffma2_rn(dz, qi3, az[g]);
  }
}

// One warp per work item and group of MR_G right-hand sides (grid.y): runs of records in bulk-copy stages, one target
// per lane (two would need 64 accumulator registers more), lane groups for small leaves, packed compensated sums after
// every MR_FLUSH records of a stage.  With the groups one after the other in a warp, 4,096 leaves of 61 gave 1.7 waves
// of long items: 3.7 -> 2.45 ms with the groups on the grid, items of 32 targets and stages of 48 records instead of 32
// (250k points x 16).  One compensated sum per 48 records let the FP32 chains grow: against FP64 the potential's error
// was 1.0-1.3 and the forces' 1.0-1.2 times that of one per 32 (seven clouds, 8 seeds).  With one per 24 they are
// 0.81-1.0 and 0.88-1.0 times, for 2.56 ms.  Two warps per CTA.
__global__ void __launch_bounds__(P2P32_WARPS * 32, 8) p2p_fp32_mrhs_kernel(
    int R, long long N, long long nleaves, const long long *__restrict__ leaf_start, const int *__restrict__ nbr,
    int variant, const int *__restrict__ rank_of, const long long *__restrict__ rec_base,
    const long long *__restrict__ chunk_base, int whole, int isize, const long long *__restrict__ shard,
    const float4 *__restrict__ pq, const float4 *__restrict__ plo, const float *__restrict__ qt,
    const float4 *__restrict__ src,
    double4 *__restrict__ res, int *__restrict__ status) {
  __shared__ __align__(128) float4 buf[P2P32_WARPS][P2P32_NBUF][MR_REC * MR_STAGE];
  __shared__ __align__(8) unsigned long long bar[P2P32_WARPS][P2P32_NBUF];
  __shared__ long long rbase[P2P32_WARPS][27];
  __shared__ int rcount[P2P32_WARPS][27];
  __shared__ unsigned char rself[P2P32_WARPS][27];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    for (int b = 0; b < P2P32_NBUF; ++b) mbar_init(&bar[w][b], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  // the work items of the targets' leaves: all, or the shard's [shard[0], shard[1])
  const long long leaf_lo = shard ? shard[0] : 0, leaf_hi = shard ? shard[1] : nleaves;
  const long long item0 = chunk_base ? chunk_base[leaf_lo] : leaf_lo;
  const long long item1 = chunk_base ? chunk_base[leaf_hi] : leaf_hi;
  const long long item = item0 + (long long)blockIdx.x * P2P32_WARPS + w;
  long long leaf, c0, c1;
  if (item >= item1 || !p2p_item(item, nleaves, leaf_start, chunk_base, whole, isize, leaf, c0, c1)) return;
  const long long P = p2p_pairs_capacity(N);
  const long long t0 = leaf_start[leaf];
  const int my_rank = rank_of ? rank_of[leaf] : (int)leaf;
  const long long self_rec = rec_begin(rec_base, leaf_start, my_rank);
  int nr = 0;
  {
    const int e = lane < 27 ? lane : 26;
    int nb = lane < 27 ? nbr[leaf * 27 + e] : -1;
    if (variant == 1 && e == 13) nb = -1;
    const int rk = nb >= 0 ? (rank_of ? rank_of[nb] : nb) : -1;
    const int dz = e % 3;
    const int rk_prev = __shfl_up_sync(0xffffffffu, rk, 1);
    const int rk_next = __shfl_down_sync(0xffffffffu, rk, 1);
    const int rk_next2 = __shfl_down_sync(0xffffffffu, rk, 2);
    const bool start = lane < 27 && rk >= 0 && !(dz > 0 && rk_prev >= 0 && rk_prev + 1 == rk);
    int last = rk;
    if (dz < 2 && rk_next >= 0 && rk_next == last + 1) {
      last = rk_next;
      if (dz == 0 && rk_next2 >= 0 && rk_next2 == last + 1) last = rk_next2;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, start);
    if (start) {
      const int k = __popc(mask & ((1u << lane) - 1u));
      const long long b0 = rec_begin(rec_base, leaf_start, rk), b1 = rec_begin(rec_base, leaf_start, last + 1);
      rbase[w][k] = b0;
      rcount[w][k] = (int)(b1 - b0);
      rself[w][k] = (variant == 0 && e / 3 == 4 && rk <= my_rank && my_rank <= last) ? 1 : 0;
    }
    nr = __popc(mask);
    __syncwarp();
  }
  unsigned phase_bits = 0;
  const int G = (R + MR_G - 1) / MR_G;
  for (int grp = blockIdx.y; grp < G; grp += gridDim.y) {
    const float4 *sr = src + (long long)grp * P * MR_REC;
    for (long long tb = c0; tb < c1; tb += 32) {
      const int m = (int)min(32LL, c1 - tb);
      const int T = m <= 8 ? 8 : (m <= 16 ? 16 : 32);
      const int Gl = 32 / T;  // lane groups, each on every Gl-th record
      const int tl = lane & (T - 1), g = lane / T;
      const long long i = tb + tl;
      const bool active = tl < m;
      const float4 me = active ? pq[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 mel = active ? plo[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      const long long self_slot = 2 * self_rec + (i - t0);
      const float2 th_x = make_float2(me.x, me.x), th_y = make_float2(me.y, me.y), th_z = make_float2(me.z, me.z);
      const float2 tl_x = make_float2(mel.x, mel.x), tl_y = make_float2(mel.y, mel.y), tl_z = make_float2(mel.z, mel.z);
      // compensated potential and force sums of the right-hand sides 2 v (.x) and 2 v + 1 (.y)
      float2 hi[4][MR_G / 2], lo[4][MR_G / 2];
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int v = 0; v < MR_G / 2; ++v) hi[c][v] = lo[c][v] = make_float2(0.f, 0.f);
      int ie = 0, ip = 0, ce = 0, cp = 0, issued = 0, done = 0;
      auto next_stage = [&](int &e, int &p0, int &n) -> bool {
        while (e < nr && p0 >= rcount[w][e]) {
          ++e;
          p0 = 0;
        }
        if (e >= nr) return false;
        n = min(MR_STAGE, rcount[w][e] - p0);
        return true;
      };
      auto issue = [&]() {
        int n;
        if (!next_stage(ie, ip, n)) return false;
        const int b = issued % P2P32_NBUF;
        if (lane == 0) {
          mbar_expect_tx(&bar[w][b], n * MR_REC * 16);
          bulk_g2s(&buf[w][b][0], sr + (rbase[w][ie] + ip) * MR_REC, n * MR_REC * 16, &bar[w][b]);
        }
        ip += n;
        ++issued;
        return true;
      };
      for (int k = 0; k < P2P32_NBUF - 1; ++k)
        if (!issue()) break;
      while (done < issued) {
        int cn;
        next_stage(ce, cp, cn);
        const int b = done % P2P32_NBUF;
        if (!mbar_wait_warp(&bar[w][b], (phase_bits >> b) & 1u)) {
          if (lane == 0) {
            atomicExch(status, 1);
            for (int k = done; k < issued; ++k) {
              const int bk = k % P2P32_NBUF;
              mbar_wait(&bar[w][bk], (phase_bits >> bk) & 1u);
            }
          }
          __syncwarp();
          return;
        }
        phase_bits ^= 1u << b;
        const float4 *s = buf[w][b];
        const bool own = rself[w][ce];
        const int self_rel = (int)(self_slot - 2 * (rbase[w][ce] + cp));
#pragma unroll 1
        for (int k0 = 0; k0 < cn; k0 += MR_FLUSH) {
          const int k1 = min(cn, k0 + MR_FLUSH);
          float2 acc[4][MR_G];
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int k = 0; k < MR_G; ++k) acc[c][k] = make_float2(0.f, 0.f);
          if (own) {
            for (int k = k0 + g; k < k1; k += Gl)
              p2p_record_mrhs<true>(s, k, self_rel, th_x, th_y, th_z, tl_x, tl_y, tl_z, acc[0], acc[1], acc[2], acc[3]);
          } else {
#pragma unroll 1  // by two: 40 bytes of spills, no faster
            for (int k = k0 + g; k < k1; k += Gl)
              p2p_record_mrhs<false>(s, k, 0, th_x, th_y, th_z, tl_x, tl_y, tl_z, acc[0], acc[1], acc[2], acc[3]);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int v = 0; v < MR_G / 2; ++v)
              two_sum2(hi[c][v], lo[c][v], make_float2(acc[c][2 * v].x + acc[c][2 * v].y,
                                                       acc[c][2 * v + 1].x + acc[c][2 * v + 1].y));
        }
        cp += cn;
        ++done;
        __syncwarp();
        issue();
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int v = 0; v < MR_G / 2; ++v)
          for (int off = T; off < 32; off <<= 1) {
            const float2 oh = make_float2(__shfl_xor_sync(0xffffffffu, hi[c][v].x, off),
                                          __shfl_xor_sync(0xffffffffu, hi[c][v].y, off));
            const float2 ol = make_float2(__shfl_xor_sync(0xffffffffu, lo[c][v].x, off),
                                          __shfl_xor_sync(0xffffffffu, lo[c][v].y, off));
            two_sum2(hi[c][v], lo[c][v], oh);
            lo[c][v] = __fadd2_rn(lo[c][v], ol);
          }
#pragma unroll
      for (int k = 0; k < MR_G; ++k) {
        const int r = MR_G * grp + k;
        if (active && g == 0 && r < R) {
          const long long j = (long long)r * N + i;
          const double nq = -(double)qt[j];
          double v[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float2 h = hi[c][k / 2], l = lo[c][k / 2];
            v[c] = k % 2 == 0 ? (double)h.x + (double)l.x : (double)h.y + (double)l.y;
          }
          add_result(res + j, v[0], nq * v[1], nq * v[2], nq * v[3]);
        }
      }
    }
  }
}

}  // namespace

b200fmm_status run_p2p(Context &c, int variant, const long long *shard) {
  const int LL = c.H - 1;
  const Level &L = c.lv[LL];
  if (L.n == 0) return B200FMM_OK;
  // a graph builds the tables that it needs itself: what is only captured has not run, and may never
  const bool captured = stream_captured(c);
  if (c.cfg.precision == B200FMM_MIXED && c.R > 1) {
    // several right-hand sides: targets hi [N], lo [N], charges [R][N] (floats), then the record groups; the
    // buffer sized for the single-RHS layout of R vectors holds this one
    float4 *hi = c.d_pq32, *lo = c.d_pq32 + c.N;
    float *qt = (float *)(c.d_pq32 + 2 * c.N);
    float4 *src = c.d_pq32 + 2 * c.N + (c.N * c.R + 3) / 4;
    if (!c.packed32 || captured) {
      if (c.column_serial != c.tree_serial) {
        B200_CHECK(leaf_column_order(c));
        if (!captured) c.column_serial = c.tree_serial;
      }
      c.packed32 = !captured;
      const double W = c.cfg.box_width;
      pack_records32_mrhs<<<(unsigned)L.n, 64, 0, c.stream>>>(
          c.N, c.R, c.d_leaf_start, c.d_leaf_rank, c.d_rec_base, c.d_x, c.d_y, c.d_z, c.d_q, c.cfg.center[0] - W / 2,
          c.cfg.center[1] - W / 2, c.cfg.center[2] - W / 2, hi, lo, qt, src);
      ++c.launches;
    }
    // work items (p2p_leaf_items per leaf): nleaves + N / item bounds their count
    const unsigned blocks = grid_for(L.n + c.N / c.p2p_item, P2P32_WARPS);
    B200_CUDA(record_event(c, 10));
    p2p_fp32_mrhs_kernel<<<dim3(blocks, (c.R + MR_G - 1) / MR_G), P2P32_WARPS * 32, 0, c.stream>>>(
        c.R, c.N, L.n, c.d_leaf_start, c.d_leaf_nbr, variant, c.d_leaf_rank, c.d_rec_base, c.d_chunk_base, c.p2p_whole,
        c.p2p_item, shard, hi, lo, qt, src, c.d_res, c.d_status);
    B200_CUDA(record_event(c, 11));
    ++c.launches;
  } else if (c.cfg.precision == B200FMM_MIXED) {
    float4 *hi = c.d_pq32, *lo = c.d_pq32 + c.N * c.R, *src = c.d_pq32 + c.N * (c.R + 1);
    if (!c.packed32 || captured) {
      if (c.column_serial != c.tree_serial) {
        B200_CHECK(leaf_column_order(c));
        if (!captured) c.column_serial = c.tree_serial;
      }
      c.packed32 = !captured;
      const double W = c.cfg.box_width;
      pack_records32<<<(unsigned)L.n, 64, 0, c.stream>>>(c.N, c.R, c.d_leaf_start, c.d_leaf_rank, c.d_rec_base, c.d_x,
                                                         c.d_y, c.d_z, c.d_q, c.cfg.center[0] - W / 2,
                                                         c.cfg.center[1] - W / 2, c.cfg.center[2] - W / 2, hi, lo, src);
      ++c.launches;
    }
    int *status = c.d_status;
    // work items (p2p_leaf_items per leaf): nleaves + N / item bounds their count
    const unsigned blocks = grid_for(L.n + c.N / c.p2p_item, P2P32_WARPS);
    B200_CUDA(record_event(c, 10));
    p2p_fp32_kernel<<<blocks, P2P32_WARPS * 32, 0, c.stream>>>(
        c.R, c.N, L.n, c.d_leaf_start, c.d_leaf_nbr, variant, c.d_leaf_rank, c.d_rec_base, c.d_chunk_base, c.p2p_whole,
        c.p2p_item, shard, hi, lo, src, OutRecords{c.d_res}, status);
    B200_CUDA(record_event(c, 11));
    ++c.launches;
  } else {
    if (c.column_serial != c.tree_serial) {
      B200_CHECK(leaf_items(c, P2P64_TGT, P2P64_TGT));
      if (!captured) c.column_serial = c.tree_serial;
    }
    B200_CUDA(record_event(c, 10));
    // nleaves + N / 32 bounds the work items; several right-hand sides share a pair's geometry four at a time
    const unsigned blocks = grid_for(L.n + c.N / P2P64_TGT, 1);
    auto kernel = c.R > 1 ? p2p_fp64_kernel<4> : p2p_fp64_kernel<1>;
    kernel<<<blocks, P2P64_THREADS, 0, c.stream>>>(c.R, c.N, L.n, c.d_leaf_start, c.d_leaf_nbr, c.d_chunk_base, variant,
                                                   c.d_x, c.d_y, c.d_z, c.d_q, c.d_res, shard);
    B200_CUDA(record_event(c, 11));
    ++c.launches;
  }
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

}  // namespace b200

// ---- allocation-free entry point -------------------------------------------------------------------
// Scratch of b200fmm_p2p_noalloc: the FP32 copies of the particles -- targets (hi, lo) and
// pair-packed sources, 6 float4 per particle plus 8 (24 MiB at 2^18 particles) -- and the status words:
// [0] a bounded wait of the near-field kernel ran out, [1] the caller's leaf tables failed the checks.  In host
// code these names are host-side stand-ins, not device addresses: the host passes the addresses looked up with
// cudaGetSymbolAddress.
static __device__ __align__(256) float4 g_noalloc_stage[6 * B200FMM_NOALLOC_MAX_PARTICLES + 8];
static __device__ __align__(256) int g_noalloc_status[4];

namespace b200 {
namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
float4 *g_noalloc_stage_ptr[kMaxDevices] = {};
int *g_noalloc_status_ptr[kMaxDevices] = {};

// Once per device, with that device current: the device addresses of the file-scope arrays.
b200fmm_status noalloc_addresses(float4 **stage, int **status) {
  int dev = -1;
  B200_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(B200FMM_ERR_UNSUPPORTED, "device ordinal out of range");
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_stage_ptr[dev]) {
    void *a = nullptr, *b = nullptr;
    B200_CUDA(cudaGetSymbolAddress(&a, g_noalloc_stage));
    B200_CUDA(cudaGetSymbolAddress(&b, g_noalloc_status));
    g_noalloc_stage_ptr[dev] = (float4 *)a;
    g_noalloc_status_ptr[dev] = (int *)b;
  }
  *stage = g_noalloc_stage_ptr[dev];
  *status = g_noalloc_status_ptr[dev];
  return B200FMM_OK;
}

// The caller's leaf tables are checked before any kernel indexes memory through them: leaf_start rises from 0
// to n, the leaf keys rise strictly inside the leaf level, every neighbour entry is -1 or a leaf index, and
// position 13 names the leaf itself.  With these, every particle index the packing and near-field kernels form
// lies in [0, n) and every source record in [0, n + 2), inside the scratch array.  A failure sets status[1].
__global__ void noalloc_check_tables(long long n, long long nleaves, const long long *__restrict__ leaf_keys,
                                     const long long *__restrict__ leaf_start, const int *__restrict__ nbr,
                                     long long key_end, int *__restrict__ status) {
  bool bad = false;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nleaves * 27; i += stride) {
    const int v = nbr[i];
    const long long leaf = i / 27;
    bad |= v < -1 || v >= nleaves || (i % 27 == 13 && v != leaf);
    if (i % 27 == 0) {
      const long long s0 = leaf_start[leaf], s1 = leaf_start[leaf + 1], k = leaf_keys[leaf];
      bad |= s0 < 0 || s1 < s0 || s1 > n || k < 0 || k >= key_end;
      bad |= leaf == 0 && s0 != 0;
      bad |= leaf == nleaves - 1 && s1 != n;
      bad |= leaf > 0 && leaf_keys[leaf - 1] >= k;
    }
  }
  if (bad) atomicExch(status + 1, 1);
}
}  // namespace
}  // namespace b200

extern "C" b200fmm_status b200fmm_p2p_noalloc(long long n, const double *x, const double *y, const double *z,
                                              const double *q, long long nleaves, const long long *leaf_keys,
                                              const long long *leaf_start, const int *leaf_nbr, int height,
                                              double box_width, const double *center, int variant, double *phi,
                                              double *fx, double *fy, double *fz, void *stream) {
  using namespace b200;
  if (n < 1 || nleaves < 1 || nleaves > n) return fail(B200FMM_ERR_INVALID, "p2p_noalloc: bad particle/leaf count");
  if (n > B200FMM_NOALLOC_MAX_PARTICLES)
    return fail(B200FMM_ERR_INVALID, "p2p_noalloc: more than B200FMM_NOALLOC_MAX_PARTICLES (262144) particles");
  if (!x || !y || !z || !q || !leaf_keys || !leaf_start || !leaf_nbr || !center || !phi || !fx || !fy || !fz)
    return fail(B200FMM_ERR_INVALID, "p2p_noalloc: null pointer");
  if (height < 2 || height > kMaxHeight) return fail(B200FMM_ERR_INVALID, "p2p_noalloc: height out of range");
  if (variant != 0 && variant != 1) return fail(B200FMM_ERR_INVALID, "p2p_noalloc: variant must be 0 or 1");
  if (!(box_width > 0)) return fail(B200FMM_ERR_INVALID, "p2p_noalloc: bad box width");
  float4 *stage = nullptr;
  int *status = nullptr;
  B200_CHECK(noalloc_addresses(&stage, &status));
  cudaStream_t s = (cudaStream_t)stream;
  int st[2] = {0, 0};
  // 1) the tables, read back before anything indexes through them
  B200_CUDA(cudaMemsetAsync(status, 0, sizeof(int) * 4, s));
  const long long key_end = 1LL << (3 * (height - 1));
  noalloc_check_tables<<<grid_for(nleaves * 27, 256) < 1184 ? grid_for(nleaves * 27, 256) : 1184, 256, 0, s>>>(
      n, nleaves, leaf_keys, leaf_start, leaf_nbr, key_end, status);
  B200_CUDA(cudaGetLastError());
  B200_CUDA(cudaMemcpyAsync(st, status, sizeof(st), cudaMemcpyDeviceToHost, s));
  B200_CUDA(cudaStreamSynchronize(s));
  if (st[1])
    return fail(B200FMM_ERR_INVALID,
                "p2p_noalloc: inconsistent leaf tables (leaf_start must rise from 0 to n, leaf keys rise strictly "
                "inside the leaf level, neighbour entries be -1 or a leaf index with position 13 the leaf itself)");
  // 2) the FP32 copies and the near field
  pack_records32<<<(unsigned)nleaves, 64, 0, s>>>(n, 1, leaf_start, nullptr, nullptr, x, y, z, q,
                                                 center[0] - box_width / 2, center[1] - box_width / 2,
                                                 center[2] - box_width / 2, stage, stage + n, stage + 2 * n);
  p2p_fp32_kernel<<<grid_for(nleaves, P2P32_WARPS), P2P32_WARPS * 32, 0, s>>>(
      1, n, nleaves, leaf_start, leaf_nbr, variant, nullptr, nullptr, nullptr, 0, 0, nullptr, stage, stage + n,
      stage + 2 * n, OutArrays{phi, fx, fy, fz}, status);
  B200_CUDA(cudaGetLastError());
  B200_CUDA(cudaMemcpyAsync(st, status, sizeof(st), cudaMemcpyDeviceToHost, s));
  B200_CUDA(cudaStreamSynchronize(s));
  if (st[0]) return fail(B200FMM_ERR_CUDA, "p2p_noalloc: a device wait ran out of its iteration budget");
  return B200FMM_OK;
}
