// P2M / M2M / L2L / L2P in FP64 for the Chebyshev and Lagrange bases.
//
//  P2M  M[n] += sum_particles q * prod_d S_{n_d}(x_d)      (FChebInterpolator::applyP2M,
//                                                            Src/Kernels/Chebyshev/FChebInterpolator.hpp:627-762)
//  M2M  parent[n] += sum_m prod_d S[c][d][n_d][m_d] child[m] (applyM2M, FChebInterpolator.hpp:560-584)
//  L2L  child[m]  += sum_n prod_d S[c][d][n_d][m_d] parent[n] (applyL2L, FChebInterpolator.hpp:587-611)
//  L2P  phi += sum_n L[n] prod_d S_{n_d}(x_d); F += q * grad (applyL2PTotal, FChebInterpolator.hpp:1222-1417)
// with x mapped to [-1,1] around the leaf centre (map_glob_loc, Src/Kernels/Interpolation/FInterpMapping.hpp:
// 101-114; leaf centre FAbstractChebKernel.hpp:54-59).  Lagrange: FUnifInterpolator.hpp:340-549.
// Every contraction is done one axis at a time (p^4 work per cell instead of p^6); leaves are handled one
// CTA (P2M) or warp (L2P) each, parent cells one CTA each with one warp per child.
#include "common.cuh"

namespace b200 {

namespace {

// Interpolation nodes of every built order (3..8) and basis (Chebyshev, Lagrange), and the Chebyshev values
// T_o(node_j): read by P2M and L2P as constant-bank operands, so that the tables hold no registers.  The same for
// the child-to-parent interpolators of M2M and L2L, which are the same along every axis: one for the lower and one
// for the upper child.  Set per device when a handle builds its tables (upload_basis_constants); every handle of an
// order and basis writes the same values.
__constant__ double c_roots[2][kMaxOrder - 2][kMaxOrder];      // [basis: 1 = Lagrange][p - 3][j]
__constant__ double c_Tr[kMaxOrder - 2][kMaxOrder * kMaxOrder];  // [p - 3][o * p + j], Chebyshev
__constant__ double c_S[2][kMaxOrder - 2][2][kMaxOrder * kMaxOrder];  // [basis][p - 3][child bit][n * p + m]

// S_j(x) and dS_j/dx for j < p.  Chebyshev: 1/p + 2/p sum_o T_o(x) T_o(xbar_j), dT_o = o U_{o-1}.
// Lagrange (equispaced nodes): prod_{m != j} (x - x_m) / (x_j - x_m) and its derivative.  Compile-time order
// and basis, every loop unrolled, so that S and dS stay in registers.
template <int P, bool LAGR>
__device__ __forceinline__ void basis_eval(double x, double *S, double *dS) {
  constexpr int p = P;
  const double *roots = c_roots[LAGR ? 1 : 0][P - 3];
  if constexpr (LAGR) {
    if (x > 1.0) x = 1.0;
    if (x < -1.0) x = -1.0;
#pragma unroll
    for (int j = 0; j < p; ++j) {
      double num = 1.0, den = 1.0, dsum = 0.0;
#pragma unroll
      for (int m = 0; m < p; ++m) {
        if (m == j) continue;
        den *= roots[j] - roots[m];
        num *= x - roots[m];
      }
      if (dS) {
#pragma unroll
        for (int k = 0; k < p; ++k) {
          if (k == j) continue;
          double t = 1.0;
#pragma unroll
          for (int m = 0; m < p; ++m)
            if (m != j && m != k) t *= x - roots[m];
          dsum += t;
        }
        dS[j] = dsum / den;
      }
      S[j] = num / den;
    }
  } else {
    double T[P], U[P];
    T[0] = 1.0;
    T[1] = x;
    U[0] = 1.0;
    U[1] = 2.0 * x;
#pragma unroll
    for (int o = 2; o < p; ++o) {
      T[o] = 2.0 * x * T[o - 1] - T[o - 2];
      U[o] = 2.0 * x * U[o - 1] - U[o - 2];
    }
    const double ip = 1.0 / p;
#pragma unroll
    for (int j = 0; j < p; ++j) {
      double s = ip, ds = 0.0;
#pragma unroll
      for (int o = 1; o < p; ++o) {
        const double t = 2.0 * ip * c_Tr[P - 3][o * p + j];
        s += T[o] * t;
        ds += (double)o * U[o - 1] * t;
      }
      S[j] = s;
      if (dS) dS[j] = ds;
    }
  }
}

// Record the largest |value| a warp wrote (mx per lane; every lane of the warp calls it) into one of the
// level's kMmaxSlots slots, chosen by block: non-negative doubles order like their bit patterns.
__device__ __forceinline__ void record_max(unsigned long long *slots, double mx) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0 && mx > 0.0)
    atomicMax(slots + blockIdx.x % kMmaxSlots, (unsigned long long)__double_as_longlong(mx));
}

// ---- P2M: one 64-thread block per leaf -------------------------------------------------------------
// M[nx,ny,nz] = sum_j q_j Sx_j[nx] Sy_j[ny] Sz_j[nz].  The threads first evaluate the 1-D weights of up to 64
// particles (one each) into shared memory; then thread t < p^2 owns the node line (ny, nz) = (t % p, t / p)
// and keeps its p sums over nx in registers: per particle one product q Sy Sz and p FMAs with the
// broadcast Sx row, instead of three shared-memory reads per node and particle.  Several right-hand sides are taken
// two at a time, with the weights of a leaf of one chunk evaluated once (250k points x 16, order 7: 0.48 -> 0.29 ms:
// the shared-memory reads of the weights bound it).  (Measured slower, 1M uniform, order 7, height 6: 128 threads, the
// weights along rows of particles, two particles per load and two node lines per lane, 0.250 against 0.148 ms: 96
// registers with spills and three more barriers per leaf cost more than the halved shared-memory reads give.)
constexpr int P2M_THREADS = 64;
constexpr int L2P_WARPS = 1;  // L2P: leaves per CTA, one warp each (static shared memory <= 48 KB at order 8)

template <int P, bool LAGR, int NR>
__global__ void __launch_bounds__(P2M_THREADS, 8) p2m_kernel(
    int R, long long N, long long nleaves, const long long *__restrict__ keys,
    const long long *__restrict__ leaf_start, const double *__restrict__ x, const double *__restrict__ y,
    const double *__restrict__ z, const double *__restrict__ q, double cx0, double cy0, double cz0, double leaf_w,
    double *__restrict__ M, unsigned long long *__restrict__ mmax) {
  constexpr int p = P, nn = P * P * P;
  constexpr int PX = P <= 6 ? (P + 1) & ~1 : 10;  // Sx rows: 16-byte steps, spread over the banks
  __shared__ __align__(16) double Wx[P2M_THREADS][PX];
  __shared__ double Wy[P2M_THREADS][P], Wz[P2M_THREADS][P], Q[NR][P2M_THREADS];
  const int t = threadIdx.x;
  const long long leaf = blockIdx.x;
  int ix, iy, iz;
  morton_decode3(keys[leaf], ix, iy, iz);
  const double ctr[3] = {cx0 + (ix + 0.5) * leaf_w, cy0 + (iy + 0.5) * leaf_w, cz0 + (iz + 0.5) * leaf_w};
  const long long s0 = leaf_start[leaf], s1 = leaf_start[leaf + 1];
  const int ny = t % p, nz = t / p;
  const bool owner = t < p * p;
  for (int r0 = 0; r0 < R; r0 += NR) {
    double acc[NR][P];
#pragma unroll
    for (int u = 0; u < NR; ++u)
#pragma unroll
      for (int k = 0; k < p; ++k) acc[u][k] = 0.0;
    for (long long b = s0; b < s1; b += P2M_THREADS) {
      const int cnt = (int)min((long long)P2M_THREADS, s1 - b);
      __syncthreads();
      if (t < cnt) {
        const long long i = b + t;
        if (r0 == 0 || s1 - s0 > P2M_THREADS) {
          const double pos[3] = {x[i], y[i], z[i]};
          double wv[P];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const double a = ctr[d] - leaf_w / 2, bb = ctr[d] + leaf_w / 2;
            basis_eval<P, LAGR>((2.0 * pos[d] - bb - a) / (bb - a), wv, nullptr);
            double *dst = d == 0 ? Wx[t] : (d == 1 ? Wy[t] : Wz[t]);
#pragma unroll
            for (int k = 0; k < p; ++k) dst[k] = wv[k];
          }
        }
#pragma unroll
        for (int u = 0; u < NR; ++u) Q[u][t] = r0 + u < R ? q[(long long)(r0 + u) * N + i] : 0.0;
      }
      __syncthreads();
      if (owner) {
        for (int j = 0; j < cnt; ++j) {
          const double wyz = Wy[j][ny] * Wz[j][nz];
#pragma unroll
          for (int u = 0; u < NR; ++u) {
            const double w = Q[u][j] * wyz;
#pragma unroll
            for (int k = 0; k < p; ++k) acc[u][k] += w * Wx[j][k];
          }
        }
      }
    }
    double mx = 0.0;
    if (owner) {
#pragma unroll
      for (int u = 0; u < NR; ++u) {
        if (r0 + u >= R) break;
        double *out = M + (leaf * R + r0 + u) * nn + (nz * p + ny) * p;
#pragma unroll
        for (int k = 0; k < p; ++k) {
          const double v = out[k] + acc[u][k];
          out[k] = v;
          mx = fmax(mx, fabs(v));
        }
      }
    }
    if (mmax) record_max(mmax, mx);
  }
}

// ---- M2M / L2L: one warp per child ------------------------------------------------------------------
// Each warp applies the child's three 1-D interpolators, one axis at a time, in place in its shared-memory block
// (rows of p values padded to an odd length).  A lane owns whole lines along the axis: it loads the line's p values
// into registers and writes the p results; the p x p interpolator is read as constant-bank operands, by a branch on
// the child's bit of that axis.  (Loaded from global memory by every lane it cost 147 broadcast loads per child: the
// load pipe was 75 % busy.)  M2M: the 8 children's contributions to the parent are then added in child order
// (deterministic).  1M uniform, order 7, height 6, all levels: M2M 0.124 -> 0.087 ms, L2L 0.113 -> 0.072 ms.
template <int P>
struct Block {
  static constexpr int PR = P | 1;             // row length
  static constexpr int SIZE = P * P * PR;      // doubles
  static __device__ __forceinline__ int at(int e) { return e / P * PR + e % P; }
};

template <int P, bool LAGR, bool TRANSPOSE, int D, int BIT>
__device__ __forceinline__ void warp_lines_bit(const double *in, double *out, int lane) {
  constexpr int p = P, nl = P * P, PR = Block<P>::PR;
  constexpr int stride = D == 0 ? 1 : (D == 1 ? PR : PR * P);
  constexpr int LN = (nl + 31) / 32;  // a lane's lines, together: each interpolator value is read once
  const double *A = c_S[LAGR ? 1 : 0][P - 3][BIT];
  int base[LN];
  double v[LN][P];
#pragma unroll
  for (int u = 0; u < LN; ++u) {
    const int l = lane + 32 * u;
    // first element of line l: the two other indices of the line, in increasing axis order
    base[u] = D == 0 ? l * PR : (D == 1 ? (l % p) + (l / p) * PR * p : (l % p) + (l / p) * PR);
#pragma unroll
    for (int m = 0; m < p; ++m) v[u][m] = l < nl ? in[base[u] + m * stride] : 0.0;
  }
#pragma unroll
  for (int i = 0; i < p; ++i) {
    double s[LN];
#pragma unroll
    for (int u = 0; u < LN; ++u) s[u] = 0.0;
#pragma unroll
    for (int m = 0; m < p; ++m)
#pragma unroll
      for (int u = 0; u < LN; ++u) s[u] += A[TRANSPOSE ? m * p + i : i * p + m] * v[u][m];
#pragma unroll
    for (int u = 0; u < LN; ++u)
      if (lane + 32 * u < nl) out[base[u] + i * stride] = s[u];
  }
}
template <int P, bool LAGR, bool TRANSPOSE, int D>
__device__ __forceinline__ void warp_lines(int child, const double *in, double *out, int lane) {
  if ((child >> (2 - D)) & 1)
    warp_lines_bit<P, LAGR, TRANSPOSE, D, 1>(in, out, lane);
  else
    warp_lines_bit<P, LAGR, TRANSPOSE, D, 0>(in, out, lane);
}

template <int P, bool LAGR>
__global__ void __launch_bounds__(256, 2) m2m_kernel(int R, long long nparents, const int *__restrict__ child,
                                                  const double *__restrict__ Mc, double *__restrict__ Mp,
                                                  unsigned long long *__restrict__ mmax) {
  constexpr int nn = P * P * P, K = (nn + 31) / 32, KP = (nn + 255) / 256;
  using B = Block<P>;
  extern __shared__ double sh[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *b = sh + (size_t)w * B::SIZE;  // the child's multipole, then its contribution
  const long long pc = blockIdx.x;
  const int ci = child[pc * 8 + w];
  for (int r = 0; r < R; ++r) {
    double *out = Mp + (pc * R + r) * nn;
    double old[KP];
    if (ci >= 0) {
      const double *src = Mc + ((long long)ci * R + r) * nn;
      double v[K];
#pragma unroll
      for (int k = 0; k < K; ++k) v[k] = lane + 32 * k < nn ? src[lane + 32 * k] : 0.0;
#pragma unroll
      for (int k = 0; k < KP; ++k) old[k] = threadIdx.x + 256 * k < nn ? out[threadIdx.x + 256 * k] : 0.0;
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (lane + 32 * k < nn) b[B::at(lane + 32 * k)] = v[k];
      __syncwarp();
      warp_lines<P, LAGR, false, 0>(w, b, b, lane);
      __syncwarp();
      warp_lines<P, LAGR, false, 1>(w, b, b, lane);
      __syncwarp();
      warp_lines<P, LAGR, false, 2>(w, b, b, lane);
    } else {
#pragma unroll
      for (int k = 0; k < KP; ++k) old[k] = threadIdx.x + 256 * k < nn ? out[threadIdx.x + 256 * k] : 0.0;
      for (int e = lane; e < B::SIZE; e += 32) b[e] = 0.0;
    }
    __syncthreads();
    double mx = 0.0;
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int e = threadIdx.x + 256 * k;
      if (e >= nn) continue;
      double s = 0.0;
#pragma unroll
      for (int c = 0; c < 8; ++c) s += sh[(size_t)c * B::SIZE + B::at(e)];
      const double v = old[k] + s;
      out[e] = v;
      mx = fmax(mx, fabs(v));
    }
    if (mmax) record_max(mmax, mx);
    __syncthreads();
  }
}

template <int P, bool LAGR>
__global__ void __launch_bounds__(256, 2) l2l_kernel(int R, long long nparents, const int *__restrict__ child,
                                                  const double *__restrict__ Lp, double *__restrict__ Lc) {
  constexpr int nn = P * P * P, K = (nn + 31) / 32, KP = (nn + 255) / 256;
  using B = Block<P>;
  extern __shared__ double sh[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *par = sh;  // parent local
  double *b = sh + (size_t)(w + 1) * B::SIZE;
  const long long pc = blockIdx.x;
  const int ci = child[pc * 8 + w];
  for (int r = 0; r < R; ++r) {
    const double *src = Lp + (pc * R + r) * nn;
    double *out = Lc + ((long long)ci * R + r) * nn;
    double v[KP], old[K];
#pragma unroll
    for (int k = 0; k < KP; ++k) v[k] = threadIdx.x + 256 * k < nn ? src[threadIdx.x + 256 * k] : 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) old[k] = ci >= 0 && lane + 32 * k < nn ? out[lane + 32 * k] : 0.0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KP; ++k)
      if (threadIdx.x + 256 * k < nn) par[B::at(threadIdx.x + 256 * k)] = v[k];
    __syncthreads();
    if (ci < 0) continue;
    warp_lines<P, LAGR, true, 0>(w, par, b, lane);
    __syncwarp();
    warp_lines<P, LAGR, true, 1>(w, b, b, lane);
    __syncwarp();
    warp_lines<P, LAGR, true, 2>(w, b, b, lane);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (lane + 32 * k < nn) out[lane + 32 * k] = old[k] + b[B::at(lane + 32 * k)];
    __syncwarp();
  }
}

// Copy NN doubles with T threads, all loads issued before the first store (one memory latency per copy
// instead of one per element).
template <int NN, int T>
__device__ __forceinline__ void copy_block(double *dst, const double *__restrict__ src, int tid) {
  constexpr int K = (NN + T - 1) / T;
  double v[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int e = tid + k * T;
    v[k] = e < NN ? src[e] : 0.0;
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int e = tid + k * T;
    if (e < NN) dst[e] = v[k];
  }
}

// ---- L2P: one warp per leaf, one particle per lane ----------------------------------------------------
// The leaf's local expansion sits in shared memory; each lane contracts it with its particle's weights one
// axis at a time: the x weights in registers, the y and z weights (and derivatives) in the lane's own
// shared-memory row, so that the loops over y and z need no register indexing and the kernel stays small.
// One warp per CTA, so that a leaf that ends frees its place at once, and all lanes through the last round together: 1M
// points, order 7, height 6 0.206 -> 0.184 ms, 2M on a surface 0.368 -> 0.348 ms, 200k clustered 0.139 -> 0.115 ms (two
// warps per CTA, lanes leaving one by one before).  Capping the registers for more CTAs, or two right-hand sides at a
// time, was slower.
template <int P, bool LAGR>
__global__ void __launch_bounds__(L2P_WARPS * 32) l2p_kernel(
    int R, long long N, long long nleaves, const long long *__restrict__ keys,
    const long long *__restrict__ leaf_start, const double *__restrict__ x, const double *__restrict__ y,
    const double *__restrict__ z, const double *__restrict__ q, double cx0, double cy0, double cz0, double leaf_w,
    const double *__restrict__ L,
    double4 *__restrict__ res, const long long *__restrict__ shard) {
  constexpr int p = P, nn = P * P * P;
  __shared__ double sL[L2P_WARPS][nn];
  __shared__ double sW[L2P_WARPS][32][4 * P + 1];  // wy, dwy, wz, dwz of each lane's particle (+1: banks)
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // every leaf, or the shard's [shard[0], shard[1])
  const long long leaf = (shard ? shard[0] : 0) + (long long)blockIdx.x * L2P_WARPS + w;
  if (leaf >= (shard ? shard[1] : nleaves)) return;
  double *Lw = sL[w];
  double *wy = sW[w][lane], *dwy = wy + P, *wz = wy + 2 * P, *dwz = wy + 3 * P;
  int ix, iy, iz;
  morton_decode3(keys[leaf], ix, iy, iz);
  const double cx = cx0 + (ix + 0.5) * leaf_w, cy = cy0 + (iy + 0.5) * leaf_w, cz = cz0 + (iz + 0.5) * leaf_w;
  const double jac = 2.0 / leaf_w;
  const long long s0 = leaf_start[leaf], s1 = leaf_start[leaf + 1];
  for (long long i0 = s0; i0 < s1; i0 += 32) {
    // every lane goes through a last partial round (a leaf's first particle where there is none)
    const bool on = i0 + lane < s1;
    const long long i = on ? i0 + lane : s0;
    double wx[P], dwx[P];
    {
      double t[P], dt[P];
      basis_eval<P, LAGR>((2.0 * y[i] - 2.0 * cy) / leaf_w, t, dt);
#pragma unroll
      for (int k = 0; k < p; ++k) {
        wy[k] = t[k];
        dwy[k] = dt[k];
      }
      basis_eval<P, LAGR>((2.0 * z[i] - 2.0 * cz) / leaf_w, t, dt);
#pragma unroll
      for (int k = 0; k < p; ++k) {
        wz[k] = t[k];
        dwz[k] = dt[k];
      }
    }
    basis_eval<P, LAGR>((2.0 * x[i] - 2.0 * cx) / leaf_w, wx, dwx);
    for (int r = 0; r < R; ++r) {
      if (i0 == s0 || R > 1) {
        __syncwarp();
        copy_block<nn, 32>(Lw, L + (leaf * R + r) * nn, lane);
        __syncwarp();
      }
      double pv = 0, gx = 0, gy = 0, gz = 0;
#pragma unroll 1
      for (int kz = 0; kz < p; ++kz) {
        double bz = 0, bzx = 0, bzy = 0;
#pragma unroll 1
        for (int ky = 0; ky < p; ++ky) {
          const double *row = Lw + (kz * p + ky) * p;
          double a = 0, ad = 0;
#pragma unroll
          for (int kx = 0; kx < p; ++kx) {
            const double v = row[kx];
            a += wx[kx] * v;
            ad += dwx[kx] * v;
          }
          const double yk = wy[ky];
          bz += yk * a;
          bzx += yk * ad;
          bzy += dwy[ky] * a;
        }
        const double zk = wz[kz];
        pv += zk * bz;
        gx += zk * bzx;
        gy += zk * bzy;
        gz += dwz[kz] * bz;
      }
      if (on) {
        const long long j = (long long)r * N + i;
        const double qq = q[j];
        add_result(res + j, pv, gx * jac * qq, gy * jac * qq, gz * jac * qq);
      }
    }
  }
}

}  // namespace

b200fmm_status upload_basis_constants(const Context &c, const double *roots, const double *Tr, const double *S) {
  const int p = c.p;
  if (p < 3 || p > kMaxOrder) return B200FMM_OK;  // no P2M / L2P kernel is built for this order
  const int lag = c.cfg.kernel == B200FMM_LAGRANGE ? 1 : 0;
  B200_CUDA(cudaMemcpyToSymbol(c_roots, roots, sizeof(double) * p,
                               sizeof(double) * ((size_t)(lag * (kMaxOrder - 2) + p - 3) * kMaxOrder)));
  // S [8 children][3 axes][p][p]: children 0 and 4 differ in the bit of axis 0
  const size_t table = sizeof(double) * kMaxOrder * kMaxOrder;
  for (int bit = 0; bit < 2; ++bit)
    B200_CUDA(cudaMemcpyToSymbol(c_S, S + (size_t)bit * 4 * 3 * p * p, sizeof(double) * p * p,
                                 table * ((lag * (kMaxOrder - 2) + p - 3) * 2 + bit)));
  if (!lag) B200_CUDA(cudaMemcpyToSymbol(c_Tr, Tr, sizeof(double) * p * p, table * (p - 3)));
  return B200FMM_OK;
}

b200fmm_status run_p2m(Context &c) {
  const int LL = c.H - 1;
  const Level &L = c.lv[LL];
  if (L.n == 0) return B200FMM_OK;
  const double W = c.cfg.box_width;
  const double x0 = c.cfg.center[0] - W / 2, y0 = c.cfg.center[1] - W / 2, z0 = c.cfg.center[2] - W / 2;
  const double lw = W / (double)(1 << LL);
  const bool lagr = c.cfg.kernel == B200FMM_LAGRANGE;
  unsigned long long *mmax = c.mmax_out ? c.mmax_out + (size_t)LL * kMmaxSlots : nullptr;
#define B200_P2M(PV)                                                                                        \
  case PV: {                                                                                                \
    auto kernel = lagr ? (c.R > 1 ? p2m_kernel<PV, true, 2> : p2m_kernel<PV, true, 1>)                      \
                       : (c.R > 1 ? p2m_kernel<PV, false, 2> : p2m_kernel<PV, false, 1>);                   \
    kernel<<<(unsigned)L.n, P2M_THREADS, 0, c.stream>>>(c.R, c.N, L.n, L.keys, c.d_leaf_start, c.d_x, c.d_y, c.d_z, \
                                                        c.d_q, x0, y0, z0, lw, L.M, mmax);                  \
    break;                                                                                                  \
  }
  switch (c.p) {
    B200_P2M(3) B200_P2M(4) B200_P2M(5) B200_P2M(6) B200_P2M(7) B200_P2M(8)
    default: return fail(B200FMM_ERR_UNSUPPORTED, "order not built");
  }
#undef B200_P2M
  ++c.launches;
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

b200fmm_status run_m2m(Context &c, int level) {
  if (level < 2 || level >= c.H - 1) return fail(B200FMM_ERR_INVALID, "m2m: parent level must be in [2, height-2]");
  const Level &P = c.lv[level], &C = c.lv[level + 1];
  if (P.n == 0) return B200FMM_OK;
  const bool lagr = c.cfg.kernel == B200FMM_LAGRANGE;
  unsigned long long *mmax = c.mmax_out ? c.mmax_out + (size_t)level * kMmaxSlots : nullptr;
#define B200_M2M(PV)                                                                                        \
  case PV: {                                                                                                \
    constexpr int sh = (int)sizeof(double) * 8 * Block<PV>::SIZE;                                           \
    auto kernel = lagr ? m2m_kernel<PV, true> : m2m_kernel<PV, false>;                                      \
    kernel<<<(unsigned)P.n, 256, sh, c.stream>>>(c.R, P.n, P.child, C.M, P.M, mmax);                        \
    break;                                                                                                  \
  }
  switch (c.p) {
    B200_M2M(3) B200_M2M(4) B200_M2M(5) B200_M2M(6) B200_M2M(7) B200_M2M(8)
    default: return fail(B200FMM_ERR_UNSUPPORTED, "order not built");
  }
#undef B200_M2M
  ++c.launches;
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

b200fmm_status run_l2l(Context &c, int level) {
  if (level < 2 || level >= c.H - 1) return fail(B200FMM_ERR_INVALID, "l2l: parent level must be in [2, height-2]");
  const Level &P = c.lv[level], &C = c.lv[level + 1];
  if (P.n == 0) return B200FMM_OK;
  const bool lagr = c.cfg.kernel == B200FMM_LAGRANGE;
#define B200_L2L(PV)                                                                                        \
  case PV: {                                                                                                \
    constexpr int sh = (int)sizeof(double) * 9 * Block<PV>::SIZE;                                           \
    auto kernel = lagr ? l2l_kernel<PV, true> : l2l_kernel<PV, false>;                                      \
    kernel<<<(unsigned)P.n, 256, sh, c.stream>>>(c.R, P.n, P.child, P.L, C.L);                              \
    break;                                                                                                  \
  }
  switch (c.p) {
    B200_L2L(3) B200_L2L(4) B200_L2L(5) B200_L2L(6) B200_L2L(7) B200_L2L(8)
    default: return fail(B200FMM_ERR_UNSUPPORTED, "order not built");
  }
#undef B200_L2L
  ++c.launches;
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

b200fmm_status run_l2p(Context &c, const long long *shard) {
  const int LL = c.H - 1;
  const Level &L = c.lv[LL];
  if (L.n == 0) return B200FMM_OK;
  const double W = c.cfg.box_width;
  const double x0 = c.cfg.center[0] - W / 2, y0 = c.cfg.center[1] - W / 2, z0 = c.cfg.center[2] - W / 2;
  const double lw = W / (double)(1 << LL);
  const bool lagr = c.cfg.kernel == B200FMM_LAGRANGE;
#define B200_L2P(PV)                                                                                         \
  case PV:                                                                                                   \
    if (lagr)                                                                                                \
      l2p_kernel<PV, true><<<grid_for(L.n, L2P_WARPS), L2P_WARPS * 32, 0, c.stream>>>(                      \
          c.R, c.N, L.n, L.keys, c.d_leaf_start, c.d_x, c.d_y, c.d_z, c.d_q, x0, y0, z0, lw, L.L, c.d_res,       \
          shard);                                                                                            \
    else                                                                                                     \
      l2p_kernel<PV, false><<<grid_for(L.n, L2P_WARPS), L2P_WARPS * 32, 0, c.stream>>>(                     \
          c.R, c.N, L.n, L.keys, c.d_leaf_start, c.d_x, c.d_y, c.d_z, c.d_q, x0, y0, z0, lw, L.L, c.d_res,       \
          shard);                                                                                            \
    break;
  switch (c.p) {
    B200_L2P(3) B200_L2P(4) B200_L2P(5) B200_L2P(6) B200_L2P(7) B200_L2P(8)
    default: return fail(B200FMM_ERR_UNSUPPORTED, "order not built");
  }
#undef B200_L2P
  ++c.launches;
  B200_CUDA(cudaGetLastError());
  return B200FMM_OK;
}

}  // namespace b200
