// Batched one-sided (Hestenes) Jacobi SVD in FP64: problems that fit one CTA's
// shared memory by a pivoted QR and Jacobi on its R (jacobi_qrp_kernel), the
// others by plain Jacobi in global memory (jacobi_solve), one CTA per problem
// or a cluster of CTAs per wide problem.
//
// Replaces the LAPACK dgesdd calls of hmat_lib (src/lapack_wrapper.c:8-59
// via src/constructors.c:323 for compression; src/hodlr_algebra.c:153 and
// :301 for recompression) on blocks small enough for one CTA.  Columns of the
// tall orientation are orthogonalised pairwise in round-robin order: each
// round pairs every column with one other (C/2 disjoint pairs, one warp per
// pair), so a sweep is C-1 rounds separated by barriers.  The singular
// values come out with high relative accuracy, so the relative truncation
// rule picks the same rank as the reference's dgesdd on its test matrices.
// Every loop is bounded: a problem that has not converged after max_sweeps
// sweeps still writes its outputs and raises SVD_FAILURE in the status word.
#include <algorithm>

#include <cooperative_groups.h>

#include "jacobi.h"

namespace cg = cooperative_groups;

namespace hb {

namespace {

constexpr int kJThreads = 256;
constexpr int kJCluster = 8;        // CTAs per problem cluster
constexpr int kJUnroll = 8;         // column elements per lane in flight in the pair loops

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Global loads and stores of G and W.  A problem solved by a cluster of CTAs
// reads columns that other CTAs of the cluster rotated in the previous round,
// so it bypasses L1 (cache-global) and relies on the cluster barrier's
// release / acquire ordering at L2.
template <bool kTeam>
__device__ __forceinline__ double gld(const double *p) {
  if constexpr (kTeam) return __ldcg(p);
  return *p;
}
template <bool kTeam>
__device__ __forceinline__ void gst(double *p, double v) {
  if constexpr (kTeam)
    __stcg(p, v);
  else
    *p = v;
}

template <bool kTeam>
__device__ __forceinline__ void team_sync() {
  if constexpr (kTeam)
    cg::this_cluster().sync();
  else
    __syncthreads();
}

// (x, y) <- (c x - s y, s x + c y) over `len` elements, the warp's lanes
// striding by 32, eight elements per lane in flight.
template <bool kTeam>
__device__ __forceinline__ void rotate_pair(double *xp, double *yp, int len, int lane, double cs,
                                            double sn) {
  for (int i0 = lane; i0 < len; i0 += 32 * kJUnroll) {
    double x[kJUnroll], y[kJUnroll];
#pragma unroll
    for (int u = 0; u < kJUnroll; ++u) {
      const int i = i0 + 32 * u;
      x[u] = i < len ? gld<kTeam>(xp + i) : 0.0;
      y[u] = i < len ? gld<kTeam>(yp + i) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kJUnroll; ++u) {
      const int i = i0 + 32 * u;
      if (i < len) {
        gst<kTeam>(xp + i, cs * x[u] - sn * y[u]);
        gst<kTeam>(yp + i, sn * x[u] + cs * y[u]);
      }
    }
  }
}

// One problem, by one CTA (kTeam false) or by the kJCluster CTAs of a
// cluster (kTeam true, `crank` = this CTA's rank in it): the disjoint pairs
// of a round are spread over every warp of the team, rounds are separated by
// a barrier of the team, and the team agrees on convergence through the
// CTAs' shared memory.  Every pair's arithmetic is the same in both modes.
template <bool kTeam>
__device__ void jacobi_solve(const JacobiProb &P, const JacobiParams &prm, int *status,
                             int crank, int team, const KernelSpec &gen) {
  const int m = P.m, n = P.n;
  const bool tall = m >= n;
  const int R = tall ? m : n, C = tall ? n : m;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  extern __shared__ double sh[];
  double *s_sig = sh;                              // C
  int *s_perm = reinterpret_cast<int *>(sh + C);   // C
  __shared__ double s_off[32];
  __shared__ double s_team_off;

  double *G = P.G, *W = P.W;
  const int gtid = crank * blockDim.x + tid, gthreads = team * blockDim.x;
  double fro2 = 0.0;   // this thread's share of ||A||_F^2
  for (long long e = gtid; e < (long long)R * C; e += gthreads) {
    const int r = (int)(e % R), c = (int)(e / R);
    // logical element (i, j) of the m x n input
    const int i = tall ? r : c, j = tall ? c : r;
    double a;
    if (P.gen_r0 >= 0)
      a = P.transA ? kernel_entry(gen, P.gen_r0 + j, P.gen_c0 + i)
                   : kernel_entry(gen, P.gen_r0 + i, P.gen_c0 + j);
    else
      a = P.transA ? P.A[j + (long long)i * P.lda] : P.A[i + (long long)j * P.lda];
    fro2 = fma(a, a, fro2);
    gst<kTeam>(G + e, a);
  }
  for (long long e = gtid; e < (long long)C * C; e += gthreads)
    gst<kTeam>(W + e, ((e % C) == (e / C)) ? 1.0 : 0.0);
  team_sync<kTeam>();

  // ||A||_F over the team
  fro2 = warp_sum(fro2);
  if (lane == 0) s_off[warp] = fro2;
  __syncthreads();
  double f2 = 0.0;
  for (int w = 0; w < nwarps; ++w) f2 += s_off[w];
  if constexpr (kTeam) {
    cg::cluster_group cl = cg::this_cluster();
    if (tid == 0) s_team_off = f2;
    cl.sync();
    f2 = 0.0;
    for (int rk = 0; rk < team; ++rk) f2 += *cl.map_shared_rank(&s_team_off, rk);
    cl.sync();
  }
  __syncthreads();
  // Pairs with a column of norm below theta are neither rotated nor tested:
  // all such columns together hold at most sqrt(C) theta = 1e-3 tol s_0 of the
  // matrix (||A||_F / C <= s_0 / sqrt(C) for the relative rule), so no
  // singular value moves by more than 0.1% of the truncation threshold
  // (Weyl) and none of theirs reaches it.  Columns at rounding level otherwise
  // keep the sweeps going: their computed cosines with any column are
  // rounding noise.  No skipping when every singular value is kept.
  double theta = 0.0;
  if (prm.trunc == Truncation::Relative)
    theta = 1e-3 * prm.tol * sqrt(f2) / C;
  else if (prm.trunc == Truncation::Absolute)
    theta = 1e-3 * prm.tol / sqrt((double)C);
  theta = fmax(theta, P.skip_abs);
  const double skip2 = theta * theta;
  const double cscale = P.conv_scale > 0.0 ? P.conv_scale : (prm.norm_stop ? sqrt(f2) : 0.0);

  // a computed dot product of length R carries ~sqrt(R) eps relative noise:
  // below that no rotation can make progress
  const double conv = fmax(prm.conv_tol, 4.0 * sqrt((double)R) * 2.220446049250313e-16);
  const int players = C + (C & 1);
  const int gwarp = crank * nwarps + warp, gwarps = team * nwarps;
  int sweep = 0;
  bool converged = (C == 1);
  for (; sweep < prm.max_sweeps && !converged; ++sweep) {
    double off = 0.0;
    for (int r = 0; r < players - 1; ++r) {
      for (int k = gwarp; k < players / 2; k += gwarps) {
        int a, b;
        if (k == 0) {
          a = r;
          b = players - 1;
        } else {
          a = (r + k) % (players - 1);
          b = (r - k + (players - 1)) % (players - 1);
        }
        if (a >= C || b >= C) continue;
        const int p = min(a, b), q = max(a, b);
        double *gp = G + (long long)p * R, *gq = G + (long long)q * R;
        // eight elements per lane in flight, the last chunk predicated (each
        // sum keeps the element order of a plain loop: arithmetic unchanged)
        double al = 0.0, be = 0.0, ga = 0.0;
        for (int i0 = lane; i0 < R; i0 += 32 * kJUnroll) {
          double x[kJUnroll], y[kJUnroll];
#pragma unroll
          for (int u = 0; u < kJUnroll; ++u) {
            const int i = i0 + 32 * u;
            x[u] = i < R ? gld<kTeam>(gp + i) : 0.0;
            y[u] = i < R ? gld<kTeam>(gq + i) : 0.0;
          }
#pragma unroll
          for (int u = 0; u < kJUnroll; ++u)
            if (i0 + 32 * u < R) {
              al = fma(x[u], x[u], al);
              be = fma(y[u], y[u], be);
              ga = fma(x[u], y[u], ga);
            }
        }
        al = warp_sum(al);
        be = warp_sum(be);
        ga = warp_sum(ga);
        if (ga == 0.0 || al <= 0.0 || be <= 0.0) continue;
        if (al <= skip2 || be <= skip2) continue;
        double rel = fabs(ga) / (sqrt(al) * sqrt(be));
        // coupling at rounding level of the problem's own scale (a block of a
        // larger matrix, whose columns were recomputed by a GEMM) counts as
        // converged: it moves no singular value by more than that level
        if (cscale > 0.0) rel = fmin(rel, fabs(ga) / (cscale * fmax(sqrt(al), sqrt(be))));
        off = fmax(off, rel);
        if (rel <= conv) continue;
        const double zeta = (be - al) / (2.0 * ga);
        // tan of the rotation angle; for |zeta| beyond 1e100 zeta^2 would
        // overflow and the exact value is 1 / (2 zeta) to double precision
        const double t = fabs(zeta) > 1e100
                             ? 0.5 / zeta
                             : (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
        const double cs = 1.0 / sqrt(1.0 + t * t), sn = cs * t;
        rotate_pair<kTeam>(gp, gq, R, lane, cs, sn);
        rotate_pair<kTeam>(W + (long long)p * C, W + (long long)q * C, C, lane, cs, sn);
      }
      team_sync<kTeam>();
    }
    // team-wide max of `off`
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) off = fmax(off, __shfl_xor_sync(0xffffffffu, off, o));
    if (lane == 0) s_off[warp] = off;
    __syncthreads();
    double mx = 0.0;
    for (int w = 0; w < nwarps; ++w) mx = fmax(mx, s_off[w]);
    if constexpr (kTeam) {
      // every CTA reads every CTA's maximum, so all take the same decision;
      // the second barrier keeps every CTA (and its shared memory) alive and
      // unchanged until all reads are done
      cg::cluster_group cl = cg::this_cluster();
      if (tid == 0) s_team_off = mx;
      cl.sync();
      mx = 0.0;
      for (int rk = 0; rk < team; ++rk) mx = fmax(mx, *cl.map_shared_rank(&s_team_off, rk));
      cl.sync();
    }
    converged = mx <= conv;
    __syncthreads();
  }
  if (crank != 0) return;
  if (!converged && tid == 0) atomicExch(status, (int)SVD_FAILURE);
  if (tid == 0 && P.sweeps) *P.sweeps = converged ? sweep : prm.max_sweeps + 1;

  // singular values = column norms of G
  for (int j = warp; j < C; j += nwarps) {
    const double *gj = G + (long long)j * R;
    double s = 0.0;
    for (int i = lane; i < R; i += 32) {
      const double x = gld<kTeam>(gj + i);
      s = fma(x, x, s);
    }
    s = warp_sum(s);
    if (lane == 0) s_sig[j] = sqrt(s);
  }
  __syncthreads();
  // descending order, ties by index (stable)
  for (int j = tid; j < C; j += blockDim.x) {
    const double sj = s_sig[j];
    int pos = 0;
    for (int i = 0; i < C; ++i) {
      const double si = s_sig[i];
      pos += (si > sj) || (si == sj && i < j);
    }
    s_perm[pos] = j;
  }
  __syncthreads();
  if (tid == 0) {
    const double s0 = s_sig[s_perm[0]];
    int k = 1;
    if (prm.trunc == Truncation::Relative) {
      if (s0 > prm.tol)
        while (k < C && s_sig[s_perm[k]] >= prm.tol * s0) ++k;
    } else if (prm.trunc == Truncation::Absolute) {
      while (k < C && s_sig[s_perm[k]] > prm.tol) ++k;
    } else {
      k = C;
    }
    if (P.rank) *P.rank = k;
  }
  for (int k = tid; k < C; k += blockDim.x)
    if (P.sigma) P.sigma[k] = s_sig[s_perm[k]];
  // outputs, one warp per column
  for (int k = warp; k < C; k += nwarps) {
    const int j = s_perm[k];
    const double sg = s_sig[j];
    const double *gj = G + (long long)j * R;
    const double *wj = W + (long long)j * C;
    double *u = P.U + (long long)k * P.ldu;
    double *v = P.V + (long long)k * P.ldv;
    if (tall) {  // A = (G / sigma) Sigma W^T
      for (int i = lane; i < m; i += 32) {
        double x = gld<kTeam>(gj + i);
        if (!prm.scale_u) x = sg > 0.0 ? x / sg : (i == k % m ? 1.0 : 0.0);
        u[i] = x;
      }
      for (int i = lane; i < n; i += 32) v[i] = gld<kTeam>(wj + i);
    } else {     // A^T = (G / sigma) Sigma W^T  =>  A = W Sigma (G / sigma)^T
      for (int i = lane; i < m; i += 32) {
        const double x = gld<kTeam>(wj + i);
        u[i] = prm.scale_u ? x * sg : x;
      }
      for (int i = lane; i < n; i += 32) {
        const double x = gld<kTeam>(gj + i);
        v[i] = sg > 0.0 ? x / sg : (i == k % n ? 1.0 : 0.0);
      }
    }
  }
}

// One CTA per problem.
__global__ void __launch_bounds__(kJThreads)
jacobi_svd_kernel(const JacobiProb *__restrict__ probs, JacobiParams prm, int *status,
                  KernelSpec gen) {
  const JacobiProb P = probs[blockIdx.x];
  const int C = P.m < P.n ? P.m : P.n;
  if (C == 0) {
    if (threadIdx.x == 0 && P.rank) *P.rank = 0;
    return;
  }
  jacobi_solve<false>(P, prm, status, 0, 1, gen);
}

// A cluster of kJCluster CTAs per problem; problems with at least
// `team_min_c` columns are solved by the whole cluster, the others by its
// first CTA alone (the rest return at once, before any cluster barrier).
__global__ void __cluster_dims__(kJCluster, 1, 1) __launch_bounds__(kJThreads)
jacobi_svd_cluster_kernel(const JacobiProb *__restrict__ probs, JacobiParams prm, int *status,
                          int team_min_c, KernelSpec gen) {
  const int crank = (int)cg::this_cluster().block_rank();
  const JacobiProb P = probs[blockIdx.x / kJCluster];
  const int C = P.m < P.n ? P.m : P.n;
  if (C == 0) {
    if (crank == 0 && threadIdx.x == 0 && P.rank) *P.rank = 0;
    return;
  }
  if (C >= team_min_c) {
    jacobi_solve<true>(P, prm, status, crank, kJCluster, gen);
  } else {
    if (crank != 0) return;
    jacobi_solve<false>(P, prm, status, 0, 1, gen);
  }
}

// ---- problems that fit one CTA's shared memory ------------------------------------
//
// One CTA per problem: pivoted QR first, Jacobi on the few rows of R that
// matter, everything in shared memory.  With T the tall orientation (R x C):
//   1. T P = Q Rf by Householder reflections with column pivoting, stopped
//      after k steps when the columns left hold at most 1e-3 tol s_0 in the
//      Frobenius norm (s_0 bounded below by the largest column and the first
//      row of Rf): no kept singular value moves by more than 0.1% of the
//      truncation threshold (Weyl), the bound that the skip rule of
//      jacobi_solve states for the columns it leaves alone.  Norms of the
//      remaining columns are recomputed in the pass that updates them.
//   2. one-sided Jacobi on the k columns of X = P Rf^T (C x k), rotations
//      accumulated in W (k x k): X W = G, so T = (Q W) G^T.  Columns of Rf^T
//      are graded and nearly orthogonal (Drmac and Veselic, SIAM J. Matrix
//      Anal. Appl. 29, 2008, use the same preconditioning), which takes 5 to
//      8 sweeps of k - 1 rounds instead of 25 to 35 sweeps of C - 1.
//   3. one side's vectors are G / sigma, the other's the reflections applied
//      to W's columns.
// Every pass over columns gives eight lanes a column (or a pair of columns):
// 16-byte accesses, one 128-byte row of banks per eight lanes, the values held
// in registers between the dot products and the update.  The QR is bound by
// the latency of its steps, a Jacobi round by shared-memory bandwidth (k (C +
// k) values read and written).  W moves to global memory when X and W do not
// fit together.
// 256 blocks of 128 x 128 (n = 32768, 2D Matern-3/2, tol 1e-8, k about 60):
// 55 ms by jacobi_solve (two passes over 128 columns a round, 29 sweeps),
// 3.6 ms so; 64 blocks of the 3D exponential kernel (k about 118): 48 -> 6.6 ms.
constexpr int kQrpThreads = 512;
constexpr int kQrpMaxDim = 176;          // 11 chunks of 16 rows per eight lanes
constexpr size_t kQrpSmem = 227 * 1024;  // shared memory of one CTA
constexpr int kQrpArrays = 8;            // C-long arrays beside the matrices (doubles)

__host__ __device__ inline int pad16(int x) { return (x + 15) & ~15; }

// Bytes that a problem needs at least (its matrix), and the most it can use
// (X and W of full rank).
inline size_t qrp_smem_min(int R, int C) {
  return sizeof(double) * ((size_t)pad16(R) * C + kQrpArrays * (size_t)pad16(C));
}
inline size_t qrp_smem_max(int R, int C) {
  return sizeof(double) *
         ((size_t)pad16(R) * C + (size_t)pad16(C) * C + kQrpArrays * (size_t)pad16(C));
}

__device__ __forceinline__ double group_sum(double v) {   // over the eight lanes of a column
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v + __shfl_xor_sync(0xffffffffu, v, 4);
}

template <int NC>
__global__ void __launch_bounds__(kQrpThreads, 1)
jacobi_qrp_kernel(const JacobiProb *__restrict__ probs, JacobiParams prm, int *status,
                  int smem_doubles, KernelSpec gen) {
  extern __shared__ __align__(16) double sh[];
  __shared__ double s_red[kQrpThreads / 32];
  const JacobiProb P = probs[blockIdx.x];
  const int m = P.m, n = P.n;
  const bool tall = m >= n;
  const int R = tall ? m : n, C = tall ? n : m;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarps = kQrpThreads / 32, kGroups = kQrpThreads / 8;
  if (C == 0) {
    if (tid == 0 && P.rank) *P.rank = 0;
    return;
  }
  const int grp = tid >> 3, gl = tid & 7;      // column group, lane within it
  const int lda = pad16(R), Cp = pad16(C);
  double *norms = sh;                          // 2 x Cp: squared norms left, by parity
  double *hh = sh + 2 * Cp;                    // 2 / ||v_j||^2
  double *vd = hh + Cp;                        // v_j's first entry
  double *rd = vd + Cp;                        // diagonal of Rf
  double *sig = rd + Cp;                       // singular values
  int *order = reinterpret_cast<int *>(sig + Cp);   // pivot column of step j
  int *perm = order + Cp;
  double *A = sh + kQrpArrays * Cp;            // 16-byte aligned: Cp is a multiple of 16
  const int mat_doubles = smem_doubles - kQrpArrays * Cp;

  // ---- load T, rows past R zero -------------------------------------------------------
  double amax = 0.0;
  auto entry = [&](int r, int c) {
    const int i = tall ? r : c, j = tall ? c : r;
    if (P.gen_r0 >= 0)
      return P.transA ? kernel_entry(gen, P.gen_r0 + j, P.gen_c0 + i)
                      : kernel_entry(gen, P.gen_r0 + i, P.gen_c0 + j);
    return P.transA ? P.A[j + (long long)i * P.lda] : P.A[i + (long long)j * P.lda];
  };
  if (tall != (P.transA != 0)) {               // T's columns are contiguous in memory
    for (int c = warp; c < C; c += kWarps)
      for (int r = lane; r < lda; r += 32) {
        const double a = r < R ? entry(r, c) : 0.0;
        amax = fmax(amax, fabs(a));
        A[r + c * lda] = a;
      }
  } else {
    for (int r = warp; r < lda; r += kWarps)
      for (int c = lane; c < C; c += 32) {
        const double a = r < R ? entry(r, c) : 0.0;
        amax = fmax(amax, fabs(a));
        A[r + c * lda] = a;
      }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (lane == 0) s_red[warp] = amax;
  __syncthreads();
  for (int w = 0; w < kWarps; ++w) amax = fmax(amax, s_red[w]);
  // entries whose squares would leave the range of a double: work on a power
  // of two times T
  double scale = 1.0;
  if ((amax > 0.0 && amax < 1e-100) || (amax > 1e100 && amax < 1.8e308))
    scale = scalbn(1.0, max(-1000, min(1000, -ilogb(amax))));

  // squared column norms; a group's share of a column is rows 16 i + 2 gl, + 1
  const int nch = lda / 16;
  for (int c0 = 0; c0 < C; c0 += kGroups) {
    const int c = c0 + grp;
    double s = 0.0;
    if (c < C)
      for (int i = 0; i < nch; ++i) {
        double2 &a = *reinterpret_cast<double2 *>(A + c * lda + 16 * i + 2 * gl);
        if (scale != 1.0) a = make_double2(scale * a.x, scale * a.y);
        s = fma(a.x, a.x, fma(a.y, a.y, s));
      }
    s = group_sum(s);
    if (c < C && gl == 0) norms[c] = s;
  }
  __syncthreads();
  double f2 = 0.0;
  for (int c = lane; c < C; c += 32) f2 += norms[c];
  f2 = warp_sum(f2);                           // ||T||_F^2
  const double tol_abs = prm.tol * scale;

  // ---- 1. QR with column pivoting ------------------------------------------------------
  int k = 0;
  double s0sq = 0.0;                           // lower bound of s_0^2
  for (int j = 0; j < C; ++j) {
    const double *nr = norms + (j & 1) * Cp;
    double *nw = norms + ((j + 1) & 1) * Cp;
    // pivot: the largest norm to 12 bits (upper word of the square, its low
    // byte replaced by the column), the same choice in every warp
    unsigned key = 0;
    for (int c = lane; c < C; c += 32) {
      const double v = nr[c];
      if (!(v < 0.0))
        key = max(key, (((unsigned)__double2hiint(v) & 0x7fffff00u) | (unsigned)c));
    }
    key = __reduce_max_sync(0xffffffffu, key);
    const int p = (int)(key & 0xffu);
    const double n2 = nr[p];
    // columns left hold at most (C - j) n2 (1 + 2^-11) of the square
    double lim = 0.0;
    if (prm.trunc == Truncation::Relative)
      lim = 1e-6 * prm.tol * prm.tol * s0sq;
    else if (prm.trunc == Truncation::Absolute)
      lim = 1e-6 * tol_abs * tol_abs;
    if (n2 < 1e-300 || 1.001 * (C - j) * n2 <= lim) break;   // not on a NaN
    const double alpha = A[j + p * lda];
    const double nrm = sqrt(n2);
    const double beta = alpha >= 0.0 ? -nrm : nrm;
    const double h = 1.0 / (beta * (beta - alpha));
    double2 v[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int r = 16 * i + 2 * gl;
      v[i] = make_double2(0.0, 0.0);
      if (i < nch && r + 1 >= j) {
        v[i] = *reinterpret_cast<const double2 *>(A + p * lda + r);
        if (r <= j) v[i].x = r == j ? alpha - beta : 0.0;
        if (r + 1 == j) v[i].y = alpha - beta;
      }
    }
    for (int c0 = 0; c0 < C; c0 += kGroups) {
      const int c = c0 + grp;
      const bool live = c < C && c != p && !(nr[c] < 0.0);
      double2 a[NC];
      double dot = 0.0, s = 0.0;
      if (live) {
#pragma unroll
        for (int i = 0; i < NC; ++i)
          if (i < nch && 16 * i + 15 >= j) {
            a[i] = *reinterpret_cast<const double2 *>(A + c * lda + 16 * i + 2 * gl);
            dot = fma(v[i].x, a[i].x, fma(v[i].y, a[i].y, dot));
          }
      }
      dot = -h * group_sum(dot);
      if (live) {
#pragma unroll
        for (int i = 0; i < NC; ++i)
          if (i < nch && 16 * i + 15 >= j) {
            const int r = 16 * i + 2 * gl;
            a[i].x = fma(dot, v[i].x, a[i].x);
            a[i].y = fma(dot, v[i].y, a[i].y);
            *reinterpret_cast<double2 *>(A + c * lda + r) = a[i];
            if (r > j) s = fma(a[i].x, a[i].x, s);
            if (r + 1 > j) s = fma(a[i].y, a[i].y, s);
          }
      }
      s = group_sum(s);
      if (c < C && gl == 0) nw[c] = live ? s : -1.0;
    }
    if (tid == 0) {
      order[j] = p;
      hh[j] = h;
      vd[j] = alpha - beta;
      rd[j] = beta;
    }
    __syncthreads();
    if (j == 0) {
      double s = 0.0;                          // first row of Rf (column p holds alpha)
      for (int c = lane; c < C; c += 32)
        if (c != p) s = fma(A[c * lda], A[c * lda], s);
      s0sq = n2 + warp_sum(s);
    }
    k = j + 1;
  }
  __syncthreads();

  // ---- reflectors to P.G (R x k), X staged through P.W (C x k) -------------------------
  // Rf's rows change sign so that its diagonal is positive (Q's columns with
  // them): a block with one entry keeps that entry's sign in U
  for (int j = warp; j < k; j += kWarps) {
    const double *col = A + order[j] * lda;
    for (int r = lane; r < R; r += 32)
      P.G[r + (long long)j * R] = r < j ? 0.0 : r == j ? vd[j] : col[r];
  }
  for (int i = tid; i < C; i += kQrpThreads) perm[i] = C;   // step of column i, C: none
  __syncthreads();
  for (int j = tid; j < k; j += kQrpThreads) perm[order[j]] = j;
  __syncthreads();
  for (int c = warp; c < C; c += kWarps) {
    const int step = perm[c];
    for (int j = lane; j < k; j += 32) {
      const double x = j < step ? A[j + c * lda] : j == step ? rd[j] : 0.0;
      P.W[c + (long long)j * C] = rd[j] < 0.0 ? -x : x;
    }
  }
  __syncthreads();
  const int ldw = pad16(k);
  double *X = A;                               // Cp x k
  double *Ws = A + (long long)lda * k;         // ldw x k, if it fits
  const bool w_sh = (long long)(lda + ldw) * k <= mat_doubles;
  for (int j = warp; j < k; j += kWarps)
    for (int c = lane; c < Cp; c += 32)
      X[c + j * Cp] = c < C ? P.W[c + (long long)j * C] : 0.0;
  __syncthreads();
  if (w_sh) {
    for (int e = tid; e < ldw * k; e += kQrpThreads) Ws[e] = (e % ldw == e / ldw) ? 1.0 : 0.0;
  } else {
    for (int e = tid; e < k * k; e += kQrpThreads)
      P.W[(e % k) + (long long)(e / k) * C] = (e % k == e / k) ? 1.0 : 0.0;
  }
  __syncthreads();

  // ---- 2. one-sided Jacobi on X's columns (tests of jacobi_solve) ------------------------
  double theta = 0.0;
  if (prm.trunc == Truncation::Relative)
    theta = 1e-3 * prm.tol * sqrt(f2) / C;
  else if (prm.trunc == Truncation::Absolute)
    theta = 1e-3 * tol_abs / sqrt((double)C);
  theta = fmax(theta, P.skip_abs * scale);
  const double skip2 = theta * theta;
  const double cscale = P.conv_scale > 0.0 ? P.conv_scale * scale : (prm.norm_stop ? sqrt(f2) : 0.0);
  const double conv = fmax(prm.conv_tol, 4.0 * sqrt((double)R) * 2.220446049250313e-16);
  const int players = k + (k & 1), npairs = players / 2;
  const int nchx = Cp / 16, nchw = ldw / 16;
  int sweep = 0;
  bool converged = k <= 1;
  for (; sweep < prm.max_sweeps && !converged; ++sweep) {
    double off = 0.0;
    for (int r = 0; r < players - 1; ++r) {
      for (int q0 = 0; q0 < npairs; q0 += kGroups) {
        const int pi = q0 + grp;
        int a = 0, b = 0;
        bool live = pi < npairs;
        if (live) {
          if (pi == 0) {
            a = r;
            b = players - 1;
          } else {
            a = r + pi;
            if (a >= players - 1) a -= players - 1;
            b = r - pi;
            if (b < 0) b += players - 1;
          }
          live = a < k && b < k;
        }
        const int p = min(a, b), q = max(a, b);
        double2 x[NC], y[NC];
        double al = 0.0, be = 0.0, ga = 0.0;
        if (live) {
#pragma unroll
          for (int i = 0; i < NC; ++i)
            if (i < nchx) {
              x[i] = *reinterpret_cast<const double2 *>(X + p * Cp + 16 * i + 2 * gl);
              y[i] = *reinterpret_cast<const double2 *>(X + q * Cp + 16 * i + 2 * gl);
              al = fma(x[i].x, x[i].x, fma(x[i].y, x[i].y, al));
              be = fma(y[i].x, y[i].x, fma(y[i].y, y[i].y, be));
              ga = fma(x[i].x, y[i].x, fma(x[i].y, y[i].y, ga));
            }
        }
        al = group_sum(al);
        be = group_sum(be);
        ga = group_sum(ga);
        if (!live || ga == 0.0 || al <= 0.0 || be <= 0.0 || al <= skip2 || be <= skip2) continue;
        double rel = fabs(ga) / (sqrt(al) * sqrt(be));
        if (cscale > 0.0) rel = fmin(rel, fabs(ga) / (cscale * fmax(sqrt(al), sqrt(be))));
        off = fmax(off, rel);
        if (rel <= conv) continue;
        const double zeta = (be - al) / (2.0 * ga);
        const double t = fabs(zeta) > 1e100
                             ? 0.5 / zeta
                             : (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
        const double cs = 1.0 / sqrt(1.0 + t * t), sn = cs * t;
#pragma unroll
        for (int i = 0; i < NC; ++i)
          if (i < nchx) {
            const int o = 16 * i + 2 * gl;
            *reinterpret_cast<double2 *>(X + p * Cp + o) =
                make_double2(cs * x[i].x - sn * y[i].x, cs * x[i].y - sn * y[i].y);
            *reinterpret_cast<double2 *>(X + q * Cp + o) =
                make_double2(sn * x[i].x + cs * y[i].x, sn * x[i].y + cs * y[i].y);
          }
        if (w_sh) {
#pragma unroll
          for (int i = 0; i < NC; ++i)
            if (i < nchw) {
              const int o = 16 * i + 2 * gl;
              double2 &wp = *reinterpret_cast<double2 *>(Ws + p * ldw + o);
              double2 &wq = *reinterpret_cast<double2 *>(Ws + q * ldw + o);
              const double2 u = wp, z = wq;
              wp = make_double2(cs * u.x - sn * z.x, cs * u.y - sn * z.y);
              wq = make_double2(sn * u.x + cs * z.x, sn * u.y + cs * z.y);
            }
        } else {
          double *wp = P.W + (long long)p * C, *wq = P.W + (long long)q * C;
          double u[2 * NC], z[2 * NC];
#pragma unroll
          for (int i = 0; i < 2 * NC; ++i) {
            const int o = 8 * i + gl;
            u[i] = o < k ? wp[o] : 0.0;
            z[i] = o < k ? wq[o] : 0.0;
          }
#pragma unroll
          for (int i = 0; i < 2 * NC; ++i) {
            const int o = 8 * i + gl;
            if (o < k) {
              wp[o] = cs * u[i] - sn * z[i];
              wq[o] = sn * u[i] + cs * z[i];
            }
          }
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) off = fmax(off, __shfl_xor_sync(0xffffffffu, off, o));
    if (lane == 0) s_red[warp] = off;
    __syncthreads();
    double mx = 0.0;
    for (int w = 0; w < kWarps; ++w) mx = fmax(mx, s_red[w]);
    converged = mx <= conv;
    __syncthreads();
  }
  if (tid == 0) {
    if (!converged) atomicExch(status, (int)SVD_FAILURE);
    if (P.sweeps) *P.sweeps = converged ? sweep : prm.max_sweeps + 1;
  }

  // ---- singular values in descending order (ties by index), rank -----------------------
  const double inv = 1.0 / scale;
  for (int c0 = 0; c0 < C; c0 += kGroups) {
    const int c = c0 + grp;
    double s = 0.0;
    if (c < k)
      for (int i = 0; i < nchx; ++i) {
        const double2 a = *reinterpret_cast<const double2 *>(X + c * Cp + 16 * i + 2 * gl);
        s = fma(a.x, a.x, fma(a.y, a.y, s));
      }
    s = group_sum(s);
    if (c < C && gl == 0) sig[c] = sqrt(s) * inv;
  }
  __syncthreads();
  for (int c = tid; c < C; c += kQrpThreads) {
    const double sc = sig[c];
    int pos = 0;
    for (int i = 0; i < C; ++i) pos += (sig[i] > sc) || (sig[i] == sc && i < c);
    perm[pos] = c;
  }
  __syncthreads();
  int rank = 1;
  {
    const double s0 = sig[perm[0]];
    if (prm.trunc == Truncation::Relative) {
      if (s0 > prm.tol)
        while (rank < C && sig[perm[rank]] >= prm.tol * s0) ++rank;
    } else if (prm.trunc == Truncation::Absolute) {
      while (rank < C && sig[perm[rank]] > prm.tol) ++rank;
    } else {
      rank = C;
    }
  }
  if (tid == 0 && P.rank) *P.rank = rank;
  for (int i = tid; i < C; i += kQrpThreads)
    if (P.sigma) P.sigma[i] = sig[perm[i]];

  // ---- 3. vectors of the first `rank` singular values ------------------------------------
  // the C side: G / sigma (sigma carried when it is U, scaled)
  const bool c_scaled = !tall && prm.scale_u;
  for (int i = warp; i < rank; i += kWarps) {
    const int j = perm[i];
    const double sg = sig[j];
    double *out = tall ? P.V + (long long)i * P.ldv : P.U + (long long)i * P.ldu;
    for (int c = lane; c < C; c += 32) {
      const double x = j < k ? inv * X[c + j * Cp] : 0.0;
      out[c] = c_scaled ? x : (sg > 0.0 ? x / sg : (c == i % C ? 1.0 : 0.0));
    }
  }
  // the R side: the reflections, last first, applied to W's columns (signs of
  // Rf's rows included), eight lanes per column; the reflectors come back from
  // P.G into X's place (and W's: W is in registers by then)
  constexpr int kMaxPass = (kQrpMaxDim + kGroups - 1) / kGroups;
  const bool r_scaled = tall && prm.scale_u;
  double2 yv[NC];
  for (int pass = 0; pass < kMaxPass; ++pass) {
    if (pass * kGroups >= rank) break;         // uniform
    const int i = pass * kGroups + grp;
    const int j = i < rank ? perm[i] : C;
    __syncthreads();                           // X (or the last pass) is read no more
#pragma unroll
    for (int u = 0; u < NC; ++u) {
      const int r = 16 * u + 2 * gl;
      double e[2] = {0.0, 0.0};
#pragma unroll
      for (int z = 0; z < 2; ++z)
        if (j < k && r + z < k) {
          const double w = w_sh ? Ws[(r + z) + j * ldw] : P.W[(r + z) + (long long)j * C];
          e[z] = rd[r + z] < 0.0 ? -w : w;
        }
      yv[u] = make_double2(e[0], e[1]);
    }
    if (pass == 0) {
      // X is free now; W's shared copy starts past lda k doubles
      for (int jj = warp; jj < k; jj += kWarps)
        for (int r = lane; r < lda; r += 32)
          A[r + jj * lda] = r < R ? P.G[r + (long long)jj * R] : 0.0;
      __syncthreads();
    }
    for (int jj = k - 1; jj >= 0; --jj) {
      double2 v[NC];
      double dot = 0.0;
#pragma unroll
      for (int u = 0; u < NC; ++u)
        if (u < nch && 16 * u + 15 >= jj) {
          v[u] = *reinterpret_cast<const double2 *>(A + jj * lda + 16 * u + 2 * gl);
          dot = fma(v[u].x, yv[u].x, fma(v[u].y, yv[u].y, dot));
        }
      dot = -hh[jj] * group_sum(dot);
#pragma unroll
      for (int u = 0; u < NC; ++u)
        if (u < nch && 16 * u + 15 >= jj) {
          yv[u].x = fma(dot, v[u].x, yv[u].x);
          yv[u].y = fma(dot, v[u].y, yv[u].y);
        }
    }
    if (i < rank) {
      const double sg = r_scaled ? sig[j] : 1.0;
      double *out = tall ? P.U + (long long)i * P.ldu : P.V + (long long)i * P.ldv;
#pragma unroll
      for (int u = 0; u < NC; ++u) {
        const int r = 16 * u + 2 * gl;
        if (j >= k) yv[u] = make_double2(r == i % R ? 1.0 : 0.0, r + 1 == i % R ? 1.0 : 0.0);
        if (r < R) out[r] = sg * yv[u].x;
        if (r + 1 < R) out[r + 1] = sg * yv[u].y;
      }
    }
  }
}

// dst (+)= src for every descriptor: CTAs take columns, threads rows (no
// division per element).
template <bool kAdd>
__global__ void copy2d_kernel(const CopyDesc *__restrict__ descs) {
  const CopyDesc D = descs[blockIdx.y];
  for (int c = blockIdx.x; c < D.cols; c += gridDim.x) {
    const double *src = D.src + (long long)c * D.lds;
    double *dst = D.dst + (long long)c * D.ldd;
    for (int r = threadIdx.x; r < D.rows; r += blockDim.x) dst[r] = kAdd ? dst[r] + src[r] : src[r];
  }
}

template <bool kAdd>
void run_copies2d(const std::vector<CopyDesc> &descs, cudaStream_t stream) {
  if (descs.empty()) return;
  int cols = 1;
  for (const CopyDesc &d : descs) cols = std::max(cols, d.cols);
  CopyDesc *d = nullptr;
  pool_alloc(&d, sizeof(CopyDesc) * descs.size(), stream);
  h2d_async(d, descs.data(), sizeof(CopyDesc) * descs.size(), stream);
  for (size_t off = 0; off < descs.size(); off += 65535) {
    dim3 grid((unsigned)std::min(cols, 32), (unsigned)std::min<size_t>(65535, descs.size() - off));
    copy2d_kernel<kAdd><<<grid, 256, 0, stream>>>(d + off);
    HB_LAUNCHED();
  }
  cudaFreeAsync(d, stream);
}

}  // namespace

namespace {

template <int NC>
void launch_qrp(const JacobiProb *d_probs, int nprobs, const JacobiParams &prm, int *d_status,
                size_t smem, cudaStream_t stream, const KernelSpec &gen) {
  // one value for every launch: the attribute is shared by all threads
  HB_CUDA(cudaFuncSetAttribute(jacobi_qrp_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(kQrpSmem - 512)));
  jacobi_qrp_kernel<NC><<<nprobs, kQrpThreads, smem, stream>>>(
      d_probs, prm, d_status, (int)(smem / sizeof(double)), gen);
  HB_LAUNCHED();
}

// Problems past the shared-memory kernel's sizes: a cluster of CTAs each when
// the widest reaches team_min_c columns, else one CTA each.
void launch_general(const JacobiProb *d_probs, int nprobs, const JacobiParams &prm, int *d_status,
                    int max_c, cudaStream_t stream, const KernelSpec &gen) {
  const size_t smem = (size_t)std::max(max_c, 1) * (sizeof(double) + sizeof(int));
  HB_REQUIRE(smem <= 200 * 1024, INPUT_ERROR, "Jacobi SVD problem too wide for one CTA");
  const int team_min_c = (int)std::min(option("jacobi_cluster_min_c", 192.0), 1e9);
  if (max_c >= team_min_c) {
    if (smem > 48 * 1024)
      HB_CUDA(cudaFuncSetAttribute(jacobi_svd_cluster_kernel,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    jacobi_svd_cluster_kernel<<<nprobs * kJCluster, kJThreads, smem, stream>>>(
        d_probs, prm, d_status, team_min_c, gen);
  } else {
    if (smem > 48 * 1024)
      HB_CUDA(cudaFuncSetAttribute(jacobi_svd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
    jacobi_svd_kernel<<<nprobs, kJThreads, smem, stream>>>(d_probs, prm, d_status, gen);
  }
  HB_LAUNCHED();
}

}  // namespace

void jacobi_svd_batched(const std::vector<JacobiProb> &probs, const JacobiParams &prm,
                        int *d_status, cudaStream_t stream, const KernelSpec &gen) {
  if (probs.empty()) return;
  // problems whose matrix fits one CTA's shared memory first, the rest after
  std::vector<JacobiProb> list;
  list.reserve(probs.size());
  auto fits = [](const JacobiProb &p) {
    const int R = std::max(p.m, p.n), C = std::min(p.m, p.n);
    return R <= kQrpMaxDim && qrp_smem_min(R, C) <= kQrpSmem - 512;
  };
  int small_r = 1, large_c = 1;
  size_t smem = 0;
  for (const JacobiProb &p : probs)
    if (fits(p)) {
      const int R = std::max(p.m, p.n), C = std::min(p.m, p.n);
      small_r = std::max(small_r, R);
      smem = std::max(smem, std::min(qrp_smem_max(R, C), kQrpSmem - 512));
      list.push_back(p);
    }
  const int nsmall = (int)list.size();
  for (const JacobiProb &p : probs)
    if (!fits(p)) {
      large_c = std::max(large_c, std::min(p.m, p.n));
      list.push_back(p);
    }
  JacobiProb *d = nullptr;
  pool_alloc(&d, sizeof(JacobiProb) * list.size(), stream);
  h2d_async(d, list.data(), sizeof(JacobiProb) * list.size(), stream);
  if (nsmall > 0) {
    if (small_r <= 128)
      launch_qrp<8>(d, nsmall, prm, d_status, smem, stream, gen);
    else
      launch_qrp<kQrpMaxDim / 16>(d, nsmall, prm, d_status, smem, stream, gen);
  }
  if (nsmall < (int)list.size())
    launch_general(d + nsmall, (int)list.size() - nsmall, prm, d_status, large_c, stream, gen);
  cudaFreeAsync(d, stream);
}

void copy2d_batched(const std::vector<CopyDesc> &descs, cudaStream_t stream) {
  run_copies2d<false>(descs, stream);
}

void add2d_batched(const std::vector<CopyDesc> &descs, cudaStream_t stream) {
  run_copies2d<true>(descs, stream);
}

}  // namespace hb
