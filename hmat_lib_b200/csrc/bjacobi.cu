// Block one-sided Jacobi SVD (see bjacobi.h).
//
// Per problem, one workspace holds X (the columns being orthogonalised,
// Lp x Lp, Lp = L rounded up to whole 32-column blocks, padding rows and
// columns zero)
// and V (the accumulated right rotations, Lp x Lp).  A round is ONE launch of
// bj_pair_kernel for every pair of every active problem: a cluster of CTAs
// per pair of blocks (64 columns), each CTA owning a slice of the rows.
//   1. Gram matrix of the pair, G = X_pair^T X_pair (64 x 64), on the FP64
//      tensor cores (mma m8n8k4), each CTA over its rows, then summed over the
//      cluster through distributed shared memory in rank order, so every CTA
//      of the cluster holds the same G bit for bit;
//   2. if some column pair of G is coupled above the convergence test, every
//      CTA runs sweeps of cyclic two-sided Jacobi on G, G = W diag W^T (the
//      same arithmetic in every CTA, so the same W), and sorts the diagonal in
//      descending order; pairs inside a block once a sweep, else pairs across;
//   3. X[:, pair] = X[:, pair] W and V[:, pair] = V[:, pair] W over its rows
//      (mma m8n8k4 again), in place, a 32-row tile at a time.
// Phases 1 and 3 read 32 x 64 tiles through a ring of asynchronous copies and
// are bound by the FP64 tensor cores (2.6 x 64 x 64 multiply-adds per row and
// pair); phase 2 by the latency of its 63 steps a sweep, which is why a step
// has one barrier and its angle comes from single precision (see rotation()).
// Core stage (254 cores of up to 704 columns, n = 32768 2D): 61 -> 28 ms; 62
// cores of up to 1600 columns (n = 8192 3D): 179 -> 74 ms (33 and 79 with all
// 63 steps in every round); 21 and 71 ms with starts and ends in one launch
// each, 18.6 and 61 ms with the norm-relative test of needs_rotation().  A round of 1600-row pairs, a CTA each: Gram 89k cycles, eigensolver 45k
// a sweep, rotation 290k (205k at the FP64 tensor peak).
// Rotations act on the columns themselves (no re-factorisation of a pair), so
// small columns keep their relative accuracy; the rotation is applied only
// when the pair needs it, so the late sweeps are mostly Gram passes.
// Round r of a sweep pairs blocks as the round-robin tournament does (block
// players - 1 fixed, the others rotating), so a sweep of players - 1 rounds
// pairs every block with every other once.  All active problems advance one
// round per launch: problem p is in round g mod (players_p - 1) of global
// round g.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <numeric>

#include "bjacobi.h"
#include "dmma.cuh"
#include "dtree.h"
#include "jacobi.h"
#include "tsqr.h"

namespace cg = cooperative_groups;

namespace hb {

namespace {

constexpr int kBj = 32;          // columns per block
constexpr int kPair = 2 * kBj;   // columns per pair
constexpr int kLd = 68;          // leading dimension of the 64 x 64 tiles in shared memory
constexpr int kPW = 8;           // warps of the pair kernel that hold G and W
constexpr int kPT = 32 * (kPW + 1);   // threads: one more warp computes the rotations
constexpr int kHalf = kPair / 2; // column pairs of a step
// Sweeps of a pair's eigensolver at most (option bj_inner_sweeps).  A pair need
// not be finished: its rotation is orthogonal all the same, and the outer
// sweeps finish the job.  Core stage with 4 / 3 / 2 / 1: 32 / 30 / 28 / 33 ms at
// n = 32768 (2D), 82 / 78 / 74 / 92 ms at n = 8192 (3D).
constexpr int kInner = 2;
constexpr int kT = 32;           // transpose tile, rows of a staged tile
constexpr int kLdT = kT + 4;     // leading dimension of a staged tile (column by column)
constexpr int kRing = 3;         // staged tiles in flight
constexpr int kMaxCluster = 8;

template <class T>
T *upload_vec(const std::vector<T> &v, cudaStream_t s) {
  T *d = nullptr;
  pool_alloc(&d, sizeof(T) * std::max<size_t>(v.size(), 1), s);
  if (!v.empty())
    h2d_async(d, v.data(), sizeof(T) * v.size(), s);
  return d;
}

// One problem's start and end.
struct BjIo {
  const double *A;   // the core's transpose (L x L, ld lda)
  long long lda;
  double *X, *V;     // Lp x Lp
  int L, Lp;
  int rank;          // end: columns wanted
  const int *perm;   // end: where they are, in order
  double *U, *Vout;  // end: L x rank each, ld L
};

// X = A^T with zero padding, V = I (32 x 32 tiles through shared memory, one
// padding column against bank conflicts): all of both is written.
__global__ void bj_start_kernel(const BjIo *__restrict__ probs) {
  const BjIo P = probs[blockIdx.y];
  __shared__ double tile[kT][kT + 1];
  const int tx = threadIdx.x, ty = threadIdx.y;   // 32 x 8 threads
  const int nt = P.Lp / kT;
  for (int t = blockIdx.x; t < nt * nt; t += gridDim.x) {
    const int i0 = t % nt * kT, j0 = t / nt * kT;
    // tile[jj][ii] = A[(j0 + ii) + (i0 + jj) lda]: coalesced along ii
    for (int jj = ty; jj < kT; jj += 8)
      tile[jj][tx] =
          i0 + jj < P.L && j0 + tx < P.L ? P.A[(j0 + tx) + (long long)(i0 + jj) * P.lda] : 0.0;
    __syncthreads();
    // X[(i0 + ii) + (j0 + jj) Lp] = A[(j0 + jj) + (i0 + ii) lda] = tile[ii][jj]
    for (int jj = ty; jj < kT; jj += 8) {
      const long long o = (i0 + tx) + (long long)(j0 + jj) * P.Lp;
      P.X[o] = tile[tx][jj];
      P.V[o] = i0 + tx == j0 + jj ? 1.0 : 0.0;
    }
    __syncthreads();
  }
}

// The wanted columns of X and V in order.
__global__ void bj_gather_kernel(const BjIo *__restrict__ probs) {
  const BjIo P = probs[blockIdx.y];
  for (int c = blockIdx.x; c < P.rank; c += gridDim.x) {
    const long long from = (long long)P.perm[c] * P.Lp, to = (long long)c * P.L;
    for (int r = threadIdx.x; r < P.L; r += blockDim.x) {
      P.U[to + r] = P.X[from + r];
      P.Vout[to + r] = P.V[from + r];
    }
  }
}

// Blocks (a, b), a < b, of pair k in round r of a round-robin over `players` (even).
__host__ __device__ inline void round_pair(int k, int r, int players, int &a, int &b) {
  if (k == 0) {
    a = r;
    b = players - 1;
  } else {
    a = (r + k) % (players - 1);
    b = (r - k + (players - 1)) % (players - 1);
  }
  if (a > b) {
    const int t = a;
    a = b;
    b = t;
  }
}

struct BjDev {
  double *X, *V;   // Lp x Lp (ld Lp); rows of X past the problem's size are zero
  int Lp, nblk, players;
  double gscale;   // power of two that brings the Gram entries to order one
  double theta2;   // columns of squared norm at or below this are not rotated (times gscale)
  double fro;      // ||A||_F, the scale of the norm-relative test (times sqrt(gscale))
  double conv;     // convergence threshold of a column pair
  int *rot;        // 1 + the last round in which a pair of the problem rotated
};

// Shared memory of the pair kernel.  gp: this CTA's partial Gram (tiles I <= J),
// later W with sorted columns, element (i, j) at i + j kLd.  pl: the pair's Gram
// by place, two buffers of four planes [K][M], K <= M: the
// products of K's first / second column with M's first / second.
struct PairSmem {
  double gp[kPair * kLd];
  double pl[2][4][kHalf][kHalf];
  double2 cs[2][kHalf + kHalf / 8];   // rotations by pair, a pad after every eight (cs_at)
  double dg[kPair];      // diagonal by column, then by place
  int perm[kPair];
};

// At the start of a sweep pair k holds column k of the first block and column
// k of the second (first / second place).
__device__ __forceinline__ int column_at(int k, int second) { return k + second * kHalf; }
// One step moves every column to its next place.  All pairs of the 64 columns
// (`all`): the round-robin (the second column of pair 0 stays), back after 63
// steps.  Pairs across the two blocks only: the second columns move on by one,
// back after 32 steps.
__device__ __forceinline__ void next_place(int &k, int &second, bool all) {
  if (!all) {
    if (second) k = (k + 1) % kHalf;
  } else if (!second) {
    second = k == 0;
    k = k == 0 ? 1 : k - 1;
  } else if (k == kHalf - 1) {
    second = 0;
  } else if (k > 0) {
    ++k;
  }
}
// The place whose column comes to place (k, second) in a step.
__device__ __forceinline__ void prev_place(int &k, int &second, bool all) {
  if (!all) {
    if (second) k = (k + kHalf - 1) % kHalf;
  } else if (!second) {
    if (k == kHalf - 1)
      second = 1;
    else
      ++k;
  } else if (k == 1) {
    k = 0;
    second = 0;
  } else if (k > 1) {
    --k;
  }
}
// Where pair k's rotation is kept: the four lanes of a row of W read pairs
// eight apart at a time.
__device__ __forceinline__ int cs_at(int k) { return k + (k >> 3); }
// Offset in a buffer's planes of the product of the columns at two places.
__device__ __forceinline__ int plane_offset(int k, int sk, int m, int sm) {
  if (k > m) {
    int t = k;
    k = m;
    m = t;
    t = sk;
    sk = sm;
    sm = t;
  }
  if (k == m) {   // the coupling of a pair
    sk = 0;
    sm = 1;
  }
  return ((2 * sk + sm) * kHalf + k) * kHalf + m;
}

// The test of a column pair with squared norms al, be and product ga: true
// when it must be rotated.  Columns at or below theta are neither rotated nor
// tested (all of them together hold at most sqrt(L) theta = 1e-3 tol ||A||_F
// / sqrt(L) of the matrix: no kept singular value moves by more than 0.1% of
// the truncation threshold).  The cosine is taken against ||A||_F in place of
// the smaller column: a coupling at rounding level of the problem's own scale
// counts as converged, because a column recomputed from others carries an error
// of about eps ||A|| times its weight, which no rotation removes.  Against the
// smaller column itself, sweeps at a tolerance of zero chase that error and never
// end.  All squared: no square root on the eigensolver's critical path (entries
// are of order one, so the squares of columns above theta do not vanish).
__device__ __forceinline__ bool needs_rotation(double al, double be, double ga, double theta2,
                                               double fro2, double conv2) {
  return al > theta2 && be > theta2 && ga * ga > conv2 * (fro2 * fmax(al, be));
}

// tan, cos of the rotation that zeroes the product g of two columns whose
// squared norms differ by d = |x_b|^2 - |x_a|^2.  Any angle keeps W orthogonal
// as long as c^2 (1 + t^2) = 1; the angle itself only has to make the product
// small, so t comes from single precision (the product left is about 1e-7 of
// g; needs_rotation() passes only 2 |g| > 1e-13 max(|x_a|^2, |x_b|^2), far inside
// a float's range, so a pair that must turn does) and c is then corrected to double precision for that t: with y close to
// (1 + t^2)^-1/2 and r = 1 - (1 + t^2) y^2, c = y (1 - r)^-1/2, whose binomial
// series to second order is exact beyond 1e-18 at r = 1e-6.  A double-precision
// square root, division and reciprocal square root in a row were about half
// of a step.
__device__ __forceinline__ void rotation(double d, double g, double &t, double &c) {
  const double e = 2.0 * g;
  // both scaled by a power of two near 1 / max(|d|, |e|)
  const int ex = max((__double2hiint(d) >> 20) & 0x7ff, (__double2hiint(e) >> 20) & 0x7ff);
  const double sc = __hiloint2double(max(1, min(2046, 2046 - ex)) << 20, 0);
  const float df = (float)(d * sc), ef = (float)(e * sc);
  const float tf = __fdividef(ef, df + copysignf(sqrtf(fmaf(df, df, ef * ef)), df));
  t = (double)tf;
  const double y = (double)rsqrtf(fmaf(tf, tf, 1.0f));
  const double r = fma(-fma(t, t, 1.0), y * y, 1.0);
  c = fma(y, r * fma(0.375, r, 0.5), y);
}

// One 32-row tile of a pair's 64 columns into shared memory (column by
// column, ld kLdT): 256 contiguous bytes per column, 16-byte copies.
__device__ __forceinline__ void stage_tile(double *buf, const double *xa, const double *xb,
                                           long long ld, int row0) {
  if (threadIdx.x < 32 * kPW) {
#pragma unroll
    for (int q = 0; q < kPair * (kT / 2) / (32 * kPW); ++q) {
      const int e = threadIdx.x + 32 * kPW * q, c = e / (kT / 2), ch = e % (kT / 2);
      const double *src = (c < kBj ? xa + c * ld : xb + (c - kBj) * ld) + row0 + 2 * ch;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                       (unsigned)__cvta_generic_to_shared(buf + c * kLdT + 2 * ch)),
                   "l"(src));
    }
  }
  asm volatile("cp.async.commit_group;\n" ::);
}

// Adds the Gram tiles (I, J), I <= J, of two 4-row steps of a staged tile;
// kSet: rows I = 0, 1, 5 of the 8 x 8 tiling, or the others (18 tiles each).
template <int kSet>
__device__ __forceinline__ void gram_tiles(const double *buf, int s0, int gq, int tq,
                                           double (&acc)[18][2]) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    double f[8];
#pragma unroll
    for (int I = 0; I < 8; ++I) f[I] = buf[(8 * I + gq) * kLdT + 4 * (s0 + q) + tq];
    int t = 0;
#pragma unroll
    for (int I = 0; I < 8; ++I)
      if ((I == 0 || I == 1 || I == 5) == (kSet == 0)) {
#pragma unroll
        for (int J = I; J < 8; ++J) dmma884(acc[t++], f[I], f[J]);
      }
  }
}

template <int kSet>
__device__ __forceinline__ void gram_store(double *gp, const double (&acc)[18][2], bool first,
                                           int gq, int tq) {
  int t = 0;
#pragma unroll
  for (int I = 0; I < 8; ++I)
    if ((I == 0 || I == 1 || I == 5) == (kSet == 0)) {
#pragma unroll
      for (int J = I; J < 8; ++J) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          double &e = gp[(8 * I + gq) + (8 * J + 2 * tq + h) * kLd];
          e = (first ? 0.0 : e) + acc[t][h];
        }
        ++t;
      }
    }
}

// One round for every pair slot: blockIdx.x / cluster size = slot.
__global__ void __launch_bounds__(kPT, 2)
bj_pair_kernel(const BjDev *__restrict__ probs, const int2 *__restrict__ slots, long long g_round,
               int inner_max) {
  extern __shared__ __align__(16) unsigned char bj_smem_raw[];
  PairSmem &S = *reinterpret_cast<PairSmem *>(bj_smem_raw);
  cg::cluster_group cl = cg::this_cluster();
  const int ncl = (int)cl.num_blocks();
  const int crank = (int)cl.block_rank();
  const int2 sl = slots[blockIdx.x / ncl];
  const BjDev P = probs[sl.x];
  int a, b;
  round_pair(sl.y, (int)(g_round % (P.players - 1)), P.players, a, b);
  if (b >= P.nblk) return;   // the bye of an odd block count (the whole cluster)

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const long long Lp = P.Lp;
  double *xa = P.X + (long long)a * kBj * Lp, *xb = P.X + (long long)b * kBj * Lp;
  double *va = P.V + (long long)a * kBj * Lp, *vb = P.V + (long long)b * kBj * Lp;
  // this CTA's rows of X and of V, in 32-row tiles
  const int tiles = P.Lp / kT, per = (tiles + ncl - 1) / ncl;
  const int t0 = min(tiles, crank * per), nt = min(tiles, t0 + per) - t0;
  double *ring = &S.pl[0][0][0][0];   // the planes are free outside the eigensolver
  constexpr int kTile = kPair * kLdT;
  static_assert(kRing * kTile <= 2 * 4 * kHalf * kHalf, "the ring fits the planes");

  // ---- 1. Gram of this CTA's rows: the 36 tiles I <= J of the 8 x 8 tiling
  // (column j of the pair is fragment j / 8, lane row j % 8) in two sets of 18,
  // even and odd warps; a pair of warps takes two of a tile's eight 4-row steps
  {
    double acc[18][2] = {};
    for (int t = 0; t < kRing - 1; ++t)
      if (t < nt)
        stage_tile(ring + t * kTile, xa, xb, Lp, (t0 + t) * kT);
      else
        asm volatile("cp.async.commit_group;\n" ::);
    for (int t = 0; t < nt; ++t) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(kRing - 2));
      __syncthreads();                 // tile t has landed, tile t - 1 is used up
      if (t + kRing - 1 < nt)
        stage_tile(ring + (t + kRing - 1) % kRing * kTile, xa, xb, Lp, (t0 + t + kRing - 1) * kT);
      else
        asm volatile("cp.async.commit_group;\n" ::);
      const double *buf = ring + t % kRing * kTile;
      if (warp < kPW) {
        if (warp & 1)
          gram_tiles<1>(buf, 2 * (warp >> 1), gq, tq, acc);
        else
          gram_tiles<0>(buf, 2 * (warp >> 1), gq, tq, acc);
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    // added into gp in warp order (deterministic)
    for (int w = 0; w < kPW / 2; ++w) {
      if (warp < kPW && warp >> 1 == w) {
        if (warp & 1)
          gram_store<1>(S.gp, acc, w == 0, gq, tq);
        else
          gram_store<0>(S.gp, acc, w == 0, gq, tq);
      }
      __syncthreads();
    }
  }
  // ---- the cluster's sum, in rank order, into every CTA's planes
  if (ncl > 1) cl.sync();
  for (int e = tid; e < kPair * kPair; e += kPT) {
    const int i = e % kPair, j = e / kPair;
    if (i > j) continue;
    const int off = i + j * kLd;
    double s = 0.0;
    if (ncl == 1) {
      s = S.gp[off];
    } else {
      for (int rk = 0; rk < ncl; ++rk) s += *cl.map_shared_rank(S.gp + off, rk);
    }
    s *= P.gscale;
    if (i == j) {
      S.dg[i] = s;
    } else {
      (&S.pl[0][0][0][0])[plane_offset(i % kHalf, i / kHalf, j % kHalf, j / kHalf)] = s;
    }
  }
  // after this barrier no CTA reads another's gp any more
  if (ncl > 1) cl.sync();
  __syncthreads();

  // ---- 2. eigensolver: cyclic two-sided Jacobi.  Columns sit at 64 places, 32
  // pairs, and move to their next place after every step, so each thread
  // always handles the same places.  Warps 0 .. kPW - 1 apply a step: two
  // off-diagonal 2 x 2 blocks each (in the planes, read from one buffer and
  // written to their next places in the other) and a quarter of a row of W (in
  // registers).  Meanwhile warp kPW, which keeps the diagonal in registers,
  // computes the next step's 32 rotations: lane k applies the step to the one
  // block that holds the next product of pair k itself.  So a step has one
  // barrier and lasts as long as that chain (a block, an angle).
  // Pairs inside a block are tested and rotated once a sweep, in its first
  // round (the block with the bye there: in the second); otherwise the 32
  // steps of pairs across the blocks do, half the 63 of all pairs.
  const int r_sweep = (int)(g_round % (P.players - 1));
  const bool all = r_sweep == 0 || (r_sweep == 1 && a == 0);
  const bool solver = warp == kPW;
  constexpr int kBlocks = kHalf * (kHalf - 1) / 2;   // off-diagonal blocks K < M
  constexpr int kPlane = kHalf * kHalf;
  int from[2], to[2][4], bk[2], bm[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    // rows i and 30 - i of the triangle make 32 blocks together
    const int e = tid + 32 * kPW * u, i = e / kHalf, l = e % kHalf;
    const bool lower = l >= kHalf - 1 - i;
    bk[u] = lower ? kHalf - 2 - i : i;
    bm[u] = lower ? l : i + 1 + l;
    if (solver || e >= kBlocks) bk[u] = -1;
    from[u] = bk[u] * kHalf + bm[u];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int k = bk[u], sk = q >> 1, m = bm[u], sm = q & 1;
      next_place(k, sk, all);
      next_place(m, sm, all);
      to[u][q] = plane_offset(k, sk, m, sm);
    }
  }
  const double fro2 = P.fro * P.fro, conv2 = P.conv * P.conv;
  // solver lane k: the diagonal of pair k's columns, what its pending rotation
  // moves between them and leaves of their product, where that goes, and the
  // block and element that become the pair's next product
  double d0 = 0.0, d1 = 0.0, left = 0.0, moved = 0.0;
  int to_pair = 0, nk = 0, nm = 0, nq = 0;
  {
    int k = lane, sk = 0, m = lane, sm = 1;
    next_place(k, sk, all);
    next_place(m, sm, all);
    to_pair = plane_offset(k, sk, m, sm);
    // the places whose columns come to (lane, first) and (lane, second)
    int ka = lane, sa = 0, kb = lane, sb = 1;
    prev_place(ka, sa, all);
    prev_place(kb, sb, all);
    nk = min(ka, kb);
    nm = max(ka, kb);
    nq = ka < kb ? 2 * sa + sb : 2 * sb + sa;
  }
  if (solver) {
    d0 = S.dg[column_at(lane, 0)];
    d1 = S.dg[column_at(lane, 1)];
    __syncwarp();
    S.dg[lane] = d0;
    S.dg[kHalf + lane] = d1;
  }
  __syncthreads();
  int par = 0;
  // whether some column pair of the current G that this round tests must be
  // rotated (uniform)
  auto unconverged = [&]() -> bool {
    const double *pl = &S.pl[par][0][0][0];
    bool w = false;
    if (solver) {
      w = needs_rotation(d0, d1, pl[plane_offset(lane, 0, lane, 1)], P.theta2, fro2, conv2);
    } else {
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (bk[u] >= 0) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            w = w || ((all || q == 1 || q == 2) && needs_rotation(S.dg[bk[u] + (q >> 1) * kHalf], S.dg[bm[u] + (q & 1) * kHalf],
                                    pl[from[u] + q * kPlane], P.theta2, fro2, conv2));
        }
    }
    return __syncthreads_or(w) != 0;
  };
  if (!unconverged()) return;   // the same decision in every CTA of the cluster

  // row `wrow` of W at the places of pairs 8 tq .. 8 tq + 7: first / second columns
  const int wrow = 8 * warp + gq;
  double wa[8], wb[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    wa[u] = column_at(8 * tq + u, 0) == wrow ? 1.0 : 0.0;
    wb[u] = column_at(8 * tq + u, 1) == wrow ? 1.0 : 0.0;
  }
  // the rotation of a pair with product g: published, and what it does to the
  // pair kept for the step that applies it
  auto decide = [&](double g, int buf) {
    double t, c;
    rotation(d1 - d0, g, t, c);
    if (!needs_rotation(d0, d1, g, P.theta2, fro2, conv2)) {
      t = 0.0;
      c = 1.0;
    }
    // x_a' = c x_a - s x_b, x_b' = s x_a + c x_b
    S.cs[buf][cs_at(lane)] = make_double2(c, c * t);
    // the norms change by t times the product before and after
    left = c * c * fma(t, d0 - d1, fma(-t * t, g, g));
    moved = t * (g + left);
  };
  if (solver) decide(S.pl[par][1][lane][lane], par);
  __syncthreads();
  for (int sweep = 0; sweep < inner_max; ++sweep) {
    for (int step = all ? kPair - 1 : kHalf; step > 0; --step) {
      const double *src = &S.pl[par][0][0][0];
      double *dst = &S.pl[par ^ 1][0][0][0];
      if (solver) {
        const double2 K = S.cs[par][cs_at(nk)], M = S.cs[par][cs_at(nm)];
        const double *blk = src + nk * kHalf + nm;
        const double b00 = blk[0], b01 = blk[kPlane], b10 = blk[2 * kPlane], b11 = blk[3 * kPlane];
        dst[to_pair] = left;
        const double x = (nq & 2) ? K.y : K.x, y = (nq & 2) ? K.x : -K.y;
        const double z = (nq & 1) ? M.y : M.x, w = (nq & 1) ? M.x : -M.y;
        const double g = z * (x * b00 + y * b10) + w * (x * b01 + y * b11);
        const double n0 = d0 - moved, n1 = d1 + moved;
        const double dn = __shfl_sync(0xffffffffu, n1, (lane + kHalf - 1) % kHalf);
        if (all) {
          const double up = __shfl_down_sync(0xffffffffu, n0, 1);
          const double first = __shfl_sync(0xffffffffu, n0, 0);
          d0 = lane == kHalf - 1 ? n1 : up;
          d1 = lane == 0 ? n1 : lane == 1 ? first : dn;
        } else {
          d0 = n0;
          d1 = dn;
        }
        decide(g, par ^ 1);
      } else {
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (bk[u] >= 0) {
            const double2 K = S.cs[par][cs_at(bk[u])], M = S.cs[par][cs_at(bm[u])];
            const double b00 = src[from[u]], b01 = src[from[u] + kPlane];
            const double b10 = src[from[u] + 2 * kPlane], b11 = src[from[u] + 3 * kPlane];
            const double r00 = K.x * b00 - K.y * b10, r01 = K.x * b01 - K.y * b11;
            const double r10 = K.y * b00 + K.x * b10, r11 = K.y * b01 + K.x * b11;
            dst[to[u][0]] = M.x * r00 - M.y * r01;
            dst[to[u][1]] = M.y * r00 + M.x * r01;
            dst[to[u][2]] = M.x * r10 - M.y * r11;
            dst[to[u][3]] = M.y * r10 + M.x * r11;
          }
        // W = W J, then every column to its next place
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const double2 cs = S.cs[par][cs_at(8 * tq + u)];
          const double x = wa[u], y = wb[u];
          wa[u] = cs.x * x - cs.y * y;
          wb[u] = cs.y * x + cs.x * y;
        }
        const double bn = __shfl_sync(0xffffffffu, wb[7], (lane & ~3) | ((lane + 3) & 3));
        if (all) {
          const double an = __shfl_down_sync(0xffffffffu, wa[0], 1);
          const double a0 = wa[0], b7 = wb[7], b0 = wb[0];
#pragma unroll
          for (int u = 0; u < 7; ++u) wa[u] = wa[u + 1];
          wa[7] = tq == 3 ? b7 : an;
#pragma unroll
          for (int u = 7; u > 0; --u) wb[u] = wb[u - 1];
          if (tq == 0) {
            wb[0] = b0;
            wb[1] = a0;
          } else {
            wb[0] = bn;
          }
        } else {
#pragma unroll
          for (int u = 7; u > 0; --u) wb[u] = wb[u - 1];
          wb[0] = bn;
        }
      }
      par ^= 1;
      __syncthreads();
    }
    if (solver) {
      S.dg[lane] = d0;
      S.dg[kHalf + lane] = d1;
    }
    __syncthreads();
    if (!unconverged()) break;   // the rotations decided last are not applied
  }

  // ---- sort the eigenvalues in descending order (ties by column); the
  // sorted W into gp
  if (solver) {
    S.dg[column_at(lane, 0)] = d0;
    S.dg[column_at(lane, 1)] = d1;
  }
  __syncthreads();
  if (tid < kPair) {
    const double d = S.dg[tid];
    int pos = 0;
    for (int j = 0; j < kPair; ++j) {
      const double dj = S.dg[j];
      pos += (dj > d || (dj == d && j < tid)) ? 1 : 0;
    }
    S.perm[tid] = pos;
  }
  __syncthreads();
  if (!solver) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      S.gp[wrow + S.perm[column_at(8 * tq + u, 0)] * kLd] = wa[u];
      S.gp[wrow + S.perm[column_at(8 * tq + u, 1)] * kLd] = wb[u];
    }
  }
  if (crank == 0 && tid == 0) *P.rot = (int)g_round + 1;
  __syncthreads();

  // ---- 3. the rotation of this CTA's rows of X and V, in place, a 32-row
  // tile of 64 columns at a time: warp w computes columns 8 w .. 8 w + 7 and
  // keeps its part of W in registers
  double bw[kPair / 4];
  if (!solver) {
#pragma unroll
    for (int kk = 0; kk < kPair / 4; ++kk) bw[kk] = S.gp[(4 * kk + tq) + (8 * warp + gq) * kLd];
  }
  auto stage = [&](int t) {            // tiles of X, then of V
    if (t >= 2 * nt)
      asm volatile("cp.async.commit_group;\n" ::);
    else if (t < nt)
      stage_tile(ring + t % kRing * kTile, xa, xb, Lp, (t0 + t) * kT);
    else
      stage_tile(ring + t % kRing * kTile, va, vb, Lp, (t0 + t - nt) * kT);
  };
  for (int t = 0; t < kRing - 1; ++t) stage(t);
  for (int t = 0; t < 2 * nt; ++t) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kRing - 2));
    __syncthreads();
    stage(t + kRing - 1);
    if (!solver) {
      const double *buf = ring + t % kRing * kTile;
      double c[kT / 8][2] = {};
#pragma unroll
      for (int kk = 0; kk < kPair / 4; ++kk)
#pragma unroll
        for (int i = 0; i < kT / 8; ++i)
          dmma884(c[i], buf[(4 * kk + tq) * kLdT + 8 * i + gq], bw[kk]);
      double *pa = t < nt ? xa : va, *pb = t < nt ? xb : vb;
      const int row0 = (t0 + (t < nt ? t : t - nt)) * kT;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = 8 * warp + 2 * tq + h;
        double *dst = (j < kBj ? pa + j * Lp : pb + (j - kBj) * Lp) + row0 + gq;
#pragma unroll
        for (int i = 0; i < kT / 8; ++i) dst[8 * i] = c[i][h];
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
}

// The integer outputs of one problem.
struct BjIntOut {
  int *rank, *sweeps;
  int r, sw;
};

__global__ void bj_int_out_kernel(const BjIntOut *__restrict__ o, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    *o[i].rank = o[i].r;
    if (o[i].sweeps) *o[i].sweeps = o[i].sw;
  }
}

struct Work {
  int L = 0, Lp = 0, nblk = 0, players = 0, npairs = 0;
  long long x = 0, v = 0;
  int sweep = 0;
  bool active = true, converged = false;
};

}  // namespace

void block_jacobi_svd(const std::vector<BjProb> &probs, double tol, int max_sweeps,
                      int *d_status, cudaStream_t s) {
  const int np = (int)probs.size();
  if (np == 0) return;
  // ---- layout ------------------------------------------------------------------------
  std::vector<Work> wk(np);
  long long total = 0;
  auto take = [&](long long e) {
    const long long o = total;
    total += align_up(std::max<long long>(e, 1));
    return o;
  };
  int lmax = 0;
  for (int p = 0; p < np; ++p) {
    Work &W = wk[p];
    W.L = probs[p].L;
    HB_REQUIRE(W.L >= kPair, INPUT_ERROR, "block Jacobi SVD: problem narrower than 64 columns");
    W.Lp = (W.L + kBj - 1) / kBj * kBj;
    W.nblk = W.Lp / kBj;
    W.players = W.nblk + (W.nblk & 1);
    W.npairs = W.players / 2;
    W.x = take((long long)W.Lp * W.Lp);
    W.v = take((long long)W.Lp * W.Lp);
    lmax = std::max(lmax, W.L);
  }
  std::vector<long long> noff(np);   // squared column norms of X
  for (int p = 0; p < np; ++p) noff[p] = take(wk[p].Lp);
  double *w = dev_alloc(total, s);
  int *d_rot = nullptr;   // per problem: 1 + the last round that rotated a pair
  pool_alloc(&d_rot, sizeof(int) * np, s);
  HB_CUDA(cudaMemsetAsync(d_rot, 0, sizeof(int) * np, s));
  // ---- X = A^T, V = I, thresholds -------------------------------------------------------
  std::vector<NormDesc> nd;
  std::vector<BjIo> io;
  for (int p = 0; p < np; ++p) {
    const Work &W = wk[p];
    io.push_back(BjIo{probs[p].A, probs[p].lda, w + W.x, w + W.v, W.L, W.Lp, 0, nullptr,
                      probs[p].U, probs[p].V});
    nd.push_back(NormDesc{w + W.x, W.Lp, W.L, W.Lp, w + noff[p]});
  }
  // `io` in pieces of a grid's height
  auto for_problems = [&](auto launch) {
    BjIo *d = upload_vec(io, s);
    for (int off = 0; off < np; off += 65535) {
      launch(d + off, std::min(65535, np - off));
      HB_LAUNCHED();
    }
    cudaFreeAsync(d, s);
  };
  for_problems([&](const BjIo *d, int n) {
    bj_start_kernel<<<dim3(64, (unsigned)n), dim3(kT, 8), 0, s>>>(d);
  });
  column_norms2(nd, s);
  // a column pair of length L recomputed by a 64-term sum is orthogonal to
  // about sqrt(L) eps
  const double conv = 8.0 * std::sqrt((double)lmax) * 2.220446049250313e-16;
  // the column norms of every problem lie in one range of the workspace:
  // read them in one copy
  const long long n_lo = noff[0], n_hi = noff[np - 1] + wk[np - 1].Lp;
  std::vector<double> hn((size_t)(n_hi - n_lo));
  auto read_norms = [&]() {
    HB_CUDA(cudaMemcpyAsync(hn.data(), w + n_lo, sizeof(double) * (n_hi - n_lo),
                            cudaMemcpyDeviceToHost, s));
    HB_CUDA(cudaStreamSynchronize(s));
  };
  std::vector<BjDev> hd(np);
  {
    read_norms();
    for (int p = 0; p < np; ++p) {
      double f2 = 0.0;
      for (int c = 0; c < wk[p].Lp; ++c) f2 += hn[noff[p] - n_lo + c];
      const Work &W = wk[p];
      // the scalar solver's skip rule for the relative truncation
      const double fro = std::sqrt(f2);
      const double down =
          fro > 0.0 && std::isfinite(fro) ? std::ldexp(1.0, std::max(-500, std::min(500, -std::ilogb(fro))))
                                          : 1.0;
      const double theta = 1e-3 * tol * (fro * down) / W.L;
      hd[p] = BjDev{w + W.x, w + W.v, W.Lp, W.nblk, W.players, down * down, theta * theta,
                    fro * down, conv, d_rot + p};
    }
  }
  BjDev *d_probs = upload_vec(hd, s);
  std::vector<int> rot(np, 0);

  const int inner_max = std::max(1, std::min(30, (int)option("bj_inner_sweeps", kInner)));
  int dev = 0, nsm = 148;
  HB_CUDA(cudaGetDevice(&dev));
  HB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  // A launch that gives every CTA an SM of its own asks for more than half of
  // an SM's shared memory: two CTAs of a cluster otherwise share one while
  // other SMs idle, and the eigensolver's steps take turns.
  const size_t smem_two = sizeof(PairSmem), smem_one = 120 * 1024;
  static_assert(2 * (sizeof(PairSmem) + 1024) <= 228 * 1024 && sizeof(PairSmem) <= 120 * 1024,
                "two CTAs per SM, or one");
  HB_CUDA(cudaFuncSetAttribute(bj_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem_one));

  // The pair slots of the active problems and the cluster size (CTAs per
  // pair: as many as keep one wave of CTAs on the SMs, at most 8, and at
  // least 64 rows per CTA); made again when a problem leaves.
  int2 *d_slots = nullptr;
  int nslots = 0, ncl = 1;
  auto make_slots = [&]() {
    std::vector<int2> sl;
    int lmin = 1 << 30;
    for (int p = 0; p < np; ++p) {
      if (!wk[p].active) continue;
      for (int k = 0; k < wk[p].npairs; ++k) sl.push_back(make_int2(p, k));
      lmin = std::min(lmin, wk[p].L);
    }
    nslots = (int)sl.size();
    ncl = std::max(1, std::min({kMaxCluster, nsm / std::max(nslots, 1), lmin / 64}));
    if (d_slots) cudaFreeAsync(d_slots, s);
    d_slots = upload_vec(sl, s);
  };
  make_slots();

  // ---- rounds ------------------------------------------------------------------------------
  for (long long g = 0;; ++g) {
    bool any = false;
    for (const Work &W : wk) any = any || W.active;
    if (!any) break;
    {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)(nslots * ncl));
      cfg.blockDim = dim3(kPT);
      cfg.dynamicSmemBytes = nslots * ncl <= nsm ? smem_one : smem_two;
      cfg.stream = s;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)ncl;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      HB_CUDA(cudaLaunchKernelEx(&cfg, bj_pair_kernel, (const BjDev *)d_probs,
                                 (const int2 *)d_slots, g, inner_max));
      HB_LAUNCHED();
    }
    // end of a sweep of some problem: a problem whose sweep rotated nothing
    // has converged
    bool check = false;
    for (const Work &W : wk)
      if (W.active && (g + 1) % (W.players - 1) == 0) check = true;
    if (!check) continue;
    HB_CUDA(cudaMemcpyAsync(rot.data(), d_rot, sizeof(int) * np, cudaMemcpyDeviceToHost, s));
    HB_CUDA(cudaStreamSynchronize(s));
    bool changed = false;
    for (int p = 0; p < np; ++p) {
      Work &W = wk[p];
      if (!W.active || (g + 1) % (W.players - 1) != 0) continue;
      ++W.sweep;
      if (rot[p] <= g + 1 - (W.players - 1)) {   // none since the sweep began
        W.active = false;
        W.converged = true;
        changed = true;
      } else if (W.sweep >= max_sweeps) {
        W.active = false;
        changed = true;
      }
    }
    if (changed) make_slots();
  }
  if (d_slots) cudaFreeAsync(d_slots, s);
  cudaFreeAsync(d_probs, s);

  // ---- singular values, order, rank, outputs -------------------------------------------
  nd.clear();
  for (int p = 0; p < np; ++p) nd.push_back(NormDesc{w + wk[p].x, wk[p].Lp, wk[p].L, wk[p].Lp,
                                                     w + noff[p]});
  column_norms2(nd, s);
  std::vector<int> perms;
  std::vector<std::vector<double>> sig(np);
  std::vector<int> ranks(np), sweeps(np);
  read_norms();
  for (int p = 0; p < np; ++p) {
    const Work &W = wk[p];
    const std::vector<double> n2(hn.begin() + (noff[p] - n_lo),
                                 hn.begin() + (noff[p] - n_lo) + W.Lp);
    std::vector<int> perm(W.Lp);
    std::iota(perm.begin(), perm.end(), 0);
    std::stable_sort(perm.begin(), perm.end(), [&](int a, int b) { return n2[a] > n2[b]; });
    sig[p].resize(W.L);
    for (int c = 0; c < W.L; ++c) sig[p][c] = std::sqrt(std::max(n2[perm[c]], 0.0));
    const double s0 = sig[p][0];
    int r = 1;
    if (s0 > tol)
      while (r < W.L && sig[p][r] >= tol * s0) ++r;
    ranks[p] = r;
    sweeps[p] = W.converged ? W.sweep : max_sweeps + 1;
    io[p].rank = r;
    perms.insert(perms.end(), perm.begin(), perm.begin() + r);
  }
  int *d_perm = upload_vec(perms, s);
  {
    int at = 0, widest = 1;
    for (int p = 0; p < np; ++p) {
      io[p].perm = d_perm + at;
      at += ranks[p];
      widest = std::max(widest, ranks[p]);
    }
    for_problems([&](const BjIo *d, int n) {
      bj_gather_kernel<<<dim3((unsigned)std::min(widest, 64), (unsigned)n), 256, 0, s>>>(d);
    });
  }
  cudaFreeAsync(d_perm, s);
  // singular values (one upload, scattered by one copy launch), ranks and
  // sweeps (one launch)
  bool failed = false;
  {
    std::vector<double> hs;
    std::vector<long long> so(np);
    for (int p = 0; p < np; ++p) {
      so[p] = (long long)hs.size();
      hs.insert(hs.end(), sig[p].begin(), sig[p].end());
    }
    double *ds = upload_vec(hs, s);
    std::vector<CopyDesc> sc;
    std::vector<BjIntOut> ints;
    for (int p = 0; p < np; ++p) {
      sc.push_back(CopyDesc{ds + so[p], wk[p].L, probs[p].sigma, wk[p].L, wk[p].L, 1});
      ints.push_back(BjIntOut{probs[p].rank, probs[p].sweeps, ranks[p], sweeps[p]});
      failed = failed || !wk[p].converged;
    }
    copy2d_batched(sc, s);
    BjIntOut *dio = upload_vec(ints, s);
    bj_int_out_kernel<<<(np + 127) / 128, 128, 0, s>>>(dio, np);
    HB_LAUNCHED();
    cudaFreeAsync(dio, s);
    cudaFreeAsync(ds, s);
  }
  if (failed) {
    const int st = SVD_FAILURE;
    HB_CUDA(cudaMemcpyAsync(d_status, &st, sizeof(int), cudaMemcpyHostToDevice, s));
    set_last_error("block Jacobi SVD of a sketch core did not converge within "
                   "jacobi_max_sweeps sweeps");
  }
  HB_CUDA(cudaStreamSynchronize(s));
  cudaFreeAsync(d_rot, s);
  dev_free(w, s);
}

}  // namespace hb
