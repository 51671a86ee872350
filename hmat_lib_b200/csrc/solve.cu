// HODLR factorisation and solve (see solve.h for the algebra).
//
// The capacitance matrix of a node, C = [I, P; Q, I] with P = V_tr^T W2 and
// Q = V_bl^T W1, has identity diagonal blocks, so only its Schur complement
// S = I - Q P (order s_bl) is inverted; C^-1 is then assembled from P, Q and
// S^-1 by two small GEMM launches and kept, so that a solve applies it as one
// GEMM per level instead of three dependent ones.
#include <algorithm>
#include <cmath>

#include <cooperative_groups.h>

#include "dmma.cuh"
#include "gemm_f64.h"
#include "jacobi.h"
#include "solve.h"

namespace cg = cooperative_groups;

namespace hb {

namespace {

constexpr int kGjThreads = 512;
constexpr int kGjWarps = kGjThreads / 32;
constexpr int kGjB = 32;             // columns per panel, columns per update strip
constexpr int kGjMaxCluster = 8;
constexpr size_t kGjSmem = 200 * 1024;
constexpr int kGjMaxN = 25600;       // row numbers are kept as short

struct GjProb {
  const double *A;   // n x n input (ld lda)
  long long lda;
  int n;
  double *work;      // n x n scratch, ld n
  double *inv;       // n x n output (ld ldi)
  long long ldi;
  int2 *moves;       // 2 kGjB row moves (to, from) of the current panel
  int *flag;         // set when a pivot is at rounding level
};

// Leading dimension of the panel in shared memory: 4 mod 16, so that eight
// rows by four columns hit every bank once.
__host__ __device__ inline int gj_ldp(int n) { return (n + 15) / 16 * 16 + 4; }
// Shared memory beside the panel: the pivot rows of a strip, row numbers.
__host__ __device__ inline size_t gj_base_smem(int n) {
  return sizeof(double) * kGjB * (kGjB + 4) + 2 * sizeof(short) * ((size_t)n + 8);
}
inline size_t gj_panel_smem(int n) { return sizeof(double) * kGjB * (size_t)gj_ldp(n); }

// In-place blocked Gauss-Jordan inversion with partial pivoting, a cluster of
// CTAs per matrix.  Per panel of 32 columns:
//   1. rank 0 runs the 32 elimination steps on the panel alone, in shared
//      memory, pivots searched over all rows not yet used; what is left in
//      the panel is the matrix T whose product with the pivot rows is the
//      steps' effect on any other column;
//   2. every CTA takes its share of the 32-column strips: rows moved as the
//      panel's swaps moved them, then W <- W + T W[pivot rows] (pivot rows:
//      T W[pivot rows]) on the FP64 tensor cores.
// The matrix ends as the inverse of the row-permuted input, whose columns go
// to their places in the output.  The steps are a chain of n pivot searches,
// each two barriers and a pass over n x 32 values in shared memory; the rest
// is 2 n^3 flops on up to eight SMs.  W is written and read by the CTAs of the
// cluster in turn, ordered by the cluster barrier, and read past L1.  A panel
// taller than shared memory stays in global memory (ld n).  A pivot at rounding level relative to the matrix's
// largest entry sets *status (the output is then not used).
// All inverses of an n = 16384 factorisation (128 leaves of 128 rows, Schur
// complements of 60 to 280 rows): 88 ms with one CTA per matrix eliminating
// column by column in global memory, 2.5 ms so.
template <bool kShared>
__device__ void gj_invert(const GjProb &P, int *status, double *sm, int crank, int ncl) {
  cg::cluster_group cl = cg::this_cluster();
  const int n = P.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  __shared__ double s_val[kGjWarps];
  __shared__ double s_amax;
  __shared__ unsigned s_hi[2][kGjWarps], s_lo[2][kGjWarps];
  __shared__ int s_idx[2][kGjWarps], s_piv[kGjB], s_fail;
  double *Bs = sm;                                       // [k][column], ld kGjB + 4
  short *perm = reinterpret_cast<short *>(sm + kGjB * (kGjB + 4));   // rows of A by place
  short *src = perm + n + 8;                             // this panel's row moves
  double *Ps = reinterpret_cast<double *>(reinterpret_cast<char *>(sm) +
                                          (gj_base_smem(n) + 15) / 16 * 16);
  constexpr int LDB = kGjB + 4;
  double *W = P.work;
  const long long ldp = kShared ? gj_ldp(n) : n;
  const int nstrip = (n + kGjB - 1) / kGjB, ntile = (n + 7) / 8;

  // ---- copy, largest entry -----------------------------------------------------------
  double amax = 0.0;
  for (int st = crank; st < nstrip; st += ncl)
    for (int c = st * kGjB + warp; c < min(n, (st + 1) * kGjB); c += kGjWarps)
      for (int r = lane; r < n; r += 32) {
        const double a = P.A[r + (long long)c * P.lda];
        W[r + (long long)c * n] = a;
        amax = fmax(amax, fabs(a));
      }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (lane == 0) s_val[warp] = amax;
  for (int r = tid; r < n; r += kGjThreads) perm[r] = (short)r;
  __syncthreads();
  if (tid == 0) {
    for (int w = 0; w < kGjWarps; ++w) amax = fmax(amax, s_val[w]);
    s_amax = amax;
    s_fail = 0;
  }
  cl.sync();
  amax = 0.0;
  for (int rk = 0; rk < ncl; ++rk) amax = fmax(amax, *cl.map_shared_rank(&s_amax, rk));
  const double tiny = fmax(64.0 * 2.220446049250313e-16 * amax, 1e-300);
  cl.sync();

  for (int K0 = 0; K0 < n; K0 += kGjB) {
    const int b = min(kGjB, n - K0);
    double *Pp = kShared ? Ps : W + (long long)K0 * n;
    auto pl = [](const double *q) { return kShared ? *q : __ldcg(q); };
    // ---- 1. the panel ------------------------------------------------------------------
    if (crank == 0) {
      if (kShared)
        for (int c = warp; c < kGjB; c += kGjWarps)
          for (int r = lane; r < 8 * ntile; r += 32)
            Pp[r + c * ldp] = (c < b && r < n) ? __ldcg(W + r + (long long)(K0 + c) * n) : 0.0;
      for (int r = tid; r < n; r += kGjThreads) src[r] = (short)r;
      __syncthreads();
      double best = -1.0;
      int bi = 0x7fffffff;
      for (int r = K0 + tid; r < n; r += kGjThreads) {
        const double v = fabs(pl(Pp + r));
        if (v > best) {
          best = v;
          bi = r;
        }
      }
      for (int kk = 0; kk < b; ++kk) {
        const int k = K0 + kk, par = kk & 1;
        // pivot: the largest magnitude, ties to the smallest row
        auto reduce = [&](unsigned hi, unsigned lo, int id, unsigned &mh, unsigned &ml, int &mi) {
          mh = __reduce_max_sync(0xffffffffu, hi);
          ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
          mi = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? id : 0x7fffffff);
        };
        unsigned hi = 0, lo = 0, mh, ml;
        int mi;
        if (best >= 0.0) {
          hi = (unsigned)__double2hiint(best);
          lo = (unsigned)__double2loint(best);
        }
        reduce(hi, lo, bi, mh, ml, mi);
        if (lane == 0) {
          s_hi[par][warp] = mh;
          s_lo[par][warp] = ml;
          s_idx[par][warp] = mi;
        }
        __syncthreads();
        const bool in = lane < kGjWarps;
        reduce(in ? s_hi[par][lane] : 0u, in ? s_lo[par][lane] : 0u,
               in ? s_idx[par][lane] : 0x7fffffff, mh, ml, mi);
        const double big = __hiloint2double((int)mh, (int)ml);
        if (mi >= n || big <= tiny) {      // the same in every thread
          if (tid == 0) s_fail = 1;
          break;
        }
        const int p = mi;
        // swap rows k and p, scale row k by 1 / pivot, which takes the pivot's place
        if (tid < kGjB) {
          const double inv = 1.0 / pl(Pp + p + kk * ldp);
          __syncwarp();
          if (tid < b) {
            const double a = pl(Pp + k + tid * ldp), v = pl(Pp + p + tid * ldp);
            Pp[p + tid * ldp] = a;
            Pp[k + tid * ldp] = tid == kk ? inv : v * inv;
          }
        }
        if (tid == kGjB) {
          const short a = perm[k], v = src[k];
          perm[k] = perm[p];
          perm[p] = a;
          src[k] = src[p];
          src[p] = v;
          s_piv[kk] = p;
        }
        __syncthreads();
        // eliminate column kk from the other rows; a warp takes 8 rows, lane
        // (gq, tq) columns 4 s + tq; the next column's pivot search on the way
        const double inv = pl(Pp + k + kk * ldp);
        double prow[kGjB / 4];
#pragma unroll
        for (int s = 0; s < kGjB / 4; ++s)
          prow[s] = 4 * s + tq < b ? pl(Pp + k + (4 * s + tq) * ldp) : 0.0;
        best = -1.0;
        bi = 0x7fffffff;
        for (int t = warp; t < ntile; t += kGjWarps) {
          const int r = 8 * t + gq;
          const bool live = r < n && r != k;
          const double f = live ? pl(Pp + r + kk * ldp) : 0.0;
          __syncwarp();                    // f is read before column kk is written
          if (live) {
#pragma unroll
            for (int s = 0; s < kGjB / 4; ++s) {
              const int c = 4 * s + tq;
              if (c < b) {
                const double a = c == kk ? -f * inv : fma(-f, prow[s], pl(Pp + r + c * ldp));
                Pp[r + c * ldp] = a;
                if (c == kk + 1 && r > k && fabs(a) > best) {
                  best = fabs(a);
                  bi = r;
                }
              }
            }
          }
        }
      }
      __syncthreads();
      if (s_fail) {
        if (tid == 0) *P.flag = 1;
      } else {
        if (kShared)
          for (int c = warp; c < b; c += kGjWarps)
            for (int r = lane; r < n; r += 32) W[r + (long long)(K0 + c) * n] = Pp[r + c * ldp];
        for (int i = tid; i < 2 * kGjB; i += kGjThreads) {
          int2 mv = make_int2(-1, -1);
          if (i < b) {
            mv = make_int2(K0 + i, src[K0 + i]);
          } else if (i >= kGjB && i - kGjB < b) {
            const int q = s_piv[i - kGjB];   // a row may appear twice: the same move
            if (q >= K0 + b) mv = make_int2(q, src[q]);
          }
          P.moves[i] = mv;
        }
      }
    }
    cl.sync();
    if (*(volatile int *)P.flag) {
      if (crank == 0 && tid == 0) atomicExch(status, 1);
      return;                              // the whole cluster
    }
    // ---- 2. the other columns ------------------------------------------------------------
    if (kShared && crank != 0) {
      for (int c = warp; c < kGjB; c += kGjWarps)
        for (int r = lane; r < 8 * ntile; r += 32)
          Ps[r + c * ldp] = (c < b && r < n) ? __ldcg(W + r + (long long)(K0 + c) * n) : 0.0;
    }
    __syncthreads();
    for (int st = crank; st < nstrip; st += ncl) {
      if (st == K0 / kGjB) continue;
      const int c0 = st * kGjB, nc = min(kGjB, n - c0);
      // move rows; the pivot rows go to shared memory ([k][column])
      {
        const int c = tid >> 4, i0 = tid & 15;
        double v[4];
        int to[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int2 mv = P.moves[i0 + 16 * u];
          to[u] = c < nc ? mv.x : -1;
          v[u] = to[u] >= 0 ? __ldcg(W + mv.y + (long long)(c0 + c) * n) : 0.0;
        }
        __syncthreads();                   // every old value read; Bs free
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (u < 2) Bs[(i0 + 16 * u) * LDB + c] = v[u];   // moves 0 .. 31: pivot rows
          else if (to[u] >= 0) W[to[u] + (long long)(c0 + c) * n] = v[u];
        }
        __syncthreads();
      }
      // W += T Bs, a warp per 32 rows
      for (int t = warp; t < nstrip; t += kGjWarps) {
        const bool piv_rows = t == K0 / kGjB;
        double acc[4][4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int jn = 0; jn < 4; ++jn)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int r = 32 * t + 8 * i + gq, c = 8 * jn + 2 * tq + h;
              acc[i][jn][h] =
                  (!piv_rows && r < n && c < nc) ? __ldcg(W + r + (long long)(c0 + c) * n) : 0.0;
            }
#pragma unroll
        for (int s = 0; s < kGjB / 4; ++s) {
          double a[4], bb[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = 32 * t + 8 * i + gq, kx = 4 * s + tq;
            if (kShared)
              a[i] = 4 * t + i < ntile ? Ps[r + kx * ldp] : 0.0;
            else
              a[i] = (r < n && kx < b) ? __ldcg(W + r + (long long)(K0 + kx) * n) : 0.0;
          }
#pragma unroll
          for (int jn = 0; jn < 4; ++jn) bb[jn] = Bs[(4 * s + tq) * LDB + 8 * jn + gq];
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int jn = 0; jn < 4; ++jn) dmma884(acc[i][jn], a[i], bb[jn]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int jn = 0; jn < 4; ++jn)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int r = 32 * t + 8 * i + gq, c = 8 * jn + 2 * tq + h;
              if (r < n && c < nc) W[r + (long long)(c0 + c) * n] = acc[i][jn][h];
            }
      }
    }
    cl.sync();
  }

  // ---- columns to their places: inv[:, perm[c]] = W[:, c] --------------------------------
  const short *pm = cl.map_shared_rank(perm, 0);
  for (int st = crank; st < nstrip; st += ncl)
    for (int c = st * kGjB + warp; c < min(n, (st + 1) * kGjB); c += kGjWarps) {
      const long long to = pm[c];
      for (int r = lane; r < n; r += 32) P.inv[r + to * P.ldi] = __ldcg(W + r + (long long)c * n);
    }
  cl.sync();                               // rank 0's shared memory is read until here
}

__global__ void __launch_bounds__(kGjThreads, 1)
gj_inverse_kernel(const GjProb *__restrict__ probs, int *status, int smem_bytes) {
  extern __shared__ __align__(16) double gj_sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int ncl = (int)cl.num_blocks(), crank = (int)cl.block_rank();
  const GjProb P = probs[blockIdx.x / ncl];
  if ((gj_base_smem(P.n) + 15) / 16 * 16 + sizeof(double) * kGjB * gj_ldp(P.n) <=
      (size_t)smem_bytes)
    gj_invert<true>(P, status, gj_sm, crank, ncl);
  else
    gj_invert<false>(P, status, gj_sm, crank, ncl);
}

struct EyeDesc {
  double *X;
  long long ld;
  int n;
};

__global__ void eye_kernel(const EyeDesc *__restrict__ d) {
  const EyeDesc E = d[blockIdx.y];
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)E.n * E.n;
       e += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(e % E.n), c = (int)(e / E.n);
    E.X[r + (long long)c * E.ld] = (r == c) ? 1.0 : 0.0;
  }
}

template <class T>
T *upload_tmp(const std::vector<T> &v, cudaStream_t s) {
  T *d = nullptr;
  pool_alloc(&d, sizeof(T) * std::max<size_t>(v.size(), 1), s);
  if (!v.empty())
    h2d_async(d, v.data(), sizeof(T) * v.size(), s);
  return d;
}

void gj_inverse(std::vector<GjProb> probs, int *d_status, cudaStream_t s) {
  if (probs.empty()) return;
  const int np = (int)probs.size();
  long long work = 0;
  size_t smem = 0;
  for (auto &p : probs) {
    HB_REQUIRE(p.n <= kGjMaxN, INPUT_ERROR, "solve: capacitance matrix too large");
    work += align_up((long long)p.n * p.n);
    const size_t base = (gj_base_smem(p.n) + 15) / 16 * 16, all = base + gj_panel_smem(p.n);
    smem = std::max(smem, all <= kGjSmem ? all : base);
  }
  // the matrices, then per matrix its row moves and its flag
  const long long ints = (long long)np * (4 * kGjB + 1);
  double *w = dev_alloc(work + (ints + 1) / 2, s);
  int2 *moves = reinterpret_cast<int2 *>(w + work);
  int *flags = reinterpret_cast<int *>(moves + (long long)np * 2 * kGjB);
  HB_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * np, s));
  long long o = 0;
  for (int i = 0; i < np; ++i) {
    GjProb &p = probs[i];
    p.work = w + o;
    o += align_up((long long)p.n * p.n);
    p.moves = moves + (long long)i * 2 * kGjB;
    p.flag = flags + i;
  }
  GjProb *d = upload_tmp(probs, s);
  HB_CUDA(cudaFuncSetAttribute(gj_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kGjSmem));
  // as many CTAs per matrix as keep one CTA per SM
  int ncl = 1;
  while (2 * ncl <= kGjMaxCluster && 2 * ncl * np <= num_sms()) ncl *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(np * ncl));
  cfg.blockDim = dim3(kGjThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ncl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  HB_CUDA(cudaLaunchKernelEx(&cfg, gj_inverse_kernel, (const GjProb *)d, d_status, (int)smem));
  HB_LAUNCHED();
  cudaFreeAsync(d, s);
  dev_free(w, s);
}

void eye(const std::vector<EyeDesc> &v, cudaStream_t s) {
  if (v.empty()) return;
  EyeDesc *d = upload_tmp(v, s);
  for (size_t off = 0; off < v.size(); off += 65535) {
    eye_kernel<<<dim3(8, (unsigned)std::min<size_t>(65535, v.size() - off)), 256, 0, s>>>(d + off);
    HB_LAUNCHED();
  }
  cudaFreeAsync(d, s);
}

int node_index(int d, int j) { return (1 << d) - 1 + j; }

// Base slots of the solver's GEMM launches.
enum Slot { kS_Arena = 0, kS_Buf = 1, kS_X = 2, kS_B = 3, kS_T = 4, kS_Z = 5 };

GemmBases solver_bases(const HodlrFactor &f, double *X, const double *B, double *T, double *Z) {
  GemmBases b{};
  b.p[kS_Arena] = f.tree->arena;
  b.p[kS_Buf] = f.buf;
  b.p[kS_X] = X;
  b.p[kS_B] = const_cast<double *>(B);
  b.p[kS_T] = T;
  b.p[kS_Z] = Z;
  return b;
}

// Scratch of one level: t and z of node j at off[j] (q_j x k, ld q_j).
long long level_scratch(const HodlrFactor &f, int l, int k, std::vector<long long> *off) {
  long long tot = 0;
  if (off) off->assign(1 << l, 0);
  for (int j = 0; j < (1 << l); ++j) {
    if (off) (*off)[j] = tot;
    tot += align_up((long long)f.q[node_index(l, j)] * k);
  }
  return tot;
}

// The three launches of x <- (I + W_l V_l^T)^-1 x, x in slot kS_X (ld ldx, k
// columns), t in kS_T, z in kS_Z.
struct LevelBatches {
  GemmBatch vt, cz, wx;
};

LevelBatches level_batches(const HodlrFactor &f, int l, int k, long long ldx) {
  const Geometry &g = f.tree->g;
  std::vector<long long> off;
  level_scratch(f, l, k, &off);
  LevelBatches L;
  const long long wl = f.w_off[l];
  for (int j = 0; j < (1 << l); ++j) {
    const BlockDesc &tr = g.blocks[block_index(l, j, 1)], &bl = g.blocks[block_index(l, j, 2)];
    const int q = tr.s + bl.s;
    if (q == 0) continue;
    // t = [V_tr^T x[child 2]; V_bl^T x[child 1]]
    if (tr.s) {
      const int p = L.vt.add(kS_T, off[j], q, tr.s, k);
      L.vt.seg(p, kS_Arena, tr.v_off, tr.n, 1, kS_X, tr.c0, ldx, 0, tr.n);
    }
    if (bl.s) {
      const int p = L.vt.add(kS_T, off[j] + tr.s, q, bl.s, k);
      L.vt.seg(p, kS_Arena, bl.v_off, bl.n, 1, kS_X, bl.c0, ldx, 0, bl.n);
    }
    // z = C^-1 t
    const int p = L.cz.add(kS_Z, off[j], q, q, k);
    L.cz.seg(p, kS_Buf, f.cinv_off[node_index(l, j)], q, 0, kS_T, off[j], q, 0, q);
    // x[child 1] -= W1 z1, x[child 2] -= W2 z2
    if (tr.s) {
      const int p1 = L.wx.add(kS_X, tr.r0, ldx, tr.m, k, -1.0, 1.0);
      L.wx.seg(p1, kS_Buf, wl + tr.r0, g.n, 0, kS_Z, off[j], q, 0, tr.s);
    }
    if (bl.s) {
      const int p2 = L.wx.add(kS_X, bl.r0, ldx, bl.m, k, -1.0, 1.0);
      L.wx.seg(p2, kS_Buf, wl + bl.r0, g.n, 0, kS_Z, off[j] + tr.s, q, 0, bl.s);
    }
  }
  return L;
}

// X = D^-1 B: X in slot kS_X, B in kS_B (distinct).
GemmBatch leaf_batch(const HodlrFactor &f, int k, long long ldb, long long ldx) {
  const DeviceTree &t = *f.tree;
  GemmBatch gb;
  for (int i = 0; i < t.g.nleaf(); ++i) {
    const LeafDesc &L = t.leaves[i];
    if (L.m == 0) continue;
    const int p = gb.add(kS_X, L.r0, ldx, L.m, k);
    gb.seg(p, kS_Buf, f.leaf_inv_off[i], L.m, 0, kS_B, L.r0, ldb, 0, L.m);
  }
  return gb;
}

constexpr TileShape kShapeLeaves = TileShape::M128N64;
constexpr TileShape kShapeWx = TileShape::M128N64;
TileShape shape_vt(int k) { return k <= 64 ? TileShape::M64N64 : TileShape::M64N128; }

// One-shot application (factorisation, where k is a level's rank).
void apply_leaves_once(const HodlrFactor &f, const double *B, long long ldb, double *X,
                       long long ldx, int k, cudaStream_t s) {
  GemmBatch gb = leaf_batch(f, k, ldb, ldx);
  gemm_f64_run(gb, solver_bases(f, X, B, nullptr, nullptr), kShapeLeaves, s);
}

void apply_level_once(const HodlrFactor &f, int l, double *X, int k, long long ldx,
                      cudaStream_t s) {
  const long long tot = level_scratch(f, l, k, nullptr);
  if (tot == 0) return;
  double *T = dev_alloc(tot, s), *Z = dev_alloc(tot, s);
  const GemmBases b = solver_bases(f, X, nullptr, T, Z);
  LevelBatches L = level_batches(f, l, k, ldx);
  gemm_f64_run(L.vt, b, shape_vt(k), s);
  gemm_f64_run(L.cz, b, shape_vt(k), s);
  gemm_f64_run(L.wx, b, kShapeWx, s, false);
  dev_free(T, s);
  dev_free(Z, s);
}

}  // namespace

struct SolvePlan {
  GemmPlan leaves;
  std::vector<std::unique_ptr<GemmPlan>> vt, cz, wx;   // per depth
  double *T = nullptr, *Z = nullptr;                  // scratch of the largest level
  ~SolvePlan() {
    if (T) cudaFree(T);
    if (Z) cudaFree(Z);
  }
};

HodlrFactor::HodlrFactor() = default;

HodlrFactor::~HodlrFactor() {
  last_use.wait(tree ? tree->device : 0);
  plans.clear();
  if (buf) cudaFree(buf);
}

namespace {

void build_plan(GemmPlan &plan, GemmBatch &batch, TileShape shape, bool split, cudaStream_t s) {
  if (!batch.empty()) gemm_plan_build(plan, batch, shape, split ? KSplit::All : KSplit::Tail, s);
}

SolvePlan &solve_plan(HodlrFactor &f, int k, long long ldb, long long ldx, cudaStream_t s) {
  std::lock_guard<std::mutex> lk(f.plan_mutex);
  const auto key = std::make_tuple(k, ldb, ldx, s);
  auto it = f.plans.find(key);
  if (it != f.plans.end()) return *it->second;
  auto P = std::make_unique<SolvePlan>();
  const int h = f.tree->g.h;
  GemmBatch lb = leaf_batch(f, k, ldb, ldx);
  build_plan(P->leaves, lb, kShapeLeaves, true, s);
  long long scratch = 0;
  for (int l = 0; l < h; ++l) {
    scratch = std::max(scratch, level_scratch(f, l, k, nullptr));
    LevelBatches L = level_batches(f, l, k, ldx);
    P->vt.push_back(std::make_unique<GemmPlan>());
    P->cz.push_back(std::make_unique<GemmPlan>());
    P->wx.push_back(std::make_unique<GemmPlan>());
    build_plan(*P->vt.back(), L.vt, shape_vt(k), true, s);
    build_plan(*P->cz.back(), L.cz, shape_vt(k), true, s);     // K = q: split near the root
    build_plan(*P->wx.back(), L.wx, kShapeWx, false, s);
  }
  pool_alloc(&P->T, sizeof(double) * std::max<long long>(scratch, 1), s);
  pool_alloc(&P->Z, sizeof(double) * std::max<long long>(scratch, 1), s);
  HB_CUDA(cudaStreamSynchronize(s));
  auto &ref = *P;
  f.plans[key] = std::move(P);
  return ref;
}

}  // namespace

std::unique_ptr<HodlrFactor> hodlr_factorize(std::shared_ptr<DeviceTree> tp, cudaStream_t s,
                                             int *status) {
  auto f = std::make_unique<HodlrFactor>();
  f->tree = tp;
  const DeviceTree &t = *tp;
  const Geometry &g = t.g;
  const int h = g.h, n = g.n;
  *status = SUCCESS;
  // ---- layout of the factor buffer ------------------------------------------------
  long long total = 0;
  f->leaf_inv_off.resize(g.nleaf());
  for (int i = 0; i < g.nleaf(); ++i) {
    f->leaf_inv_off[i] = total;
    total += align_up((long long)g.leaf_m[i] * g.leaf_m[i]);
  }
  f->w_off.assign(h, 0);
  f->w_cols.assign(h, 0);
  for (int l = 0; l < h; ++l) {
    int w = 0;
    for (int j = 0; j < (1 << l); ++j)
      w = std::max({w, g.blocks[block_index(l, j, 1)].s, g.blocks[block_index(l, j, 2)].s});
    f->w_cols[l] = w;
    f->w_off[l] = total;
    total += align_up((long long)n * w);
  }
  const int nnodes = (1 << h) - 1;
  f->cinv_off.assign(nnodes, 0);
  f->q.assign(nnodes, 0);
  for (int d = 0; d < h; ++d)
    for (int j = 0; j < (1 << d); ++j) {
      const int q = g.blocks[block_index(d, j, 1)].s + g.blocks[block_index(d, j, 2)].s;
      f->cinv_off[node_index(d, j)] = total;
      f->q[node_index(d, j)] = q;
      total += align_up((long long)q * q);
    }
  pool_alloc(&f->buf, sizeof(double) * std::max<long long>(total, 1), s);
  HB_CUDA(cudaMemsetAsync(f->buf, 0, sizeof(double) * std::max<long long>(total, 1), s));
  int *d_status = nullptr;
  pool_alloc(&d_status, sizeof(int), s);
  HB_CUDA(cudaMemsetAsync(d_status, 0, sizeof(int), s));

  // ---- leaf inverses -----------------------------------------------------------------
  {
    std::vector<GjProb> probs;
    for (int i = 0; i < g.nleaf(); ++i) {
      const LeafDesc &lf = t.leaves[i];
      if (lf.m == 0) continue;
      probs.push_back(GjProb{t.arena + lf.off, lf.m, lf.m, nullptr,
                             f->buf + f->leaf_inv_off[i], lf.m, nullptr, nullptr});
    }
    gj_inverse(probs, d_status, s);
  }

  // ---- levels, deepest first -----------------------------------------------------------
  const int wmax = *std::max_element(f->w_cols.begin(), f->w_cols.end());
  double *tmp = dev_alloc((long long)n * std::max(wmax, 1), s);
  for (int l = h - 1; l >= 0; --l) {
    const int w = f->w_cols[l];
    if (w == 0) continue;
    double *Wl = f->buf + f->w_off[l];
    // stack the level's U blocks, band by band, then W_l = D^-1 U
    HB_CUDA(cudaMemsetAsync(tmp, 0, sizeof(double) * (long long)n * w, s));
    std::vector<CopyDesc> cp;
    for (int j = 0; j < (1 << l); ++j)
      for (int c = 1; c <= 2; ++c) {
        const BlockDesc &B = g.blocks[block_index(l, j, c)];
        if (B.s) cp.push_back(CopyDesc{t.arena + B.u_off, B.m, tmp + B.r0, n, B.m, B.s});
      }
    copy2d_batched(cp, s);
    apply_leaves_once(*f, tmp, n, Wl, n, w, s);
    for (int lev = h - 1; lev > l; --lev) apply_level_once(*f, lev, Wl, w, n, s);

    // C^-1 of every node of the level.  Scratch per node with both ranks
    // nonzero: P (s_tr x s_bl), Q (s_bl x s_tr), S (s_bl x s_bl).
    std::vector<long long> p_off(1 << l, 0), q_off(1 << l, 0), s_off(1 << l, 0);
    long long scratch = 0;
    for (int j = 0; j < (1 << l); ++j) {
      const int s1 = g.blocks[block_index(l, j, 1)].s, s2 = g.blocks[block_index(l, j, 2)].s;
      if (!s1 || !s2) continue;
      p_off[j] = scratch;
      scratch += align_up((long long)s1 * s2);
      q_off[j] = scratch;
      scratch += align_up((long long)s2 * s1);
      s_off[j] = scratch;
      scratch += align_up((long long)s2 * s2);
    }
    std::vector<EyeDesc> eyes;
    for (int j = 0; j < (1 << l); ++j) {
      const int q = f->q[node_index(l, j)];
      if (q) eyes.push_back(EyeDesc{f->buf + f->cinv_off[node_index(l, j)], q, q});
    }
    eye(eyes, s);                              // C^-1 = I where a rank is zero
    if (scratch == 0) continue;
    double *Ps = dev_alloc(scratch, s);
    const GemmBases b = solver_bases(*f, nullptr, nullptr, Ps, nullptr);
    GemmBatch gpq, gs, c1, c2;
    std::vector<EyeDesc> s_eye;
    std::vector<GjProb> inv;
    for (int j = 0; j < (1 << l); ++j) {
      const BlockDesc &tr = g.blocks[block_index(l, j, 1)], &bl = g.blocks[block_index(l, j, 2)];
      const int s1 = tr.s, s2 = bl.s, q = s1 + s2;
      if (!s1 || !s2) continue;
      const long long ci = f->cinv_off[node_index(l, j)];
      const long long br = ci + s1 + (long long)s1 * q, bl_off = ci + s1, tr_off = ci + (long long)s1 * q;
      int p = gpq.add(kS_T, p_off[j], s1, s1, s2);                 // P = V_tr^T W2
      gpq.seg(p, kS_Arena, tr.v_off, tr.n, 1, kS_Buf, f->w_off[l] + bl.r0, n, 0, tr.n);
      p = gpq.add(kS_T, q_off[j], s2, s2, s1);                     // Q = V_bl^T W1
      gpq.seg(p, kS_Arena, bl.v_off, bl.n, 1, kS_Buf, f->w_off[l] + tr.r0, n, 0, bl.n);
      p = gs.add(kS_T, s_off[j], s2, s2, s2, -1.0, 1.0);           // S = I - Q P
      gs.seg(p, kS_T, q_off[j], s2, 0, kS_T, p_off[j], s1, 0, s1);
      s_eye.push_back(EyeDesc{Ps + s_off[j], s2, s2});
      inv.push_back(GjProb{Ps + s_off[j], s2, s2, nullptr, f->buf + br, q, nullptr, nullptr});   // S^-1 -> C^-1[bl, bl]
      p = c1.add(kS_Buf, tr_off, q, s1, s2, -1.0);                 // C^-1[tr, bl] = -P S^-1
      c1.seg(p, kS_T, p_off[j], s1, 0, kS_Buf, br, q, 0, s2);
      p = c1.add(kS_Buf, bl_off, q, s2, s1, -1.0);                 // C^-1[bl, tr] = -S^-1 Q
      c1.seg(p, kS_Buf, br, q, 0, kS_T, q_off[j], s2, 0, s2);
      p = c2.add(kS_Buf, ci, q, s1, s1, -1.0, 1.0);                // C^-1[tr, tr] = I - P C^-1[bl, tr]
      c2.seg(p, kS_T, p_off[j], s1, 0, kS_Buf, bl_off, q, 0, s2);
    }
    gemm_f64_run(gpq, b, TileShape::M64N128, s);
    eye(s_eye, s);
    gemm_f64_run(gs, b, TileShape::M64N128, s, false);
    gj_inverse(inv, d_status, s);
    gemm_f64_run(c1, b, TileShape::M64N128, s, false);
    gemm_f64_run(c2, b, TileShape::M64N128, s, false);
    dev_free(Ps, s);
  }
  dev_free(tmp, s);
  int st = 0;
  HB_CUDA(cudaMemcpyAsync(&st, d_status, sizeof(int), cudaMemcpyDeviceToHost, s));
  HB_CUDA(cudaStreamSynchronize(s));
  cudaFreeAsync(d_status, s);
  f->last_use.settled();
  if (st) *status = INPUT_ERROR;
  return f;
}

void hodlr_solve(HodlrFactor &f, const double *B, int k, long long ldb, double *X,
                 long long ldx, cudaStream_t s) {
  if (k <= 0 || f.tree->g.n == 0) return;
  const InFlight use{f.last_use};
  SolvePlan &P = solve_plan(f, k, ldb, ldx, s);
  const GemmBases b = solver_bases(f, X, B, P.T, P.Z);
  gemm_plan_run(P.leaves, b, s);
  for (int l = f.tree->g.h - 1; l >= 0; --l) {
    gemm_plan_run(*P.vt[l], b, s);
    gemm_plan_run(*P.cz[l], b, s);
    gemm_plan_run(*P.wx[l], b, s);
  }
}

}  // namespace hb
