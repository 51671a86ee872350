// Batched TSQR (Householder QR of 256-row chunks in registers, reduced
// up a tree of stacked R factors, explicit Q rebuilt top-down) plus the
// small utility kernels of the randomized compression: Gaussian test
// matrices, column norms.
//
// Replaces the dgeqrt factorisations of hmat_lib (src/hodlr_algebra.c:120,
// 126) and provides the orthonormal bases of the randomized range finder
// that stands in for dgesdd on large blocks (src/constructors.c:323).
#include <algorithm>
#include <chrono>

#include "dmma.cuh"
#include "gemm_f64.h"
#include "tsqr.h"

namespace hb {

namespace {

constexpr int kQT = 256;   // threads per CTA

struct QrChunk {
  double *A;
  long long lda;
  int rows, w;
  double *R;
  long long ldr;
};

struct MulChunk {
  double *Q;
  long long ldq;
  int rows, w;
  const double *M;
  long long ldm;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

constexpr int kQWarps = kQT / 32;
constexpr int kLdG = kPanel + 1;   // leading dimension of the reflectors' products
constexpr int kLdM = kPanel + 4;   // of M: fragment loads of a half-warp hit 16 banks
static_assert(kChunk == 32 * kQWarps && kPanel == 32, "a warp per 32 rows, 4 x 8 values per lane");

// Householder QR of one chunk (rows <= 256, w <= 32), LAPACK dlarfg
// convention: H_j = I - tau_j v_j v_j^T, v_j(j) = 1, beta_j = -sign(x0)||x||.
//
// The chunk lives in registers in the fragment layout of the FP64 tensor-core
// product: lane l of a warp holds rows l / 4 + 8 i (i < 4) of the warp's 32
// and columns 4 s + l % 4 (s < 8).  A step is bound by its latency (one
// reduction, a square root, two divisions), so it has a single barrier: the
// products of column j's tail with every column, itself included, are summed
// together, and the reflector is scaled afterwards.  The same products with
// the finished columns are v_j^T v_c, which make the block form
// Q = I - V T V^T: T^-1 has 1 / tau on the diagonal and v_l^T v_j above it, so
// M = T V_1^T comes from one triangular solve and Q's columns are
// [I; 0] - V M on the tensor cores, straight from V's registers.  The slots
// rotate by one every four columns, so column j is always in slot 0 and no
// register is indexed at run time.
// 1024 chunks of 256 x 32 (a panel of every block at n = 32768): 1092 us with the
// chunk in shared memory (one CTA per SM, five barriers a step), 191 us so.
__global__ void __launch_bounds__(kQT, 2) qr_chunk_kernel(const QrChunk *__restrict__ descs) {
  const QrChunk D = descs[blockIdx.x];
  __shared__ double red[2][kQWarps][kPanel];   // per warp: products with the columns by position
  __shared__ double rowj[2][kPanel];           // row j before its step, by position
  __shared__ double coef[kQWarps][kPanel];     // per warp: tau_j v_j^T a_c
  __shared__ double G[kPanel * kLdG];          // v_j^T v_c at [j][c], c < j
  __shared__ double M[kPanel * kLdM];          // V_1^T, then T V_1^T
  __shared__ double tau[kPanel];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = lane >> 2, cg = lane & 3, row0 = 32 * warp + rg;
  const int r = D.rows, w = D.w, k = min(r, w);

  double a[4][8];
#pragma unroll
  for (int s = 0; s < 8; ++s)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = row0 + 8 * i, c = 4 * s + cg;
      a[i][s] = (row < r && c < w) ? D.A[row + (long long)c * D.lda] : 0.0;
    }

  for (int j = 0; j < kPanel; ++j) {
    const int cj = j & 3, par = j & 1;
    if (j < k) {
      // x = rows below j of column j, for every lane of the row
      double x[4], d[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[i] = __shfl_sync(0xffffffffu, a[i][0], (lane & ~3) | cj);
        if (row0 + 8 * i <= j) x[i] = 0.0;
      }
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        d[s] = x[0] * a[0][s];
#pragma unroll
        for (int i = 1; i < 4; ++i) d[s] = fma(x[i], a[i][s], d[s]);
      }
      // summed over the eight row groups; lane l ends with slot l / 4, its
      // own column group: position l
#pragma unroll
      for (int b = 4; b >= 1; b >>= 1) {
        const bool hi = (rg & b) != 0;
#pragma unroll
        for (int q = 0; q < b; ++q) {
          const double send = hi ? d[q] : d[q + b], keep = hi ? d[q + b] : d[q];
          d[q] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * b);
        }
      }
      red[par][warp][lane] = d[0];
      if (warp == 0 && rg == (j & 7)) {   // row j's owners
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          const int i = j >> 3;
          rowj[par][4 * s + cg] = i == 0 ? a[0][s] : i == 1 ? a[1][s] : i == 2 ? a[2][s] : a[3][s];
        }
      }
      __syncthreads();   // the buffers of step j are written again in step j + 2
      double dp = 0.0;
#pragma unroll
      for (int q = 0; q < kQWarps; ++q) dp += red[par][q][lane];
      const double ajp = rowj[par][lane];
      const double sigma2 = __shfl_sync(0xffffffffu, dp, cj);
      const double x0 = __shfl_sync(0xffffffffu, ajp, cj);
      double beta = x0, t = 0.0, scale = 0.0;
      if (sigma2 > 0.0) {
        const double nrm = sqrt(fma(x0, x0, sigma2));
        beta = x0 >= 0.0 ? -nrm : nrm;
        t = (beta - x0) / beta;
        scale = 1.0 / (x0 - beta);
      }
      const int c = 4 * (((j >> 2) + rg) & 7) + cg;   // column at this lane's position
      const double g = fma(scale, dp, ajp);           // v_j^T a_c
      coef[warp][lane] = c > j ? t * g : 0.0;
      if (warp == 0) {
        if (c < j) G[j * kLdG + c] = g;
        if (lane == 0) tau[j] = t;
      }
      __syncwarp();
      double v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = row0 + 8 * i == j ? 1.0 : x[i] * scale;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const double wv = coef[warp][4 * s + cg];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i][s] = fma(-v[i], wv, a[i][s]);
      }
      if (cg == cj) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = row0 + 8 * i;
          if (row < w)
            D.R[row + (long long)j * D.ldr] = row < j ? a[i][0] : row == j ? beta : 0.0;
          a[i][0] = v[i];
        }
      }
    } else {
      // no reflector: a column past the rows (its R entries are final) or
      // past the panel (zero)
      if (cg == cj) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = row0 + 8 * i;
          if (j < w && row < w) D.R[row + (long long)j * D.ldr] = row < k ? a[i][0] : 0.0;
          a[i][0] = 0.0;
        }
      }
      if (warp == 0) {
        if (lane < j) G[j * kLdG + lane] = 0.0;
        if (lane == 0) tau[j] = 0.0;
      }
    }
    if (cj == 3) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const double first = a[i][0];
#pragma unroll
        for (int s = 0; s < 7; ++s) a[i][s] = a[i][s + 1];
        a[i][7] = first;
      }
    }
  }

  // M = T V_1^T by back substitution, a lane per column, in two halves of 16
  // rows held in registers (warp 0 owns the first 32 rows and wrote G, tau)
  if (warp == 0) {
#pragma unroll
    for (int s = 0; s < 8; ++s)
#pragma unroll
      for (int i = 0; i < 4; ++i) M[(4 * s + cg) * kLdM + rg + 8 * i] = a[i][s];
    __syncwarp();
#pragma unroll
    for (int h = 1; h >= 0; --h) {
      double m[16];
#pragma unroll
      for (int l = 0; l < 16; ++l) m[l] = M[(16 * h + l) * kLdM + lane];
      if (h == 0)
        for (int j = 16; j < 32; ++j) {
          const double mj = M[j * kLdM + lane];
#pragma unroll
          for (int l = 0; l < 16; ++l) m[l] = fma(-G[j * kLdG + l], mj, m[l]);
        }
#pragma unroll
      for (int j = 15; j >= 0; --j) {
        m[j] *= tau[16 * h + j];
#pragma unroll
        for (int l = 0; l < j; ++l)
          m[l] = fma(-G[(16 * h + j) * kLdG + 16 * h + l], m[j], m[l]);
      }
#pragma unroll
      for (int l = 0; l < 16; ++l) M[(16 * h + l) * kLdM + lane] = m[l];
    }
  }
  __syncthreads();
  // Q = [I; 0] - V M (M upper triangular)
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    double q[4][2] = {};
#pragma unroll
    for (int s = 0; s < 2 * nt + 2; ++s) {
      const double b = M[(4 * s + cg) * kLdM + 8 * nt + rg];
#pragma unroll
      for (int i = 0; i < 4; ++i) dmma884(q[i], a[i][s], b);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = row0 + 8 * i, c = 8 * nt + 2 * cg + h;
        if (row < r && c < w)
          D.A[row + (long long)c * D.lda] = (row == c ? 1.0 : 0.0) - q[i][h];
      }
  }
}

// Q (rows x w) <- Q M (M: w x w)
__global__ void __launch_bounds__(kQT) mul_chunk_kernel(const MulChunk *__restrict__ descs) {
  const MulChunk D = descs[blockIdx.x];
  __shared__ double M[kPanel * kPanel];
  const int tid = threadIdx.x, w = D.w;
  for (int e = tid; e < w * w; e += kQT) M[e] = D.M[(e % w) + (long long)(e / w) * D.ldm];
  __syncthreads();
  for (int i = tid; i < D.rows; i += kQT) {
    double q[kPanel];
#pragma unroll
    for (int l = 0; l < kPanel; ++l) q[l] = l < w ? D.Q[i + (long long)l * D.ldq] : 0.0;
    for (int c = 0; c < w; ++c) {
      double acc = 0.0;
#pragma unroll
      for (int l = 0; l < kPanel; ++l) acc = fma(q[l], l < w ? M[l + c * w] : 0.0, acc);
      D.Q[i + (long long)c * D.ldq] = acc;
    }
  }
}

__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ULL;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
  return x ^ (x >> 31);
}

__global__ void gaussian_kernel(const RandDesc *__restrict__ descs, unsigned long long seed) {
  const RandDesc D = descs[blockIdx.y];
  const unsigned long long base = splitmix64(seed ^ splitmix64(D.id + 0x632BE59BD9B4E019ULL));
  const long long total = (long long)D.rows * D.cols;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const unsigned long long h1 = splitmix64(base + (unsigned long long)e);
    const unsigned long long h2 = splitmix64(h1);
    const double u1 = ((double)(h1 >> 11) + 1.0) * 0x1.0p-53;   // (0, 1]
    const double u2 = (double)(h2 >> 11) * 0x1.0p-53;           // [0, 1)
    const double z = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
    const long long i = e % D.rows, j = e / D.rows;
    D.X[i + j * D.ld] = z;
  }
}

__global__ void colnorm_kernel(const NormDesc *__restrict__ descs) {
  const NormDesc D = descs[blockIdx.y];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int c = blockIdx.x * nw + warp; c < D.cols; c += gridDim.x * nw) {
    const double *x = D.X + (long long)c * D.ld;
    double s = 0.0;
    for (int i = lane; i < D.rows; i += 32) s = fma(x[i], x[i], s);
    s = warp_sum(s);
    if (lane == 0) D.out[c] = s;
  }
}

template <class T>
T *upload(const std::vector<T> &v, cudaStream_t s) {
  T *d = nullptr;
  pool_alloc(&d, sizeof(T) * std::max<size_t>(v.size(), 1), s);
  h2d_async(d, v.data(), sizeof(T) * v.size(), s);
  return d;
}

constexpr double kCleanOrth = 1e-5;   // see panel_clean()

__global__ void panel_clean_kernel(const CleanDesc *__restrict__ descs, double rel) {
  const CleanDesc D = descs[blockIdx.y];
  static_assert(kPanel == 32, "a lane per column");
  __shared__ unsigned drop;
  if (threadIdx.x < 32) {
    const int c = threadIdx.x;
    const double *R = D.R + (long long)c * D.ldr;
    double scale2 = c < D.w ? D.prenorm2[c] : 0.0, top = 0.0, diag = 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      scale2 = fmax(scale2, __shfl_xor_sync(0xffffffffu, scale2, o));
    if (c < D.w) {
      for (int i = 0; i < c; ++i) top = fmax(top, fabs(R[i]));
      diag = fabs(R[c]);
    }
    const bool zero = c < D.w && (!(diag > rel * sqrt(scale2)) ||
                                  (D.later && diag <= kCleanOrth * top));
    const unsigned mask = __ballot_sync(0xffffffffu, zero);
    if (c == 0) drop = mask;
  }
  __syncthreads();
  for (unsigned m = drop; m; m &= m - 1) {
    const int c = __ffs(m) - 1;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < D.rows; i += gridDim.x * blockDim.x)
      D.Q[i + (long long)c * D.ldq] = 0.0;
  }
}

}  // namespace

void panel_clean(const std::vector<CleanDesc> &descs, double rel, cudaStream_t s) {
  if (descs.empty()) return;
  CleanDesc *d = upload(descs, s);
  for (size_t off = 0; off < descs.size(); off += 65535) {
    dim3 grid(8, (unsigned)std::min<size_t>(65535, descs.size() - off));
    panel_clean_kernel<<<grid, 256, 0, s>>>(d + off, rel);
    HB_LAUNCHED();
  }
  cudaFreeAsync(d, s);
}

// The chunk lists of every level of a batch of TSQR problems, uploaded, with
// the scratch of the stacked R factors: made once, run any number of times
// (the panels' contents may change between runs, not their addresses).
struct TsqrPlan {
  std::vector<QrChunk *> up;        // per level: QR of the chunks
  std::vector<int> up_n;
  std::vector<MulChunk *> down;     // per level (top first): Q times the parent's Q
  std::vector<int> down_n;
  double *buf = nullptr;
  cudaStream_t stream = nullptr;
  ~TsqrPlan() {
    for (auto *p : up) cudaFreeAsync(p, stream);
    for (auto *p : down) cudaFreeAsync(p, stream);
    if (buf) cudaFreeAsync(buf, stream);
  }
};

void TsqrPlanDeleter::operator()(TsqrPlan *p) const { delete p; }

std::unique_ptr<TsqrPlan, TsqrPlanDeleter> tsqr_plan(const std::vector<TsqrProb> &probs,
                                                     cudaStream_t s) {
  struct Clock {
    std::chrono::steady_clock::time_point t = std::chrono::steady_clock::now();
    ~Clock() {
      plan_host_ms() +=
          std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t).count();
    }
  } clock;
  std::unique_ptr<TsqrPlan, TsqrPlanDeleter> plan(new TsqrPlan);
  plan->stream = s;
  if (probs.empty()) return plan;
  // level structure of every problem: level 0 is the panel itself, level
  // l + 1 stacks the w x w R factors of level l's chunks
  struct Level {
    double *A;
    long long lda;
    int rows;
    int nchunks;
  };
  // levels of problem p: lev[lo[p] .. lo[p + 1]) (flat, no per-problem
  // allocations: a round of the build makes plans for thousands of panels)
  constexpr int kMaxLevels = 16;
  std::vector<Level> lev;
  std::vector<int> lo(probs.size() + 1, 0);
  lev.reserve(probs.size() * 3);
  long long scratch = 0;
  std::vector<long long> stack_off;   // per level >= 1, same indexing as lev
  stack_off.reserve(probs.size() * 3);
  for (size_t p = 0; p < probs.size(); ++p) {
    const TsqrProb &P = probs[p];
    HB_REQUIRE(P.w >= 1 && P.w <= kPanel, INPUT_ERROR, "TSQR panel wider than 32 columns");
    lo[p] = (int)lev.size();
    int rows = P.m;
    long long off = -1;   // stacked-R scratch of this level (-1: the panel itself)
    for (int l = 0; l < kMaxLevels; ++l) {
      const int nch = std::max(1, (rows + kChunk - 1) / kChunk);
      lev.push_back(Level{nullptr, 0, rows, nch});
      stack_off.push_back(off);
      if (nch == 1) break;
      rows = nch * P.w;
      off = scratch;
      scratch += align_up((long long)rows * P.w);
    }
  }
  lo[probs.size()] = (int)lev.size();
  if (scratch) pool_alloc(&plan->buf, scratch * sizeof(double), s);
  int max_levels = 0;
  for (size_t p = 0; p < probs.size(); ++p) {
    Level *L = lev.data() + lo[p];
    const int nl = lo[p + 1] - lo[p];
    L[0].A = probs[p].Y;
    L[0].lda = probs[p].ldy;
    for (int l = 1; l < nl; ++l) {
      L[l].A = plan->buf + stack_off[lo[p] + l];
      L[l].lda = L[l].rows;
    }
    max_levels = std::max(max_levels, nl);
  }
  // up-sweep
  for (int l = 0; l < max_levels; ++l) {
    std::vector<QrChunk> chunks;
    for (size_t p = 0; p < probs.size(); ++p) {
      const Level *L = lev.data() + lo[p];
      const int nl = lo[p + 1] - lo[p];
      if (l >= nl) continue;
      const int w = probs[p].w;
      for (int c = 0; c < L[l].nchunks; ++c) {
        QrChunk q;
        q.A = L[l].A + (long long)c * kChunk;
        q.lda = L[l].lda;
        q.rows = std::min(kChunk, L[l].rows - c * kChunk);
        q.w = w;
        if (l + 1 < nl) {
          q.R = L[l + 1].A + (long long)c * w;
          q.ldr = L[l + 1].lda;
        } else {
          q.R = probs[p].R;
          q.ldr = probs[p].ldr;
        }
        if (q.rows > 0) chunks.push_back(q);
      }
    }
    plan->up.push_back(chunks.empty() ? nullptr : upload(chunks, s));
    plan->up_n.push_back((int)chunks.size());
  }
  // down-sweep: every chunk's Q times its block of the parent's Q
  for (int l = max_levels - 2; l >= 0; --l) {
    std::vector<MulChunk> chunks;
    for (size_t p = 0; p < probs.size(); ++p) {
      const Level *L = lev.data() + lo[p];
      const int nl = lo[p + 1] - lo[p];
      if (l + 1 >= nl) continue;
      const int w = probs[p].w;
      for (int c = 0; c < L[l].nchunks; ++c) {
        MulChunk mc;
        mc.Q = L[l].A + (long long)c * kChunk;
        mc.ldq = L[l].lda;
        mc.rows = std::min(kChunk, L[l].rows - c * kChunk);
        mc.w = w;
        mc.M = L[l + 1].A + (long long)c * w;
        mc.ldm = L[l + 1].lda;
        if (mc.rows > 0) chunks.push_back(mc);
      }
    }
    plan->down.push_back(chunks.empty() ? nullptr : upload(chunks, s));
    plan->down_n.push_back((int)chunks.size());
  }
  return plan;
}

void tsqr_run(const TsqrPlan &plan, cudaStream_t s) {
  for (size_t l = 0; l < plan.up.size(); ++l)
    for (int off = 0; off < plan.up_n[l]; off += 65535) {
      const int cnt = std::min(65535, plan.up_n[l] - off);
      qr_chunk_kernel<<<cnt, kQT, 0, s>>>(plan.up[l] + off);
      HB_LAUNCHED();
    }
  for (size_t l = 0; l < plan.down.size(); ++l)
    for (int off = 0; off < plan.down_n[l]; off += 65535) {
      const int cnt = std::min(65535, plan.down_n[l] - off);
      mul_chunk_kernel<<<cnt, kQT, 0, s>>>(plan.down[l] + off);
      HB_LAUNCHED();
    }
}

void tsqr_batched(const std::vector<TsqrProb> &probs, cudaStream_t s) {
  if (probs.empty()) return;
  auto plan = tsqr_plan(probs, s);
  tsqr_run(*plan, s);
}

void gaussian_fill(const std::vector<RandDesc> &descs, unsigned long long seed, cudaStream_t s) {
  if (descs.empty()) return;
  RandDesc *d = upload(descs, s);
  for (size_t off = 0; off < descs.size(); off += 65535) {
    dim3 grid(64, (unsigned)std::min<size_t>(65535, descs.size() - off));
    gaussian_kernel<<<grid, 256, 0, s>>>(d + off, seed);
    HB_LAUNCHED();
  }
  cudaFreeAsync(d, s);
}

void column_norms2(const std::vector<NormDesc> &descs, cudaStream_t s) {
  if (descs.empty()) return;
  NormDesc *d = upload(descs, s);
  for (size_t off = 0; off < descs.size(); off += 65535) {
    dim3 grid(8, (unsigned)std::min<size_t>(65535, descs.size() - off));
    colnorm_kernel<<<grid, 256, 0, s>>>(d + off);
    HB_LAUNCHED();
  }
  cudaFreeAsync(d, s);
}

}  // namespace hb
