// Sketch products Y = A S with the test matrices S = H M of sketch.h.
//
// A column group of 64 contributes FWHT(d . A(row, group)) . e to a row of
// A H: 6 additions per entry for the transform and one to accumulate, instead
// of the 64 multiply-adds of a GEMM with 64 columns, so the product is bound
// by reading A instead of by the FP64 tensor pipe; M follows once per row.  A CTA takes 64 rows and a
// run of column groups; two threads share a row: the transform's first stage
// (the sums or the differences of entries 32 apart) splits it into two
// independent 32-point transforms of 32 registers, each with 32 accumulators.
// 64 x 64 tiles come through a ring of three stages (cp.async, 16-byte copies
// where the block's columns allow it); two CTAs per SM keep 128 KB of copies
// in flight.  The rounds of an n = 32768 build (height 7, tolerance 1e-8, 78 GB
// of A): 12.6 ms, where the GEMM took 34; the build 139 -> 116 ms.
#include "sketch.h"

#include <algorithm>
#include <cmath>

namespace hb {

namespace {

constexpr int kRows = 64;     // rows of a tile, two threads each
constexpr int kGroup = 64;    // columns of a tile: one transform
constexpr int kStages = 3;
constexpr int kThreads = 2 * kRows;
constexpr int kTile = kRows * kGroup;
constexpr int kSmem = kStages * kTile * (int)sizeof(double);

// One block and 64 of its columns of S; items [first, first + row tiles x
// splits) of the launch, the splits of a row tile next to one another.
struct Job {
  const double *A;
  double *Y;
  long long lda, ldy;
  const double *M;
  unsigned long long key;
  int r0, c0, m, n, w;
  int first, splits, vec;
};

__host__ __device__ inline unsigned long long mix64(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ULL;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
  return x ^ (x >> 31);
}

// Key of columns [64 part, 64 part + 64) of S; the signs of group g of H are
// the bits of mix64(key + 2 g) (rows) and mix64(key + 2 g + 1) (columns).
unsigned long long part_key(unsigned long long seed, unsigned long long id, int part) {
  return mix64(mix64(seed ^ mix64(id + 0x632BE59BD9B4E019ULL)) + (unsigned long long)part);
}

// v with its sign flipped when bit `bit` of `signs` is set
__device__ __forceinline__ double flip(double v, unsigned signs, int bit) {
  return __hiloint2double(__double2hiint(v) ^ (int)((signs << (31 - bit)) & 0x80000000u),
                          __double2loint(v));
}

__device__ __forceinline__ void copy_async(double *smem, const double *g, int bytes, bool vec) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  if (vec)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(g), "r"(bytes));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(g), "r"(bytes));
}

// Columns [64 g, 64 g + 64) of rows [row0, row0 + 64) into tile[column][row],
// zero outside the block.
template <bool GEN>
__device__ __forceinline__ void load_tile(double *tile, const Job &J, const KernelSpec &gen,
                                          int row0, int g) {
  const int c0 = g * kGroup;
  if (GEN) {
    for (int e = threadIdx.x; e < kTile; e += kThreads) {
      const int r = row0 + e % kRows, c = c0 + e / kRows;
      tile[e] = r < J.m && c < J.n ? kernel_entry(gen, J.r0 + r, J.c0 + c) : 0.0;
    }
    return;
  }
  if (J.vec) {
    const int r = row0 + 2 * (threadIdx.x % (kRows / 2)), c = threadIdx.x / (kRows / 2);
    const int bytes = max(0, min(16, 8 * (J.m - r)));
    const double *src = J.A + r + (long long)(c0 + c) * J.lda;
    constexpr int kStep = kThreads / (kRows / 2);
#pragma unroll
    for (int i = 0; i < kGroup / kStep; ++i) {
      const int b = c0 + c + i * kStep < J.n ? bytes : 0;
      copy_async(tile + (c + i * kStep) * kRows + r - row0,
                 b ? src + (long long)i * kStep * J.lda : J.A, b, true);
    }
  } else {
    const int r = row0 + threadIdx.x % kRows, c = threadIdx.x / kRows;
    const double *src = J.A + r + (long long)(c0 + c) * J.lda;
    constexpr int kStep = kThreads / kRows;
#pragma unroll 8
    for (int i = 0; i < kGroup / kStep; ++i) {
      const int b = r < J.m && c0 + c + i * kStep < J.n ? 8 : 0;
      copy_async(tile + (c + i * kStep) * kRows + r - row0,
                 b ? src + (long long)i * kStep * J.lda : J.A, b, false);
    }
  }
}

template <bool GEN>
__global__ void __launch_bounds__(kThreads, 2)
    sketch_kernel(const Job *__restrict__ jobs, int njobs, KernelSpec gen) {
  extern __shared__ double ring[];
  // the job of this CTA: the last one that starts at or before it
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (jobs[mid].first <= (int)blockIdx.x)
      lo = mid;
    else
      hi = mid - 1;
  }
  const Job J = jobs[lo];
  const int item = (int)blockIdx.x - J.first;
  const int row0 = item / J.splits * kRows, part = item % J.splits;
  const int groups = (J.n + kGroup - 1) / kGroup;
  const int g0 = (int)((long long)groups * part / J.splits);
  const int g1 = (int)((long long)groups * (part + 1) / J.splits);
  const int r = threadIdx.x % kRows, half = threadIdx.x / kRows;

  double acc[32];
#pragma unroll
  for (int t = 0; t < 32; ++t) acc[t] = 0.0;

#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (g0 + s < g1) load_tile<GEN>(ring + s * kTile, J, gen, row0, g0 + s);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  int stage = 0;
  for (int g = g0; g < g1; ++g) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2));
    __syncthreads();
    // the stage of tile g - 1, which every thread has finished with
    const int ahead = stage == 0 ? kStages - 1 : stage - 1;
    if (g + kStages - 1 < g1)
      load_tile<GEN>(ring + ahead * kTile, J, gen, row0, g + kStages - 1);
    asm volatile("cp.async.commit_group;\n" ::);

    const double *x = ring + stage * kTile + r;
    const unsigned long long d = mix64(J.key + 2 * (unsigned long long)g);
    const unsigned long long e = mix64(J.key + 2 * (unsigned long long)g + 1);
    const unsigned d0 = (unsigned)d, d1 = (unsigned)(d >> 32) ^ (half ? 0xFFFFFFFFu : 0u);
    const unsigned eh = (unsigned)(half ? e >> 32 : e);
    double v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i)
      v[i] = flip(x[i * kRows], d0, i) + flip(x[(i + 32) * kRows], d1, i);
#pragma unroll
    for (int len = 16; len > 0; len /= 2)
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (!(i & len)) {
          const double p = v[i], q = v[i + len];
          v[i] = p + q;
          v[i + len] = p - q;
        }
#pragma unroll
    for (int t = 0; t < 32; ++t) acc[t] += flip(v[t], eh, t);
    stage = stage == kStages - 1 ? 0 : stage + 1;
  }

  // rows of A H (ring[t][row]) times M (ms[t][column]), 32 columns a thread
  __syncthreads();
  double *ms = ring + kTile;
#pragma unroll
  for (int t = 0; t < 32; ++t) ring[(32 * half + t) * kRows + r] = acc[t];
  for (int e = threadIdx.x; e < kGroup * kGroup; e += kThreads) {
    const int t = e % kGroup, c = e / kGroup;
    ms[t * kGroup + c] = J.M[e];
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < 32; ++t) acc[t] = 0.0;
#pragma unroll 2
  for (int t = 0; t < kGroup; ++t) {
    const double y = ring[t * kRows + r];
    const double2 *g = reinterpret_cast<const double2 *>(ms + t * kGroup + 32 * half);
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const double2 q = g[c];
      acc[2 * c] = fma(y, q.x, acc[2 * c]);
      acc[2 * c + 1] = fma(y, q.y, acc[2 * c + 1]);
    }
  }

  if (row0 + r >= J.m) return;
  double *y = J.Y + row0 + r + (long long)(32 * half) * J.ldy;
  const int cols = J.w - 32 * half;
#pragma unroll
  for (int t = 0; t < 32; ++t)
    if (t < cols) {
      if (J.splits == 1)
        y[(long long)t * J.ldy] = acc[t];
      else
        atomicAdd(y + (long long)t * J.ldy, acc[t]);
    }
}

struct FillJob {
  double *X;
  long long ld;
  const double *M;
  unsigned long long key;
  int rows, cols;
};

// A thread per column of S: the same transform down e . M, 64 rows at a time.
__global__ void __launch_bounds__(kGroup) sketch_fill_kernel(const FillJob *__restrict__ jobs) {
  const FillJob F = jobs[blockIdx.y];
  const int c = threadIdx.x;
  if (c >= F.cols) return;
  for (int g = blockIdx.x; g * kGroup < F.rows; g += gridDim.x) {
    const unsigned long long d = mix64(F.key + 2 * (unsigned long long)g);
    const unsigned long long e = mix64(F.key + 2 * (unsigned long long)g + 1);
    double v[kGroup];
#pragma unroll
    for (int t = 0; t < kGroup; ++t)
      v[t] = flip(F.M[t + c * kGroup], (unsigned)(t < 32 ? e : e >> 32), t % 32);
#pragma unroll
    for (int len = kGroup / 2; len > 0; len /= 2)
#pragma unroll
      for (int i = 0; i < kGroup; ++i)
        if (!(i & len)) {
          const double p = v[i], q = v[i + len];
          v[i] = p + q;
          v[i + len] = p - q;
        }
    double *x = F.X + g * kGroup + (long long)c * F.ld;
    const int rows = F.rows - g * kGroup;
#pragma unroll
    for (int j = 0; j < kGroup; ++j)
      if (j < rows) x[j] = flip(v[j], (unsigned)(j < 32 ? d : d >> 32), j % 32);
  }
}

template <class T>
T *upload(const std::vector<T> &v, cudaStream_t s) {
  T *d = nullptr;
  pool_alloc(&d, sizeof(T) * v.size(), s);
  h2d_async(d, v.data(), sizeof(T) * v.size(), s);
  return d;
}

}  // namespace

std::vector<double> sketch_mixer(unsigned long long seed) {
  // Gram-Schmidt, twice, of a Gaussian matrix (Box-Muller)
  std::vector<double> M(kGroup * kGroup);
  const unsigned long long base = mix64(seed ^ 0x632BE59BD9B4E019ULL);
  for (int e = 0; e < kGroup * kGroup; ++e) {
    const unsigned long long h1 = mix64(base + (unsigned long long)e), h2 = mix64(h1);
    const double u1 = ((double)(h1 >> 11) + 1.0) * 0x1.0p-53, u2 = (double)(h2 >> 11) * 0x1.0p-53;
    M[e] = std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
  }
  for (int c = 0; c < kGroup; ++c) {
    double *x = M.data() + c * kGroup;
    for (int rep = 0; rep < 2; ++rep)
      for (int p = 0; p < c; ++p) {
        const double *q = M.data() + p * kGroup;
        double dot = 0.0;
        for (int i = 0; i < kGroup; ++i) dot += q[i] * x[i];
        for (int i = 0; i < kGroup; ++i) x[i] -= dot * q[i];
      }
    double norm = 0.0;
    for (int i = 0; i < kGroup; ++i) norm += x[i] * x[i];
    norm = std::sqrt(norm);
    for (int i = 0; i < kGroup; ++i) x[i] /= norm;
  }
  return M;
}

void sketch_multiply(const std::vector<SketchDesc> &descs, const double *M,
                     const KernelSpec *gen, unsigned long long seed, cudaStream_t stream) {
  // A row tile's columns are split so that the launch has about six items for
  // each of the resident CTAs, two an SM (a launch of the last rounds has few row
  // tiles, of wide blocks), but no item has less than 8 column groups: an
  // item's partial sums are 32 KB of atomics against 32 KB of A per group.
  constexpr int kWaves = 6, kMinGroups = 8;
  const long long resident = 2LL * num_sms();
  long long tiles = 0;
  for (const SketchDesc &D : descs)
    tiles += (long long)((D.m + kRows - 1) / kRows) * ((D.n + kGroup - 1) / kGroup) *
             ((D.w + kGroup - 1) / kGroup);
  const int per = (int)std::max<long long>(kMinGroups, tiles / (resident * kWaves));
  std::vector<Job> jobs;
  long long items = 0;
  auto launch = [&]() {
    if (jobs.empty()) return;
    Job *d = upload(jobs, stream);
    if (gen) {
      HB_CUDA(cudaFuncSetAttribute(sketch_kernel<true>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
      sketch_kernel<true><<<(unsigned)items, kThreads, kSmem, stream>>>(d, (int)jobs.size(), *gen);
    } else {
      HB_CUDA(cudaFuncSetAttribute(sketch_kernel<false>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
      sketch_kernel<false>
          <<<(unsigned)items, kThreads, kSmem, stream>>>(d, (int)jobs.size(), KernelSpec());
    }
    HB_LAUNCHED();
    cudaFreeAsync(d, stream);
    jobs.clear();
    items = 0;
  };
  for (const SketchDesc &D : descs) {
    if (D.m <= 0 || D.n <= 0) continue;
    const int row_tiles = (D.m + kRows - 1) / kRows, groups = (D.n + kGroup - 1) / kGroup;
    for (int p = 0; p * kGroup < D.w; ++p) {
      Job J;
      J.A = D.A;
      J.lda = D.lda;
      J.r0 = D.r0;
      J.c0 = D.c0;
      J.m = D.m;
      J.n = D.n;
      J.w = std::min(kGroup, D.w - p * kGroup);
      J.Y = D.Y + (long long)p * kGroup * D.ldy;
      J.ldy = D.ldy;
      J.M = M;
      J.key = part_key(seed, D.id, p);
      J.splits = (groups + per - 1) / per;
      J.vec = !gen && (size_t)D.A % 16 == 0 && D.lda % 2 == 0;
      if (items + (long long)row_tiles * J.splits > (1LL << 30)) launch();
      J.first = (int)items;
      items += (long long)row_tiles * J.splits;
      jobs.push_back(J);
    }
  }
  launch();
}

void sketch_fill(const std::vector<SketchFill> &descs, const double *M,
                 unsigned long long seed, cudaStream_t stream) {
  std::vector<FillJob> jobs;
  for (const SketchFill &D : descs)
    for (int p = 0; p * kGroup < D.cols; ++p)
      jobs.push_back(FillJob{D.X + (long long)p * kGroup * D.ld, D.ld,
                             M, part_key(seed, D.id, p), D.rows, std::min(kGroup, D.cols - p * kGroup)});
  if (jobs.empty()) return;
  FillJob *d = upload(jobs, stream);
  for (size_t off = 0; off < jobs.size(); off += 65535) {
    dim3 grid(64, (unsigned)std::min<size_t>(65535, jobs.size() - off));
    sketch_fill_kernel<<<grid, kGroup, 0, stream>>>(d + off);
    HB_LAUNCHED();
  }
  cudaFreeAsync(d, stream);
}

}  // namespace hb
