// HODLR x vector (one right-hand side, op N) on a device tree, the product
// behind multiply_vector (hmat_lib src/vector_algebra.c:131-197):
//   1. W_b = V_b^T x[columns of b] for every off-diagonal block of every
//      level in one launch;
//   2. y[leaf rows] = D x[leaf rows] + sum over levels U_b[rows] W_b in one
//      launch.
// Every stored double is read once, so both launches are bound by HBM, and on
// small trees by latency; what either needs is many loads in flight.
// Projections: an item is kCols columns of one V_b, by a whole CTA when the
// block has kWideRows rows or more and by one warp otherwise, each thread
// holding kCols x kRowsFlight loads; the items are listed once per tree,
// longest first.  Rows: a CTA per 32 rows of a leaf (256 contiguous bytes per
// column), its warps taking the columns of the leaf and of every U_b in turn,
// eight loads per lane in flight, summed over the warps in a fixed order.  The
// second launch starts while the first drains (programmatic launch) and does
// its leaf part before it waits for W.
// n = 32768, depth 8, 611 MB of leaves and factors: 479 -> 120 us (1.28 ->
// 5.1 TB/s of 6.55 measured) against a warp per column and one thread per
// row; n = 1024, depth 3, replayed from a graph: 18.4 -> 6.2 us.
#include <algorithm>

#include "dtree.h"
#include "products.h"

namespace hb {

// One work item of the projection launch: columns j0 .. j0 + cnt - 1 of V_b.
struct MvItem {
  int block, j0, cnt, w0;   // w0: where W_b starts
};

namespace {

constexpr int kProjThreads = 256;
constexpr int kProjWarps = kProjThreads / 32;
constexpr int kCols = 4;          // columns per item
constexpr int kRowsFlight = 4;    // rows per thread in flight (x kCols loads)
constexpr int kWideRows = 512;    // blocks at least this tall take a CTA per item
constexpr int kRowWarps = 16;
constexpr int kRowThreads = 32 * kRowWarps;
constexpr int kRowFlight = 8;     // columns per warp in flight
constexpr int kMaxDepth = 32;     // levels of a tree (2^h leaves)

// acc[c] += sum over r = r0, r0 + step, ... of V[r, c] x[r]
__device__ __forceinline__ void project_columns(const double *__restrict__ v, long long ld,
                                                const double *__restrict__ x, int n, int cnt,
                                                int r0, int step, double (&acc)[kCols]) {
  const double *col[kCols];
#pragma unroll
  for (int c = 0; c < kCols; ++c) col[c] = v + (long long)min(c, cnt - 1) * ld;
  for (int r = r0; r < n; r += step * kRowsFlight) {
    double xv[kRowsFlight], a[kRowsFlight][kCols];
#pragma unroll
    for (int u = 0; u < kRowsFlight; ++u) {
      const int i = r + u * step;
      const bool in = i < n;
      xv[u] = in ? x[i] : 0.0;
#pragma unroll
      for (int c = 0; c < kCols; ++c) a[u][c] = in ? col[c][i] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kRowsFlight; ++u)
#pragma unroll
      for (int c = 0; c < kCols; ++c) acc[c] = fma(a[u][c], xv[u], acc[c]);
  }
#pragma unroll
  for (int c = 0; c < kCols; ++c)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
}

// CTAs 0 .. nwide - 1 take one item each, the others one item per warp.
__global__ void __launch_bounds__(kProjThreads)
mv_project_kernel(const BlockDesc *__restrict__ blocks, const double *__restrict__ arena,
                  const double *__restrict__ x, const MvItem *__restrict__ items, int nwide,
                  int nitems, double *__restrict__ w) {
  cudaTriggerProgrammaticLaunchCompletion();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool wide = (int)blockIdx.x < nwide;
  const int it = wide ? blockIdx.x : nwide + ((int)blockIdx.x - nwide) * kProjWarps + warp;
  if (it >= nitems) return;   // whole warps of the last narrow CTA
  const MvItem I = items[it];
  const BlockDesc B = blocks[I.block];
  double acc[kCols] = {};
  project_columns(arena + B.v_off + (long long)I.j0 * B.n, B.n, x + B.c0, B.n, I.cnt,
                  wide ? threadIdx.x : lane, wide ? kProjThreads : 32, acc);
  if (!wide) {
#pragma unroll
    for (int c = 0; c < kCols; ++c)
      if (lane == c && c < I.cnt) w[I.w0 + I.j0 + c] = acc[c];
    return;
  }
  __shared__ double red[kProjWarps][kCols];
#pragma unroll
  for (int c = 0; c < kCols; ++c)
    if (lane == c) red[warp][c] = acc[c];
  __syncthreads();
  if ((int)threadIdx.x < I.cnt) {
    double sum = 0.0;
#pragma unroll
    for (int k = 0; k < kProjWarps; ++k) sum += red[k][threadIdx.x];
    w[I.w0 + I.j0 + threadIdx.x] = sum;
  }
}

// One segment of a row strip: sum over this warp's columns c of m[c ld] v[c].
__device__ __forceinline__ void row_columns(const double *__restrict__ m, long long ld,
                                            const double *v, int count, int warp,
                                            double (&acc)[4]) {
  for (int c0 = warp; c0 < count; c0 += kRowWarps * kRowFlight) {
    double a[kRowFlight], b[kRowFlight];
#pragma unroll
    for (int u = 0; u < kRowFlight; ++u) {
      const int c = c0 + u * kRowWarps;
      const bool in = c < count;
      a[u] = in ? m[c * ld] : 0.0;
      b[u] = in ? v[c] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kRowFlight; ++u) acc[u & 3] = fma(a[u], b[u], acc[u & 3]);
  }
}

__global__ void __launch_bounds__(kRowThreads)
mv_rows_kernel(const LeafDesc *__restrict__ leaves, const BlockDesc *__restrict__ blocks,
               int height, const double *__restrict__ arena, const double *__restrict__ x,
               const int *__restrict__ woff, const double *w, double *__restrict__ y) {
  __shared__ double red[kRowWarps][32];
  __shared__ const double *s_u[kMaxDepth];
  __shared__ int s_ld[kMaxDepth], s_s[kMaxDepth], s_w[kMaxDepth];
  const int i = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const LeafDesc L = leaves[i];
  const int r0 = 32 * blockIdx.y;
  if (r0 < L.m) {
    // descriptors of the leaf's block at every depth, one per thread: the
    // block whose rows hold leaf i is top-right if the leaf lies in the first
    // child of its depth-d ancestor, bottom-left if not
    if ((int)threadIdx.x < height) {
      const int d = threadIdx.x;
      const int b = 2 * ((1 << d) - 1 + (i >> (height - d))) + ((i >> (height - d - 1)) & 1);
      const BlockDesc B = blocks[b];
      s_u[d] = arena + B.u_off + (L.r0 - B.r0);
      s_ld[d] = B.m;
      s_s[d] = B.s;
      s_w[d] = woff[b];
    }
    const int r = min(r0 + lane, L.m - 1);
    double acc[4] = {};
    row_columns(arena + L.off + r, L.m, x + L.r0, L.m, warp, acc);
    __syncthreads();
    cudaGridDependencySynchronize();   // W is complete
    for (int d = height - 1; d >= 0; --d)
      row_columns(s_u[d] + r, s_ld[d], w + s_w[d], s_s[d], warp, acc);
    red[warp][lane] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    __syncthreads();
    if (warp == 0 && r0 + lane < L.m) {
      double sum = 0.0;
#pragma unroll
      for (int k = 0; k < kRowWarps; ++k) sum += red[k][lane];
      y[L.r0 + r0 + lane] = sum;
    }
  }
}

}  // namespace

void matvec_f64(DeviceTree &t, const double *x, double *y, cudaStream_t s) {
  const Geometry &g = t.g;
  if (g.n == 0) return;
  const int nblocks = g.nblock();
  HB_REQUIRE(g.h <= kMaxDepth, INPUT_ERROR, "matvec: tree too deep");
  {
    std::lock_guard<std::mutex> lk(t.plan_mutex);
    if (!t.mv_woff && nblocks > 0) {
      std::vector<int> woff(nblocks);
      std::vector<MvItem> items, narrow;
      long long total = 0;
      for (int b = 0; b < nblocks; ++b) {
        const BlockDesc &B = g.blocks[b];
        woff[b] = (int)total;
        if (B.n > 0)
          for (int j = 0; j < B.s; j += kCols)
            (B.n >= kWideRows ? items : narrow)
                .push_back(MvItem{b, j, std::min(kCols, B.s - j), (int)total});
        total += B.s;
      }
      HB_REQUIRE(total < (1LL << 31), INPUT_ERROR, "matvec: ranks sum past 2^31");
      // block order is top level first, so the longest items already lead
      t.mv_nwide = (int)items.size();
      items.insert(items.end(), narrow.begin(), narrow.end());
      t.mv_nitems = (int)items.size();
      const size_t wb = align_up(sizeof(int) * nblocks, 256), ib = sizeof(MvItem) * items.size();
      std::vector<char> host(wb + ib);
      std::copy(woff.begin(), woff.end(), (int *)host.data());
      std::copy(items.begin(), items.end(), (MvItem *)(host.data() + wb));
      if (!t.mv_w)
        device_alloc(&t.mv_w, sizeof(double) * std::max<long long>(total, 1));
      device_alloc(&t.mv_woff, host.size());
      t.mv_items = (MvItem *)((char *)t.mv_woff + wb);
      HB_CUDA(cudaMemcpyAsync(t.mv_woff, host.data(), host.size(), cudaMemcpyHostToDevice, s));
      HB_CUDA(cudaStreamSynchronize(s));
    }
  }
  if (t.mv_nitems > 0) {
    const int grid = t.mv_nwide + (t.mv_nitems - t.mv_nwide + kProjWarps - 1) / kProjWarps;
    mv_project_kernel<<<grid, kProjThreads, 0, s>>>(t.d_blocks, t.arena, x, t.mv_items, t.mv_nwide,
                                                    t.mv_nitems, t.mv_w);
    HB_LAUNCHED();
  }
  int mmax = 1;
  for (int m : g.leaf_m) mmax = std::max(mmax, m);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)g.nleaf(), (unsigned)((mmax + 31) / 32));
  cfg.blockDim = dim3(kRowThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // without a projection launch of this product in front, the launch before
  // could be anything: plain stream order
  cfg.numAttrs = t.mv_nitems > 0 ? 1 : 0;
  HB_CUDA(cudaLaunchKernelEx(&cfg, mv_rows_kernel, (const LeafDesc *)t.d_leaves,
                             (const BlockDesc *)t.d_blocks, g.h, (const double *)t.arena, x,
                             (const int *)t.mv_woff, (const double *)t.mv_w, y));
  HB_LAUNCHED();
}

}  // namespace hb
