// FP64 variable-batched segmented GEMM for sm_100a.
//
// Three kernels (option gemm_f64_engine): on the FP64 tensor cores (DMMA) one with
// loader warps beside the MMA warps (default, last below) and one whose warps do
// both (generated operands, 256-column tiles, 16-deep stages), and a CUDA-core
// DFMA kernel: 256 threads, a BM x BN output tile per CTA
// (128 x 64, 64 x 128, 64 x 64, 32 x 128 or 32 x 256), K advanced 16 at a time through a two-stage
// cp.async pipeline (8-byte copies with zero fill, so any leading dimension
// and any offset work), 32 accumulators per thread, operands read from shared
// memory as double2.  FP64 has no tcgen05 path; this is the FP64 roofline
// kernel (B200: 64 DFMA / clock / SM).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>

#include "dmma.cuh"
#include "gemm_f64.h"

namespace hb {

int gemm_f64_engine() { return (int)option("gemm_f64_engine", 2); }

double &gemm_flops_counter() {
  static thread_local double flops = 0.0;
  return flops;
}

double &plan_host_ms() {
  static thread_local double ms = 0.0;
  return ms;
}

namespace {

constexpr int kBK = 16;
constexpr int kThreads = 256;

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem, bool pred) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int bytes = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// bases.p[i] for a runtime i without copying the launch argument array to
// local memory (a chain of selects on the constant-bank values)
__device__ __forceinline__ double *base_ptr(const GemmBases &b, int i) {
  static_assert(kGemmBases == 6, "base_ptr selects among six slots");
  double *p = b.p[0];
  p = i == 1 ? b.p[1] : p;
  p = i == 2 ? b.p[2] : p;
  p = i == 3 ? b.p[3] : p;
  p = i == 4 ? b.p[4] : p;
  p = i == 5 ? b.p[5] : p;
  return p;
}

struct KIter {
  int si;      // segment index (absolute)
  int kk;      // position inside the segment
  int le;      // end of the valid range inside the segment
  int kbase;   // concatenated-K position of the segment start
};

template <int BM, int BN>
struct Smem {
  static constexpr int LDA = BM + 2;
  static constexpr int LDB = BN + 2;
  static constexpr size_t bytes = sizeof(double) * 2 * kBK * (LDA + LDB);
};

template <int BM, int BN>
__global__ void __launch_bounds__(kThreads, 2)
gemm_f64_kernel(const GemmSeg *__restrict__ segs, const GemmProb *__restrict__ probs,
                const GemmTile *__restrict__ tiles, GemmBases bases) {
  constexpr int TM = BM / 16, TN = BN / 16;
  constexpr int LDA = Smem<BM, BN>::LDA, LDB = Smem<BM, BN>::LDB;
  extern __shared__ __align__(16) double smem[];
  double *As = smem;                        // [2][kBK][LDA]
  double *Bs = smem + 2 * kBK * LDA;        // [2][kBK][LDB]

  const GemmTile tile = tiles[blockIdx.x];
  const GemmProb P = probs[tile.prob];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int seg_end = P.seg0 + P.nseg;

  double acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0;

  auto settle = [&](KIter &it) {
    while (it.si < seg_end) {
      const int K = segs[it.si].K;
      const int ls = max(tile.k0 - it.kbase, 0);
      const int le = min(tile.k1 - it.kbase, K);
      if (ls < le) {
        it.kk = ls;
        it.le = le;
        return;
      }
      it.kbase += K;
      ++it.si;
    }
  };
  auto advance = [&](KIter &it) {
    it.kk += kBK;
    if (it.kk >= it.le) {
      it.kbase += segs[it.si].K;
      ++it.si;
      settle(it);
    }
  };

  // One operand element into shared memory: copied from global memory, or
  // computed when the segment's operand is a generated kernel matrix (stored
  // element (row, col) of the block at gen_offset(row0, col0)).
  auto stage = [&](double *dst, bool gen, const double *base, long long off, long long row,
                   long long col, long long ld, bool p) {
    if (gen) {
      *dst = p ? kernel_entry(bases.gen, (int)(off >> 32) + (int)row,
                              (int)(off & 0xffffffffLL) + (int)col)
               : 0.0;
    } else {
      cp_async8(dst, p ? base + off + row + col * ld : base, p);
    }
  };

  auto load = [&](int buf, const KIter &it) {
    const GemmSeg S = segs[it.si];
    const bool ga = S.abase == kGenSlot, gb = S.bbase == kGenSlot;
    const double *A = ga ? nullptr : base_ptr(bases, S.abase);
    const double *B = gb ? nullptr : base_ptr(bases, S.bbase);
    double *as = As + buf * kBK * LDA;
    double *bs = Bs + buf * kBK * LDB;
    const int kk = it.kk, kend = it.le;
    if (S.ta == 0) {
      constexpr int KS = kThreads / BM;
      const int m = tid % BM;
      const bool mok = (tile.m0 + m) < P.M;
#pragma unroll
      for (int i = 0; i < BM * kBK / kThreads; ++i) {
        const int k = tid / BM + KS * i;
        const bool p = mok && (kk + k) < kend;
        stage(as + k * LDA + m, ga, A, S.a_off, tile.m0 + m, kk + k, S.lda, p);
      }
    } else {
      const int k = tid & 15;
      const bool kok = (kk + k) < kend;
#pragma unroll
      for (int i = 0; i < BM / 16; ++i) {
        const int m = (tid >> 4) + 16 * i;
        const bool p = kok && (tile.m0 + m) < P.M;
        stage(as + k * LDA + m, ga, A, S.a_off, kk + k, tile.m0 + m, S.lda, p);
      }
    }
    if (S.tb == 0) {
      const int k = tid & 15;
      const bool kok = (kk + k) < kend;
#pragma unroll
      for (int i = 0; i < BN / 16; ++i) {
        const int n = (tid >> 4) + 16 * i;
        const bool p = kok && (tile.n0 + n) < P.N;
        stage(bs + k * LDB + n, gb, B, S.b_off, kk + k, tile.n0 + n, S.ldb, p);
      }
    } else {
      constexpr int KS = kThreads / BN;
      const int n = tid % BN;
      const bool nok = (tile.n0 + n) < P.N;
#pragma unroll
      for (int i = 0; i < BN * kBK / kThreads; ++i) {
        const int k = tid / BN + KS * i;
        const bool p = nok && (kk + k) < kend;
        stage(bs + k * LDB + n, gb, B, S.b_off, tile.n0 + n, kk + k, S.ldb, p);
      }
    }
  };

  KIter it{P.seg0, 0, 0, 0};
  settle(it);
  int buf = 0;
  if (it.si < seg_end) load(0, it);
  cp_async_commit();
  while (it.si < seg_end) {
    KIter nx = it;
    advance(nx);
    if (nx.si < seg_end) load(buf ^ 1, nx);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const double *as = As + buf * kBK * LDA;
    const double *bs = Bs + buf * kBK * LDB;
#pragma unroll
    for (int k = 0; k < kBK; ++k) {
      double a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM / 2; ++i) {
        const double2 v = *reinterpret_cast<const double2 *>(as + k * LDA + 2 * ty + 32 * i);
        a[2 * i] = v.x;
        a[2 * i + 1] = v.y;
      }
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) {
        const double2 v = *reinterpret_cast<const double2 *>(bs + k * LDB + 2 * tx + 32 * j);
        b[2 * j] = v.x;
        b[2 * j + 1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
    buf ^= 1;
    it = nx;
  }
  cp_async_wait<0>();

  double *C = base_ptr(bases, P.cbase) + P.c_off;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = tile.m0 + 2 * ty + 32 * (i >> 1) + (i & 1);
    if (m >= P.M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = tile.n0 + 2 * tx + 32 * (j >> 1) + (j & 1);
      if (n >= P.N) continue;
      double *c = C + m + (long long)n * P.ldc;
      const double v = P.alpha * acc[i][j];
      if (tile.atomic)
        atomicAdd(c, v);
      else
        *c = (P.beta == 0.0) ? v : v + P.beta * (*c);
    }
  }
}

// ---- FP64 tensor-core (DMMA) variant ------------------------------------------------
// Same tiles, segments and K iteration as gemm_f64_kernel, with the multiply-adds
// on the FP64 tensor-core path (mma.sync m8n8k4 .f64: one warp instruction is an
// 8 x 8 x 4 product, 256 FMAs).  Eight warps per CTA, each owning a WM x WN
// sub-tile of the BM x BN output (WM/8 x WN/8 MMA tiles, two accumulators per
// lane each).  K advances BK (16 or 32: option gemm_f64_engine 1 / 2) at a time
// through a cp.async ring; 32-deep stages halve the per-stage work (copy set-up,
// barrier, segment bookkeeping) per MMA and were 10% faster on B200.  Each operand
// is staged in the layout that makes its global reads contiguous: an operand
// whose contiguous dimension is K is stored [row][k] (BK + 4 doubles per
// row), otherwise [k][row] (BM or BN + 4 per k); the pads make every fragment
// load of a half-warp hit 16 distinct 8-byte bank pairs.  Copies are 16 bytes
// when the operand's offset and leading dimension (and, for K-contiguous
// operands, the first K index) are even, else 8; elements past M, N or the K
// range are zero-filled.  The ring is as deep as two CTAs per SM allow (2 to
// 4 stages).  Ranks and leaf sizes are rarely multiples of a tile, so at an
// edge a warp issues only the 8 x 8 MMA tiles and the 4-deep K steps that hold
// something, and a segment's pointers are kept in registers until it ends.
// The MMA loop from shared memory alone reaches 36 of 37 TFLOP/s; what is lost
// is the loader's instructions (nine per MMA before the three copy paths of
// stage_operand and the per-layout MMA loops, under five now), during which the
// warps of a CTA issue no MMAs.  H X at n = 32768, k = 256 (ranks 38 to 349):
// 1640 us without any of this, 1512 us without MMAs on padding, 1370 us so
// (28.7 TFLOP/s; cuBLAS DGEMM 35.5); H x H at n = 16384 (many products of 5 to
// 40 columns) 3.44, 2.90, 2.47 ms.  With loader warps beside the MMA warps
// (gemm_f64_ws_kernel) 1250 us (31.5 TFLOP/s in the larger launch) and 2.25 ms.
template <int BM, int BN, int BK>
struct MmaSmem {
  static constexpr int LDKM = BM + 4;      // [k][m] layout
  static constexpr int LDKN = BN + 4;      // [k][n] layout
  static constexpr int LDK = BK + 4;      // [m][k] / [n][k] layout
  static constexpr int A_ELEMS = (BK * LDKM > BM * LDK) ? BK * LDKM : BM * LDK;
  static constexpr int B_ELEMS = (BK * LDKN > BN * LDK) ? BK * LDKN : BN * LDK;
  static constexpr int STAGE = A_ELEMS + B_ELEMS;
  static constexpr int STAGES_FIT = (int)(112 * 1024 / (sizeof(double) * STAGE));
  static constexpr int STAGES = STAGES_FIT > 4 ? 4 : (STAGES_FIT < 2 ? 2 : STAGES_FIT);
  static constexpr size_t bytes = sizeof(double) * STAGES * STAGE;
};

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
// The same, or sixteen zero bytes (nothing is read then).
__device__ __forceinline__ void cp_async16z(void *smem, const void *gmem, bool pred) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem),
               "r"(pred ? 16 : 0));
}

// One operand tile of ROWS lines (M or N side) x BK into stage memory, by
// cp.async.  `src` is element (line 0, K index 0) of the stage; K-contiguous
// operands go to [line][k], the others to [k][line].  Lines past `nlines` and
// K values past `kin` are zero-filled.  A thread's copies differ by a constant
// step in both memories.  Three ways, uniform over the CTA: the whole tile by
// plain 16-byte copies (an addition and the copy each), an edge at an even
// line or K value by 16-byte copies that read all or nothing, any other by
// 8-byte ones (a copy of a variable number of bytes compiles to some 70
// instructions).
template <int ROWS, int BK, int THREADS>
__device__ __forceinline__ void stage_operand(int tid, double *dst, const double *src, int ld,
                                              bool kcontig, bool vec, int nlines, int kin) {
  const bool full = nlines >= ROWS && kin == BK;
  if (kcontig) {
    constexpr int CH = BK / 2, LS = THREADS / CH;   // 16-byte chunks per line, lines per pass
    static_assert(ROWS % LS == 0, "whole passes");
    const int l0 = tid / CH, k = 2 * (tid % CH);
    double *d = dst + l0 * (BK + 4) + k;
    const double *q = src + (long long)l0 * ld + k;
    const long long step = (long long)LS * ld;
    if (vec && full) {
#pragma unroll(THREADS < kThreads ? 4 : 64)
      for (int i = 0; i < ROWS / LS; ++i, q += step) cp_async16(d + i * LS * (BK + 4), q);
    } else if (vec && (kin & 1) == 0) {
#pragma unroll(THREADS < kThreads ? 4 : 64)
      for (int i = 0; i < ROWS / LS; ++i, q += step) {
        const bool in = k < kin && l0 + i * LS < nlines;
        cp_async16z(d + i * LS * (BK + 4), in ? q : src, in);
      }
    } else {
#pragma unroll(THREADS < kThreads ? 4 : 64)
      for (int i = 0; i < ROWS / LS; ++i, q += step) {
        const bool in = k < kin && l0 + i * LS < nlines, in2 = in && k + 1 < kin;
        cp_async8(d + i * LS * (BK + 4), in ? q : src, in);
        cp_async8(d + i * LS * (BK + 4) + 1, in2 ? q + 1 : src, in2);
      }
    }
  } else {
    constexpr int CH = ROWS / 2, KS = THREADS / CH;   // chunks per K value, K values per pass
    static_assert(KS >= 1, "a line is no longer than a pass");
    const int line = 2 * (tid % CH), k0 = tid / CH;
    double *d = dst + k0 * (ROWS + 4) + line;
    const double *q = src + (long long)k0 * ld + line;
    const long long step = (long long)KS * ld;
    if (vec && full) {
#pragma unroll(THREADS < kThreads ? 4 : 64)
      for (int i = 0; i < BK / KS; ++i, q += step) cp_async16(d + i * KS * (ROWS + 4), q);
    } else if (vec && ((nlines & 1) == 0 || nlines >= ROWS)) {
#pragma unroll(THREADS < kThreads ? 4 : 64)
      for (int i = 0; i < BK / KS; ++i, q += step) {
        const bool in = line < nlines && k0 + i * KS < kin;
        cp_async16z(d + i * KS * (ROWS + 4), in ? q : src, in);
      }
    } else {
#pragma unroll(THREADS < kThreads ? 4 : 64)
      for (int i = 0; i < BK / KS; ++i, q += step) {
        const bool in = line < nlines && k0 + i * KS < kin, in2 = in && line + 1 < nlines;
        cp_async8(d + i * KS * (ROWS + 4), in ? q : src, in);
        cp_async8(d + i * KS * (ROWS + 4) + 1, in2 ? q + 1 : src, in2);
      }
    }
  }
}

// The same for a generated kernel matrix: (r, c) of the block at
// gen_offset(row0, col0), computed entry by entry.
template <int ROWS, int BK>
__device__ __forceinline__ void stage_generated(double *dst, const KernelSpec &gen, long long off,
                                                bool kcontig, int row0, int nlines, int kk,
                                                int kin) {
  const int gr0 = (int)(off >> 32), gc0 = (int)(off & 0xffffffffLL);
  for (int e = threadIdx.x; e < ROWS * BK; e += kThreads) {
    const int line = kcontig ? e / BK : e % ROWS, k = kcontig ? e % BK : e / ROWS;
    double v = 0.0;
    if (line < nlines && k < kin) {
      const int r = kcontig ? kk + k : row0 + line;
      const int c = kcontig ? row0 + line : kk + k;
      v = kernel_entry(gen, gr0 + r, gc0 + c);
    }
    if (kcontig)
      dst[line * (BK + 4) + k] = v;
    else
      dst[k * (ROWS + 4) + line] = v;
  }
}

// A whole stage's MMAs of one warp: ap, bp are the lane's first fragment
// elements, the steps to the next line and K value known at compile time (one
// copy of the loop per layout: every fragment load has a constant offset).
template <int MT, int NT, int BK, int A_LINE, int A_K, int B_LINE, int B_K>
__device__ __forceinline__ void stage_mmas(double (&acc)[MT][NT][2], const double *ap,
                                           const double *bp) {
#pragma unroll
  for (int k4 = 0; k4 < BK / 4; ++k4) {
    double a[MT], b[NT];
#pragma unroll
    for (int i = 0; i < MT; ++i) a[i] = ap[8 * i * A_LINE + 4 * k4 * A_K];
#pragma unroll
    for (int j = 0; j < NT; ++j) b[j] = bp[8 * j * B_LINE + 4 * k4 * B_K];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j) dmma884(acc[i][j], a[i], b[j]);
  }
}

template <int BM, int BN, int WM, int WN, int BK>
__global__ void __launch_bounds__(kThreads, 2)
gemm_f64_mma_kernel(const GemmSeg *__restrict__ segs, const GemmProb *__restrict__ probs,
                    const GemmTile *__restrict__ tiles, GemmBases bases) {
  using SM = MmaSmem<BM, BN, BK>;
  constexpr int kMmaStages = SM::STAGES;
  constexpr int MT = WM / 8, NT = WN / 8;          // MMA tiles per warp
  constexpr int WARPS_N = BN / WN;
  static_assert((BM / WM) * (BN / WN) == kThreads / 32, "eight warps per CTA");
  extern __shared__ __align__(16) double smem[];

  const GemmTile tile = tiles[blockIdx.x];
  const GemmProb P = probs[tile.prob];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  // Warps w and w + 4 share an SM sub-partition and its tensor core.  At an
  // edge whole rows or columns of warps are idle, so warp rows (four of them)
  // or columns go to different sub-partitions, and with two warp rows the
  // second is turned by two.
  int wrow, wcol;
  if constexpr (WARPS_N == 2) {
    wrow = warp & 3;
    wcol = warp >> 2;
  } else if constexpr (WARPS_N == 4) {
    wrow = warp >> 2;
    wcol = (warp + 2 * wrow) & 3;
  } else {
    wrow = warp / WARPS_N;
    wcol = warp % WARPS_N;
  }
  const int wm0 = wrow * WM, wn0 = wcol * WN;
  const int seg_end = P.seg0 + P.nseg;
  // 8-row and 8-column MMA tiles of this warp that lie inside the problem
  const int mt_in = max(0, min(MT, (P.M - tile.m0 - wm0 + 7) / 8));
  const int nt_in = max(0, min(NT, (P.N - tile.n0 - wn0 + 7) / 8));
  const bool whole = mt_in == MT && nt_in == NT;

  double acc[MT][NT][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  auto settle = [&](KIter &it) {
    while (it.si < seg_end) {
      const int K = segs[it.si].K;
      const int ls = max(tile.k0 - it.kbase, 0);
      const int le = min(tile.k1 - it.kbase, K);
      if (ls < le) {
        it.kk = ls;
        it.le = le;
        return;
      }
      it.kbase += K;
      ++it.si;
    }
  };
  auto advance = [&](KIter &it) {
    it.kk += BK;
    if (it.kk >= it.le) {
      it.kbase += segs[it.si].K;
      ++it.si;
      settle(it);
    }
  };

  // the segment being loaded: operand pointers at (this tile's first line,
  // K = 0), leading dimensions, and flags (1: A K-contiguous, 2: B, 4: A by
  // 16-byte copies, 8: B, 16: A generated, 32: B)
  const double *pa = nullptr, *pb = nullptr;
  long long goff = 0;   // offset of the generated operand
  int lda = 0, ldb = 0;
  unsigned fl = 0;
  auto open_segment = [&](const KIter &it) {
    const GemmSeg S = segs[it.si];
    // op(A) is M x K: ta = 0 stores (m, k) at m + k lda (lines contiguous),
    // ta = 1 at k + m lda (K contiguous); op(B) is K x N: tb = 0 stores (k, n)
    // at k + n ldb (K contiguous), tb = 1 at n + k ldb
    const bool ka = S.ta == 1, kb = S.tb == 0;
    const bool ga = S.abase == kGenSlot, gb = S.bbase == kGenSlot;
    lda = (int)S.lda;
    ldb = (int)S.ldb;
    fl = (ka ? 1u : 0u) | (kb ? 2u : 0u) | (ga ? 16u : 0u) | (gb ? 32u : 0u);
    goff = ga ? S.a_off : S.b_off;
    // 16-byte copies need an even element offset from a 16-byte boundary:
    // operand, leading dimension, and the first K index of a K-contiguous one
    if (!ga) {
      const double *base = base_ptr(bases, S.abase) + S.a_off;
      if (((lda | (ka ? it.kk : 0)) & 1) == 0 && ((unsigned long long)base & 15) == 0) fl |= 4u;
      pa = base + (ka ? (long long)tile.m0 * lda : tile.m0);
    }
    if (!gb) {
      const double *base = base_ptr(bases, S.bbase) + S.b_off;
      if (((ldb | (kb ? it.kk : 0)) & 1) == 0 && ((unsigned long long)base & 15) == 0) fl |= 8u;
      pb = base + (kb ? (long long)tile.n0 * ldb : tile.n0);
    }
  };

  // Stage `buf` <- K-block `it`; returns its layout bits (1: A stored [m][k],
  // 2: B stored [n][k]).
  auto load = [&](int buf, const KIter &it) -> unsigned {
    double *as = smem + buf * SM::STAGE;
    double *bs = as + SM::A_ELEMS;
    const int kin = min(BK, it.le - it.kk);
    const bool ka = fl & 1u, kb = fl & 2u;
    if (fl & 16u)
      stage_generated<BM, BK>(as, bases.gen, goff, ka, tile.m0, P.M - tile.m0, it.kk, kin);
    else
      stage_operand<BM, BK, kThreads>(tid, as,
                                      pa + (ka ? (long long)it.kk : (long long)it.kk * lda), lda,
                                      ka, fl & 4u, P.M - tile.m0, kin);
    if (fl & 32u)
      stage_generated<BN, BK>(bs, bases.gen, goff, kb, tile.n0, P.N - tile.n0, it.kk, kin);
    else
      stage_operand<BN, BK, kThreads>(tid, bs,
                                      pb + (kb ? (long long)it.kk : (long long)it.kk * ldb), ldb,
                                      kb, fl & 8u, P.N - tile.n0, kin);
    return fl & 3u;
  };
  // the next K-block of the load side, opening its segment when it changes
  auto advance_load = [&](KIter &it) {
    const int si = it.si;
    advance(it);
    if (it.si != si && it.si < seg_end) open_segment(it);
  };

  // ring of kMmaStages buffers; `lay` keeps 2 layout bits per buffer
  KIter it{P.seg0, 0, 0, 0};
  settle(it);
  if (it.si < seg_end) open_segment(it);
  unsigned lay = 0;
#pragma unroll
  for (int st = 0; st < kMmaStages - 1; ++st) {
    if (it.si < seg_end) {
      lay |= load(st, it) << (2 * st);
      advance_load(it);
    }
    cp_async_commit();
  }
  int buf = 0;
  KIter cit{P.seg0, 0, 0, 0};
  settle(cit);
  while (cit.si < seg_end) {
    cp_async_wait<kMmaStages - 2>();
    __syncthreads();
    {
      const int nb = (buf + kMmaStages - 1) % kMmaStages;
      if (it.si < seg_end) {
        lay = (lay & ~(3u << (2 * nb))) | (load(nb, it) << (2 * nb));
        advance_load(it);
      }
      cp_async_commit();
    }
    const unsigned l = (lay >> (2 * buf)) & 3u;
    const double *as = smem + buf * SM::STAGE;
    const double *bs = as + SM::A_ELEMS;
    // per-lane fragment addressing: A (m = g, k = t), B (k = t, n = g)
    const int a_line_step = (l & 1) ? SM::LDK : 1;       // next m
    const int a_k_step = (l & 1) ? 1 : SM::LDKM;          // next k
    const int b_line_step = (l & 2) ? SM::LDK : 1;       // next n
    const int b_k_step = (l & 2) ? 1 : SM::LDKN;
    const double *ap = as + (wm0 + g) * a_line_step + t * a_k_step;
    const double *bp = bs + (wn0 + g) * b_line_step + t * b_k_step;
    const int kin = min(BK, cit.le - cit.kk);   // K values of this stage
    if (whole && kin == BK) {
      switch (l) {
        case 0: stage_mmas<MT, NT, BK, 1, SM::LDKM, 1, SM::LDKN>(acc, ap, bp); break;
        case 1: stage_mmas<MT, NT, BK, SM::LDK, 1, 1, SM::LDKN>(acc, ap, bp); break;
        case 2: stage_mmas<MT, NT, BK, 1, SM::LDKM, SM::LDK, 1>(acc, ap, bp); break;
        default: stage_mmas<MT, NT, BK, SM::LDK, 1, SM::LDK, 1>(acc, ap, bp); break;
      }
    } else if (mt_in > 0 && nt_in > 0) {
      // edge of the problem or of a K range: only the MMA tiles and 4-deep
      // steps that hold something (all uniform over the warp)
      for (int k4 = 0; 4 * k4 < kin; ++k4) {
        double b[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j)
          if (j < nt_in) b[j] = bp[(8 * j) * b_line_step + 4 * k4 * b_k_step];
#pragma unroll
        for (int i = 0; i < MT; ++i)
          if (i < mt_in) {
            const double a = ap[(8 * i) * a_line_step + 4 * k4 * a_k_step];
#pragma unroll
            for (int j = 0; j < NT; ++j)
              if (j < nt_in) dmma884(acc[i][j], a, b[j]);
          }
      }
    }
    buf = (buf + 1) % kMmaStages;
    advance(cit);
  }
  cp_async_wait<0>();

  double *C = base_ptr(bases, P.cbase) + P.c_off;
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const int m = tile.m0 + wm0 + 8 * i + g;
    if (m >= P.M) continue;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = tile.n0 + wn0 + 8 * j + 2 * t + h;
        if (n >= P.N) continue;
        double *c = C + m + (long long)n * P.ldc;
        const double v = P.alpha * acc[i][j][h];
        if (tile.atomic)
          atomicAdd(c, v);
        else
          *c = (P.beta == 0.0) ? v : v + P.beta * (*c);
      }
    }
  }
}

// ---- the same product with loader warps ----------------------------------------------
// Eight warps issue MMAs only, two more the copies: in
// gemm_f64_mma_kernel every warp stops its MMAs for some 400 instructions a
// stage, and the warps of a CTA do so together, which leaves the tensor cores
// idle a fifth of the time.  Stages are handed over with named barriers (full:
// the loaders arrive, the MMA warps wait; empty: the reverse); each carries its
// operand layout and K length, a length of zero ends the tile.  Used for
// plans without generated operands (whose entries all threads should compute).
// H X at n = 32768, k = 256: 1370 -> 1253 us (tensor cores active 79 -> 84% of
// the time); H^T X and X H at n = 10007, k = 33: 265 -> 209 us.
constexpr int kWsLoaders = 64;
constexpr int kWsThreads = kThreads + kWsLoaders;

__device__ __forceinline__ void bar_sync(int id) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "n"(kWsThreads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id) {
  asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "n"(kWsThreads) : "memory");
}

template <int BM, int BN, int WM, int WN, int BK>
__global__ void __launch_bounds__(kWsThreads, 2)
gemm_f64_ws_kernel(const GemmSeg *__restrict__ segs, const GemmProb *__restrict__ probs,
                   const GemmTile *__restrict__ tiles, GemmBases bases) {
  using SM = MmaSmem<BM, BN, BK>;
  constexpr int S = SM::STAGES;
  static_assert(2 * S + 1 <= 16, "named barriers");
  extern __shared__ __align__(16) double smem[];
  __shared__ int meta[S];   // per stage: layout bits (1: A [m][k], 2: B [n][k]), K values << 2
  const GemmTile tile = tiles[blockIdx.x];
  const GemmProb P = probs[tile.prob];
  auto full = [](int st) { return 1 + st; };
  auto empty = [](int st) { return 1 + S + st; };

  if (threadIdx.x >= kThreads) {
    // ---------------- loaders ----------------
    constexpr int kLag = S - 2;   // stages in flight behind the one being issued
    const int tid = threadIdx.x - kThreads;
    const int seg_end = P.seg0 + P.nseg;
    const int nm = P.M - tile.m0, nn = P.N - tile.n0;
    int kbase = 0, t = 0;
    for (int si = P.seg0; si < seg_end; ++si) {
      const GemmSeg G = segs[si];
      int kk = max(tile.k0 - kbase, 0);
      const int le = min(tile.k1 - kbase, G.K);
      kbase += G.K;
      if (kk >= le) continue;
      const bool ka = G.ta == 1, kb = G.tb == 0;
      const int lda = (int)G.lda, ldb = (int)G.ldb;
      const double *pa = base_ptr(bases, G.abase) + G.a_off;
      const double *pb = base_ptr(bases, G.bbase) + G.b_off;
      // 16-byte copies: as in gemm_f64_mma_kernel
      const bool va = ((lda | (ka ? kk : 0)) & 1) == 0 && ((unsigned long long)pa & 15) == 0;
      const bool vb = ((ldb | (kb ? kk : 0)) & 1) == 0 && ((unsigned long long)pb & 15) == 0;
      pa += ka ? (long long)tile.m0 * lda + kk : tile.m0 + (long long)kk * lda;
      pb += kb ? (long long)tile.n0 * ldb + kk : tile.n0 + (long long)kk * ldb;
      for (; kk < le; kk += BK, ++t) {
        const int st = t % S, kin = min(BK, le - kk);
        if (t >= S) bar_sync(empty(st));
        double *as = smem + st * SM::STAGE;
        stage_operand<BM, BK, kWsLoaders>(tid, as, pa, lda, ka, va, nm, kin);
        stage_operand<BN, BK, kWsLoaders>(tid, as + SM::A_ELEMS, pb, ldb, kb, vb, nn, kin);
        cp_async_commit();
        if (tid == 0) meta[st] = (ka ? 1 : 0) | (kb ? 2 : 0) | (kin << 2);
        if (t >= kLag) {
          cp_async_wait<kLag>();
          bar_arrive(full((t - kLag) % S));
        }
        pa += ka ? (long long)BK : (long long)BK * lda;
        pb += kb ? (long long)BK : (long long)BK * ldb;
      }
    }
    cp_async_wait<0>();
    for (int u = max(0, t - kLag); u < t; ++u) bar_arrive(full(u % S));
    // the end, then the stages still being read (no arrival is left over)
    if (t >= S) bar_sync(empty(t % S));
    if (tid == 0) meta[t % S] = 0;
    __threadfence_block();
    bar_arrive(full(t % S));
    for (int u = max(0, t - S + 1); u < t; ++u) bar_sync(empty(u % S));
    return;
  }

  // ---------------- MMA warps ----------------
  constexpr int MT = WM / 8, NT = WN / 8, WARPS_N = BN / WN;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, tq = lane & 3;
  int wrow, wcol;   // warps to sub-partitions: as in gemm_f64_mma_kernel
  if constexpr (WARPS_N == 2) {
    wrow = warp & 3;
    wcol = warp >> 2;
  } else if constexpr (WARPS_N == 4) {
    wrow = warp >> 2;
    wcol = (warp + 2 * wrow) & 3;
  } else {
    wrow = warp / WARPS_N;
    wcol = warp % WARPS_N;
  }
  const int wm0 = wrow * WM, wn0 = wcol * WN;
  const int mt_in = max(0, min(MT, (P.M - tile.m0 - wm0 + 7) / 8));
  const int nt_in = max(0, min(NT, (P.N - tile.n0 - wn0 + 7) / 8));
  const bool whole = mt_in == MT && nt_in == NT;
  double acc[MT][NT][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  for (int st = 0;; st = st + 1 == S ? 0 : st + 1) {
    bar_sync(full(st));
    const int m = meta[st], kin = m >> 2;
    if (kin == 0) break;
    const double *as = smem + st * SM::STAGE;
    const double *bs = as + SM::A_ELEMS;
    const int a_line = (m & 1) ? SM::LDK : 1, a_k = (m & 1) ? 1 : SM::LDKM;
    const int b_line = (m & 2) ? SM::LDK : 1, b_k = (m & 2) ? 1 : SM::LDKN;
    const double *ap = as + (wm0 + g) * a_line + tq * a_k;
    const double *bp = bs + (wn0 + g) * b_line + tq * b_k;
    if (whole && kin == BK) {
      switch (m & 3) {
        case 0: stage_mmas<MT, NT, BK, 1, SM::LDKM, 1, SM::LDKN>(acc, ap, bp); break;
        case 1: stage_mmas<MT, NT, BK, SM::LDK, 1, 1, SM::LDKN>(acc, ap, bp); break;
        case 2: stage_mmas<MT, NT, BK, 1, SM::LDKM, SM::LDK, 1>(acc, ap, bp); break;
        default: stage_mmas<MT, NT, BK, SM::LDK, 1, SM::LDK, 1>(acc, ap, bp); break;
      }
    } else if (mt_in > 0 && nt_in > 0) {
      for (int k4 = 0; 4 * k4 < kin; ++k4) {
        double b[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j)
          if (j < nt_in) b[j] = bp[(8 * j) * b_line + 4 * k4 * b_k];
#pragma unroll
        for (int i = 0; i < MT; ++i)
          if (i < mt_in) {
            const double a = ap[(8 * i) * a_line + 4 * k4 * a_k];
#pragma unroll
            for (int j = 0; j < NT; ++j)
              if (j < nt_in) dmma884(acc[i][j], a, b[j]);
          }
      }
    }
    bar_arrive(empty(st));
  }

  double *C = base_ptr(bases, P.cbase) + P.c_off;
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const int row = tile.m0 + wm0 + 8 * i + g;
    if (row >= P.M) continue;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int col = tile.n0 + wn0 + 8 * j + 2 * tq + h;
        if (col >= P.N) continue;
        double *c = C + row + (long long)col * P.ldc;
        const double v = P.alpha * acc[i][j][h];
        if (tile.atomic)
          atomicAdd(c, v);
        else
          *c = (P.beta == 0.0) ? v : v + P.beta * (*c);
      }
  }
}

// beta pre-pass for the (m, n) tiles that several tiles add to
__global__ void gemm_scale_c_kernel(const GemmProb *__restrict__ probs,
                                    const GemmTile *__restrict__ tiles, int bm, int bn,
                                    GemmBases bases) {
  const GemmTile T = tiles[blockIdx.x];
  const GemmProb P = probs[T.prob];
  double *C = base_ptr(bases, P.cbase) + P.c_off;
  const int rows = min(bm, P.M - T.m0), cols = min(bn, P.N - T.n0);
  for (int c = threadIdx.x >> 5; c < cols; c += blockDim.x >> 5)
    for (int r = threadIdx.x & 31; r < rows; r += 32) {
      double *p = C + T.m0 + r + (long long)(T.n0 + c) * P.ldc;
      *p = (P.beta == 0.0) ? 0.0 : P.beta * (*p);
    }
}

template <int BM, int BN, int WM, int WN>
void launch_gemm(const GemmPlan &plan, const GemmBases &bases, cudaStream_t stream) {
  const int engine = gemm_f64_engine();
  if (engine == 1) {
    static SmemOptIn opt_in;
    const size_t smem = MmaSmem<BM, BN, 16>::bytes;
    opt_in(gemm_f64_mma_kernel<BM, BN, WM, WN, 16>, smem);
    gemm_f64_mma_kernel<BM, BN, WM, WN, 16><<<plan.ntiles, kThreads, smem, stream>>>(
        plan.segs, plan.probs, plan.tiles, bases);
    HB_LAUNCHED();
    return;
  }
  if constexpr (BM <= 2 * kWsLoaders && BN <= 2 * kWsLoaders) {   // a chunk per loader and line
    if (engine == 2 && !plan.generated) {
      static SmemOptIn opt_in;
      const size_t smem = MmaSmem<BM, BN, 32>::bytes;
      opt_in(gemm_f64_ws_kernel<BM, BN, WM, WN, 32>, smem);
      gemm_f64_ws_kernel<BM, BN, WM, WN, 32><<<plan.ntiles, kWsThreads, smem, stream>>>(
          plan.segs, plan.probs, plan.tiles, bases);
      HB_LAUNCHED();
      return;
    }
  }
  if (engine == 2) {
    static SmemOptIn opt_in;
    const size_t smem = MmaSmem<BM, BN, 32>::bytes;
    opt_in(gemm_f64_mma_kernel<BM, BN, WM, WN, 32>, smem);
    gemm_f64_mma_kernel<BM, BN, WM, WN, 32><<<plan.ntiles, kThreads, smem, stream>>>(
        plan.segs, plan.probs, plan.tiles, bases);
    HB_LAUNCHED();
    return;
  }
  static SmemOptIn opt_in;
  const size_t smem = Smem<BM, BN>::bytes;
  opt_in(gemm_f64_kernel<BM, BN>, smem);
  gemm_f64_kernel<BM, BN><<<plan.ntiles, kThreads, smem, stream>>>(plan.segs, plan.probs,
                                                                   plan.tiles, bases);
  HB_LAUNCHED();
}

}  // namespace

GemmPlan::~GemmPlan() {
  if (!dev) return;
  if (transient)
    cudaFreeAsync(dev, stream);
  else
    cudaFree(dev);
}

void gemm_plan_build(GemmPlan &plan, const GemmBatch &batch, TileShape shape, KSplit ksplit,
                     cudaStream_t stream, bool transient) {
  const auto t_start = std::chrono::steady_clock::now();
  struct Clock {
    std::chrono::steady_clock::time_point t;
    ~Clock() {
      plan_host_ms() +=
          std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t).count();
    }
  } clock{t_start};
  const int BM = tile_rows(shape);
  const int BN = tile_cols(shape);
  plan.shape = shape;
  const auto &probs = batch.probs;
  std::vector<long long> ktot(probs.size(), 0);
  long long base_tiles = 0;
  double work = 0.0;
  for (size_t p = 0; p < probs.size(); ++p) {
    for (int s = 0; s < probs[p].nseg; ++s) ktot[p] += batch.segs[probs[p].seg0 + s].K;
    gemm_flops_counter() += 2.0 * probs[p].M * (double)probs[p].N * (double)ktot[p];
    const long long mn =
        (long long)((probs[p].M + BM - 1) / BM) * ((probs[p].N + BN - 1) / BN);
    base_tiles += mn;
    work += (double)mn * (double)std::max<long long>(ktot[p], 1);
  }
  const long long target = 4LL * num_sms();
  // per problem: its K split and the K length of its tiles
  std::vector<long long> chunk_of(probs.size(), 0);
  std::vector<int> split_of(probs.size(), 1);
  for (size_t p = 0; p < probs.size(); ++p) {
    const GemmProb &P = probs[p];
    if (P.M <= 0 || P.N <= 0) continue;
    // Split K so that no tile carries much more than an even share of the
    // batch's work (the longest tile bounds the launch), and to fill the GPU.
    long long split = 1;
    if (ksplit == KSplit::All && ktot[p] > 2 * 256) {
      const double per_tile = work / (double)target;          // ideal work per tile
      const double mine = (double)std::max<long long>(ktot[p], 1);
      split = (long long)std::ceil(mine / std::max(per_tile, 512.0));
      split = std::max<long long>(1, std::min<long long>(split, ktot[p] / 256));
    }
    long long chunk = (ktot[p] + split - 1) / split;
    chunk = (chunk + kBK - 1) / kBK * kBK;
    if (chunk <= 0) chunk = kBK;
    split = std::max<long long>(1, (ktot[p] + chunk - 1) / chunk);
    split_of[p] = (int)split;
    chunk_of[p] = split == 1 ? ktot[p] : chunk;
  }
  // tiles of the problems with the longest K ranges first, for load balance
  // (ordering the problems, not the tiles: a problem's tiles share their K
  // length but for a shorter last split)
  std::vector<int> order(probs.size());
  for (size_t p = 0; p < probs.size(); ++p) order[p] = (int)p;
  std::stable_sort(order.begin(), order.end(),
                   [&](int a, int b) { return chunk_of[a] > chunk_of[b]; });
  std::vector<GemmTile> tiles, scale;
  tiles.reserve(base_tiles);
  for (int p : order) {
    const GemmProb &P = probs[p];
    if (P.M <= 0 || P.N <= 0) continue;
    const int mt = (P.M + BM - 1) / BM, nt = (P.N + BN - 1) / BN;
    const long long chunk = chunk_of[p];
    const int split = split_of[p];
    for (int mi = 0; mi < mt; ++mi)
      for (int ni = 0; ni < nt; ++ni) {
        GemmTile t{p, mi * BM, ni * BN, 0, 0, split > 1 ? 1 : 0};
        if (split > 1 && P.beta != 1.0) scale.push_back(t);
        for (long long si = 0; si < split; ++si) {
          t.k0 = (int)(si * chunk);
          t.k1 = split == 1 ? (int)ktot[p] : (int)std::min<long long>(ktot[p], (si + 1) * chunk);
          tiles.push_back(t);
        }
      }
  }
  // A last wave that fills part of the GPU (two CTAs per SM) runs as long as a
  // full one: its tiles are split along K into the number of parts, each at
  // least 256 long, whose waves are shortest together (3% for a part's own
  // start and end).  n = 32768, k = 256: 1024 output tiles of K about 1260,
  // 3.46 waves, the last 136 in two parts; a tree of n = 16384 whose ranks add to
  // 1000: 512 tiles, 1.73 waves, the last 216 in four (689 -> 655 us for the whole
  // product).  From three parts on the order of their sums is open.
  if (ksplit == KSplit::Tail) {
    const long long slots = 2LL * num_sms(), rest = (long long)tiles.size() % slots;
    if (rest > 0) {
      std::vector<GemmTile> tail(tiles.end() - rest, tiles.end());
      tiles.resize(tiles.size() - rest);
      int parts = 1;
      double best = 1.0;
      for (int q = 2; q <= 8 && 256 * q <= tail.front().k1; ++q) {
        const double t = (double)((rest * q + slots - 1) / slots) / q + 0.03 * q;
        if (t < best) {
          best = t;
          parts = q;
        }
      }
      for (GemmTile &t : tail) {
        const long long mine = std::max<long long>(1, std::min<long long>(parts, t.k1 / 256));
        const long long chunk = (t.k1 / mine + 31) / 32 * 32;
        if (mine == 1) {
          tiles.push_back(t);
          continue;
        }
        t.atomic = 1;
        if (probs[t.prob].beta != 1.0) scale.push_back(t);
        const int kend = t.k1;
        for (long long q = 0; q < mine; ++q) {
          t.k0 = (int)std::min<long long>(kend, q * chunk);
          t.k1 = q + 1 == mine ? kend : (int)std::min<long long>(kend, (q + 1) * chunk);
          if (t.k0 < t.k1) tiles.push_back(t);
        }
      }
    }
  }
  plan.ntiles = (int)tiles.size();
  plan.nscale = (int)scale.size();
  plan.generated = false;
  for (const GemmSeg &g : batch.segs)
    plan.generated = plan.generated || g.abase == kGenSlot || g.bbase == kGenSlot;
  tiles.insert(tiles.end(), scale.begin(), scale.end());
  const size_t bs = batch.segs.size() * sizeof(GemmSeg);
  const size_t bp = probs.size() * sizeof(GemmProb);
  const size_t bt = tiles.size() * sizeof(GemmTile);
  const size_t total = align_up(bs, 256) + align_up(bp, 256) + align_up(bt, 256) + 256;
  if (plan.dev) {
    if (plan.transient)
      cudaFreeAsync(plan.dev, plan.stream);
    else
      cudaFree(plan.dev);
    plan.dev = nullptr;
  }
  plan.transient = transient;
  plan.stream = stream;
  // stream-ordered in both cases (a cudaMalloc stops the device); a kept plan
  // is ready for any stream after the synchronisation below
  pool_alloc(&plan.dev, total, stream);
  char *base = (char *)plan.dev;
  plan.segs = (GemmSeg *)base;
  plan.probs = (GemmProb *)(base + align_up(bs, 256));
  plan.tiles = (GemmTile *)(base + align_up(bs, 256) + align_up(bp, 256));
  std::unique_ptr<char[]> host(new char[total]);   // padding bytes are never read
  if (bs) std::memcpy(host.get(), batch.segs.data(), bs);
  if (bp) std::memcpy(host.get() + align_up(bs, 256), probs.data(), bp);
  if (bt) std::memcpy(host.get() + align_up(bs, 256) + align_up(bp, 256), tiles.data(), bt);
  // staged through the pinned ring: the host buffer may go away at once, and
  // the host does not wait for the stream
  h2d_async(plan.dev, host.get(), total, stream);
  if (!transient) HB_CUDA(cudaStreamSynchronize(stream));
}

void gemm_plan_run(const GemmPlan &plan, const GemmBases &bases, cudaStream_t stream) {
  if (plan.ntiles == 0) return;
  if (plan.nscale > 0) {
    gemm_scale_c_kernel<<<plan.nscale, 256, 0, stream>>>(plan.probs, plan.tiles + plan.ntiles,
                                                         tile_rows(plan.shape),
                                                         tile_cols(plan.shape), bases);
    HB_LAUNCHED();
  }
  switch (plan.shape) {
    case TileShape::M128N64: launch_gemm<128, 64, 32, 32>(plan, bases, stream); break;
    case TileShape::M64N128: launch_gemm<64, 128, 32, 32>(plan, bases, stream); break;
    case TileShape::M32N128: launch_gemm<32, 128, 32, 16>(plan, bases, stream); break;
    case TileShape::M32N256: launch_gemm<32, 256, 32, 32>(plan, bases, stream); break;
    case TileShape::M64N64: launch_gemm<64, 64, 16, 32>(plan, bases, stream); break;
  }
}

void gemm_f64_run(GemmBatch &batch, const GemmBases &bases, TileShape shape, cudaStream_t stream,
                  bool allow_split) {
  if (batch.empty()) return;
  if (shape == TileShape::M64N128) {
    int nmax = 0;
    for (const GemmProb &P : batch.probs) nmax = std::max(nmax, P.N);
    if (nmax <= 64) shape = TileShape::M64N64;
  }
  GemmPlan plan;
  gemm_plan_build(plan, batch, shape, allow_split ? KSplit::All : KSplit::None, stream, true);
  gemm_plan_run(plan, bases, stream);
}

}  // namespace hb
