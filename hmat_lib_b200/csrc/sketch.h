// The build's random test matrices and the product of a block with one.
//
// For every 64 columns of S (n x w): S = H M, where H (n x 64) is a block-wise
// randomised Hadamard matrix of +-1 entries: for row j of H in its group
// g = j / 64,
//
//   H(j, t) = d_g(j mod 64) (-1)^popcount((j mod 64) & t) e_g(t)
//
// with random signs d_g, e_g drawn anew for every group, every 64 columns of S
// and every matrix `id` (Balabanov, Beaupere, Grigori and Lederer, "Block
// subsampled randomized Hadamard transform for low-rank approximation on
// distributed architectures", 2022), and M is a random orthogonal 64 x 64
// matrix.  Without M the leading columns of a sketch need not be independent:
// two rows 32 apart agree up to their sign in columns 0..31, which merges two
// columns of A, and the panels are orthonormalised in that order.  Entries of
// a column are uncorrelated with unit variance, so ||A S||_F^2 / w estimates
// ||A||_F^2 without bias, as with Gaussian entries.
//
// The singular values of S against those of a Gaussian matrix (smallest of
// six; 64, 512, 960 and 1024 columns): n = 1024 32 / 24, 9.8 / 9.2, 1.1 / 1.0
// and 4e-3 / 2e-3, n = 2048 45 / 37 and 23 / 22.  Two groups are the exception
// (n = 128, 128 columns: singular for half of the signs, because the Schur
// complement is a difference of two orthogonal matrices), so blocks take these
// matrices from kSketchMinCols columns on, far from it; the narrower ones are
// 2% of the sketch products' work.
#pragma once

#include <vector>

#include "common.h"
#include "kernelspec.cuh"

namespace hb {

struct SketchDesc {
  const double *A;        // m x n block, column-major (unused when generated)
  long long lda;
  int r0, c0;             // origin of the block in the kernel matrix when generated
  int m, n, w;            // S is n x w
  double *Y;              // m x w, zero before the call
  long long ldy;
  unsigned long long id;  // S depends on (seed, id) alone
};

constexpr int kSketchMinCols = 1024;

// M: 64 x 64, column-major, from the seed alone.
std::vector<double> sketch_mixer(unsigned long long seed);

// Y = A S for every block; with `gen` the entries of A are those of a kernel
// matrix, computed here.  `M` is the mixer on the device.
void sketch_multiply(const std::vector<SketchDesc> &descs, const double *M,
                     const KernelSpec *gen, unsigned long long seed, cudaStream_t stream);

// X = S (rows x cols) for every matrix.
struct SketchFill {
  double *X;
  long long ld;
  int rows, cols;
  unsigned long long id;
};
void sketch_fill(const std::vector<SketchFill> &descs, const double *M,
                 unsigned long long seed, cudaStream_t stream);

}  // namespace hb
