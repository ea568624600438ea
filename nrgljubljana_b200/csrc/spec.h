// spec.h -- internal descriptors of the spectral-weight binning and Matsubara kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace nrg {

// Weight of the term (i, j), o1 = op1(j,i), o2 = op2(j,i), x = X(j,i), y = Y(j,i):
enum SpecKind : int {
  kSpecDMNRG = 0,  // x o1 - sign y o2, energy window [Emin, Emax]
  kSpecExpI = 1,   // coef o1 o2 exp(-Ei/T)
  kSpecExpJ = 2,   // coef o1 o2 exp(-Ej/T)
  kSpecGemmX = 3,  // coef o1 x
  // sums of two of them over the same rectangle (Matsubara axis, where both go to one sum)
  kSpecExpIJ = 4,  // coef o1 o2 exp(-Ei/T) + coef2 o1 o2 exp(-Ej/T)
  kSpecExpIX = 5,  // coef o1 o2 exp(-Ei/T) + coef2 o1 x
  kSpecXExpJ = 6,  // coef o1 x + coef2 o1 o2 exp(-Ej/T)
};

// One rectangle of (i, j) index pairs of one subspace pair with one weight formula.
// The energy of a term is Ej[j] - Ei[i]; every weight is multiplied by `factor`. X and Y are
// stored for the rectangle alone: X(j,i) = X[(j - j0) ldx + i - i0].
struct SpecRegion {
  const double* Ei;
  const double* Ej;
  const double* op1;
  const double* op2;
  const double* X;
  const double* Y;
  int64_t ld1, ld2, ldx, ldy;
  int i0, i1, j0, j1;
  int kind, sign;
  int mspecial;  // Matsubara sums: a MatsSpecial
  int tile0;     // first work item of the rectangle: spec_tiles or mats_chunks of them
  double coef, coef2, factor, T, Emin, Emax;
};

// How a term enters the Matsubara sum at n = 0 for a bosonic operator when |E| <= 1e-8
// (WEIGHT_TOL, c++/numerics.hpp:318), where the reference replaces (wA + wB) / (i w_0 - E) by
// a limit: -wA / T for the D x D term of Algo_FDMmats (c++/algo_FDM.hpp:178-188), wA its
// exp(-Ei/T) part (kMatsFdmA); -op1 op2 exp(-E1/T) / (Z T) for Algo_FTmats
// (c++/algo_FT.hpp:66-71; kMatsFtB: plus the (-sign) exp(-Ej/T) part over T); -wA / T for
// Algo_DMNRGmats (c++/algo_DMNRG.hpp:88-93), wA = X(j,i) op1(j,i) (kMatsDmnrgA).
enum MatsSpecial : int { kMatsPlain = 0, kMatsFdmA = 1, kMatsFtB = 2, kMatsDmnrgA = 3 };

struct MatsParams {
  int mats;     // points n = 0 .. mats-1
  int bosonic;  // w_n = 2 n pi T (bosonic) or (2 n + 1) pi T (fermionic)
  double T;
};

struct BinParams {
  double log10emin;
  double discard_immediately;
  int bins;   // bins per decade
  int nbins;  // points per sign half
};

constexpr size_t kSpecSmemMax = 96 * 1024;  // private histograms up to 6144 bins per half

// Work items of the binning kernel: warp tiles of 32 columns x `rows` rows (a multiple of 8).
inline int64_t spec_tiles(int i0, int i1, int j0, int j1, int rows) {
  return (int64_t)((i1 - i0 + 31) / 32) * ((j1 - j0 + rows - 1) / rows);
}
// Rows of a warp tile for a call of `terms` terms.
int spec_tile_rows(int64_t terms);
cudaError_t spec_bin_launch(const SpecRegion* d_regs, int nreg, int64_t ntiles, int rows, const BinParams& bp,
                            double* pos, double* neg, bool dmnrg, cudaStream_t stream);

constexpr int kMatsChunk = 2048;  // terms of one CTA's pass of the Matsubara kernel
inline int64_t mats_chunks(int i0, int i1, int j0, int j1) {
  return ((int64_t)(i1 - i0) * (j1 - j0) + kMatsChunk - 1) / kMatsChunk;
}
// Matsubara sums: re[n] + i im[n] += factor w / (i w_n - E) for every term (accumulated).
cudaError_t spec_mats_launch(const SpecRegion* d_regs, int nreg, int64_t nchunks, const MatsParams& mp, double* re,
                             double* im, cudaStream_t stream);

}  // namespace nrg
