// Host build of tridiag_dsm_kernel (csrc/eig_large.cu) behind a C interface; the Python test cuts the
// kernel out of its source into dsm_kernel.inc and gives its mbarrier and cluster helpers bodies.
#include "cta_emulator.h"

#include "eig_small.cuh"

namespace nrg {
constexpr int NBT = 128;
struct LargeBlock {
  double *H, *W1, *d, *e, *tau;
  int* info;
  int n, ldp;
};
#include "dsm_kernel.inc"
}  // namespace nrg

template <int C>
static int run(const nrg::LargeBlock* b, int slow) {
  return emu_run(C, nrg::kDsmThreads, nrg::dsm_smem_doubles(b->n, C) + 8, 0.0, [&] { nrg::tridiag_dsm_kernel<C>(b); },
                 slow);
}

// H (n x n, upper triangle) to d, e, tau and the reflectors in W1 (n x ldp); CTA `slow` of the C lags behind as far
// as the exchange lets it (-1: none).
extern "C" int reduce(int n, int C, int slow, double* H, double* W1, int ldp, double* d, double* e, double* tau) {
  int info = 0;
  const nrg::LargeBlock b{H, W1, d, e, tau, &info, n, ldp};
  const int st = C == 2 ? run<2>(&b, slow) : C == 4 ? run<4>(&b, slow) : C == 8 ? run<8>(&b, slow) : run<16>(&b, slow);
  return st ? st : info;
}
