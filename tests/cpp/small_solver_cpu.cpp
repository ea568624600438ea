// Host build of the one-CTA eigensolver (csrc/eig_small.cu) behind a C interface; the Python
// test generates the include files.
#include "cta_emulator.h"

namespace nrg {
struct EigBlock {
  double *H, *evals, *evecs;
  int* info;
  int n;
};
}  // namespace nrg
#include "eig_small.cu"

using namespace nrg;

// Status of the block (or of emu_run) with the CTA of `threads`; H is n x n, both triangles set.
extern "C" int solve(int n, int threads, double* H, double* evals, double* evecs, double fill) {
  int info = 0;
  EigBlock b{H, evals, evecs, &info, n};
  const size_t smem = small_smem_bytes(n) / 8;
  const int run =
      threads == kTinyEigThreads ? emu_run(1, kTinyEigThreads, smem, fill, [&] { eig_small_kernel<1, kTinyEigThreads, 1>(&b); })
                                 : emu_run(1, kCtaEigThreads, smem, fill, [&] { eig_small_kernel<3, kCtaEigThreads, 1>(&b); });
  return run ? run : info;
}

// Divide and conquer alone: (d, e) -> eigenvalues (unsorted) in d, eigenvectors as rows of Z.
extern "C" int divide_and_conquer(int n, double* d, double* e, double* Z, double fill) {
  const int ld = small_ld(n);
  int st = 0;
  int* ctl = static_cast<int*>(calloc(64, sizeof(int)));
  std::vector<double> scr(dc_scratch_bytes(n) / 8 + 1, fill);
  const int run = emu_run(1, kCtaEigThreads, 2 * (size_t)n * ld, fill, [&] {
    double *z = emu_smem(), *u = z + n * ld;
    const int s = n <= 32   ? smem_dc<1>(d, e, n, z, u, ld, scr.data(), ctl)
                  : n <= 64 ? smem_dc<2>(d, e, n, z, u, ld, scr.data(), ctl)
                            : smem_dc<3>(d, e, n, z, u, ld, scr.data(), ctl);
    if (threadIdx.x == 0) {
      st = s;
      for (int i = 0; i < n; i++) std::copy(z + i * ld, z + i * ld + n, Z + i * n);
    }
  });
  free(ctl);
  return run ? run : st;
}
