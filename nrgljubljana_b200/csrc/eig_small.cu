// eig_small.cu -- one CTA per block, whole eigenproblem on one SM (n <= kSmallMaxN).
//
// Replaces LAPACK dsyev as called by diagonalise_dsyev (c++/diag.hpp:62-82 of the
// reference) for the small symmetry blocks of an NRG step: the row-major input with its
// upper triangle set is symmetrised into shared memory, reduced to tridiagonal form by
// Householder reflections in registers, solved by divide and conquer, and the reflections are
// applied to the eigenvectors. Eigenvalues are written ascending and
// eigenvectors as rows (the layout of copy_vec, c++/diag.hpp:41-48).
// A diagonal block (a subspace with one ancestor) is only sorted: 40 of order 60 take 44 us, where the
// reduction and the merges take 137.
// Measured on B200, nine blocks of order 3-29: 435 us with an implicit QL iteration, 78 us so (order
// 29: reduction 36, divide and conquer 60, back-transform 8 thousand cycles); 16 blocks of order
// 8-64 beside a step's larger ones 1600 and 168 us.
#include "eig_small.cuh"
#include "kernels.h"

#include <vector>

namespace nrg {
namespace {

__host__ __device__ inline int small_ld(int n) { return (n & 1) ? n : n + 1; }  // odd stride: no bank conflicts

__host__ __device__ inline size_t small_smem_bytes(int n) {
  // Z (first the matrix), U (first the (v, w) copies: 16 n <= n ld or the slack), V packed, d, e,
  // taus, yb, rb, the scratch of the divide and conquer, ctl, perm
  const size_t ld = small_ld(n), u = n * ld > 16 * (size_t)n ? n * ld : 16 * (size_t)n;
  return sizeof(double) * (n * ld + (u + 1) / 2 * 2 + (size_t)n * (n - 1) / 2 + 7 * (size_t)n) + dc_scratch_bytes(n) +
         sizeof(int) * ((size_t)n + 12) + 32;
}

template <int R, int T = kCtaEigThreads>
NRG_DEV void solve_block(const EigBlock& b, double* sm) {
  const int n = b.n, ld = small_ld(n), tid = threadIdx.x;
  const size_t un = n * ld > 16 * n ? n * ld : 16 * n;
  double* U = sm;  // 16-byte aligned: the (v, w) copies are read as pairs
  double* Z = U + (un + 1) / 2 * 2;
  double* d = Z + (size_t)n * ld;
  double* e = d + n;
  double* taus = e + n;
  double* yb = taus + n;   // 2n
  double* rb = yb + 2 * n;  // 2n
  double* V = rb + 2 * n;
  double* scr = V + (size_t)n * (n - 1) / 2;
  int* perm = reinterpret_cast<int*>(reinterpret_cast<char*>(scr) + dc_scratch_bytes(n));
  int* ctl = perm + n;

  // Load the upper triangle and symmetrise; flag non-finite input.
  int bad = 0, off = 0;
  for (int idx = tid; idx < n * n; idx += T) {
    const int i = idx / n, j = idx - i * n;
    if (j >= i) {
      const double h = b.H[idx];
      if (!isfinite(h)) bad = 1;
      if (j > i && h != 0.0) off = 1;
      Z[i * ld + j] = h;
      Z[j * ld + i] = h;
    }
  }
  int st = __syncthreads_or(bad) ? -2 : 0;
  const bool diagonal = !__syncthreads_or(off);
  if (!st && diagonal) {
    if (tid < n) d[tid] = Z[tid * ld + tid];
    __syncthreads();
    if (tid < n) Z[tid * ld + tid] = 1.0;
  } else if (!st) {
    cta_tridiagonalise<R, T>(Z, ld, n, d, e, taus, V, yb, rb, U);
    __syncthreads();
    bad = 0;
    if (tid < n) bad = !isfinite(d[tid]) || (tid < n - 1 && !isfinite(e[tid]));  // overflow on the way
    if (__syncthreads_or(bad)) st = -2;
  }
  if (!st && !diagonal) st = smem_dc<R, T>(d, e, n, Z, U, ld, scr, ctl);
  if (st) {
    if (tid == 0) *b.info = st;
    for (int r = tid; r < n; r += T) b.evals[r] = nan("");
    for (int idx = tid; idx < n * n; idx += T) b.evecs[idx] = nan("");
    return;
  }
  if (!diagonal) cta_apply_q<R, T>(Z, ld, n, taus, V);
  if (tid < n) {  // ascending order
    const double di = d[tid];
    int rank = 0;
    for (int j = 0; j < n; j++) rank += d[j] < di || (d[j] == di && j < tid);
    perm[rank] = tid;
    b.evals[rank] = di;
  }
  if (tid == 0) *b.info = 0;
  __syncthreads();
  for (int idx = tid; idx < n * n; idx += T) {
    const int r = idx / n, j = idx - r * n;
    b.evecs[idx] = Z[perm[r] * ld + j];
  }
}

// Blocks of order up to 32 R (kTinyEigN for 64 threads), CTAS of them at once on an SM. Calls of many more blocks
// than SMs are bound by the SMs' time, so the small ones get launches with fewer registers or threads
// (eig_small_split). Measured on B200, us of a call of 6000 blocks of one order, with an implicit QL iteration /
// one kernel of 255 registers for all orders / so: order 4 308 / 687 / 294, 8 532 / 1125 / 403, 16 1219 / 1796 / 553, 24
// 2255 / 2711 / 1528, 32 3632 / 2991 / 1690, 64 27650 / 7158 / 4902. 300 of order 24 with one, two and three CTAs
// per SM 222, 172 and 138; 64 threads with 16 CTAs (64 registers) take as long as with 8. Calls that
// the SMs hold at once take one CTA per SM, without spilled registers: nine of order 8-64 192, 202 with two.
template <int R, int T, int CTAS>
__global__ void __launch_bounds__(T, CTAS) eig_small_kernel(const EigBlock* __restrict__ blocks) {
  extern __shared__ __align__(16) double sm[];
  const EigBlock b = blocks[blockIdx.x];
  if constexpr (R > 2) {
    if (b.n > 64) return solve_block<3, T>(b, sm);
  }
  if constexpr (R > 1) {
    if (b.n > 32) return solve_block<2, T>(b, sm);
  }
  solve_block<1, T>(b, sm);
}

template <int R, int T, int CTAS>
cudaError_t launch(const EigBlock* d_blocks, int nblk, int maxn, cudaStream_t stream) {
  const size_t smem = small_smem_bytes(maxn);
  const cudaError_t err = cudaFuncSetAttribute(eig_small_kernel<R, T, CTAS>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err != cudaSuccess) return err;
  eig_small_kernel<R, T, CTAS><<<nblk, T, smem, stream>>>(d_blocks);
  return cudaGetLastError();
}

}  // namespace

// Launches follow one another, so a class of orders is cut off only where the smaller blocks are many: 600 of
// order 2-33 take 293 us with a launch for each of the three classes, 188 in one.
std::vector<int> eig_small_split(const std::vector<int>& n, int nsm) {
  auto cls = [](int m) { return m <= kTinyEigN ? 0 : m <= 32 ? 1 : m <= 64 ? 2 : 3; };
  std::vector<int> first;
  const int count = (int)n.size();
  for (int q = 0; q < count; q++)
    if (q == 0 || (cls(n[q]) != cls(n[q - 1]) && count - q > 6 * nsm)) first.push_back(q);
  return first;
}

cudaError_t eig_small_launch(const EigBlock* d_blocks, int nblk, int maxn, int nsm, cudaStream_t stream) {
  if (nblk <= 0) return cudaSuccess;
  if (maxn <= kTinyEigN) return launch<1, kTinyEigThreads, 8>(d_blocks, nblk, maxn, stream);
  if (maxn <= 32 && nblk > nsm) return launch<1, kCtaEigThreads, 3>(d_blocks, nblk, maxn, stream);
  if (maxn <= 64 && nblk <= nsm) return launch<2, kCtaEigThreads, 1>(d_blocks, nblk, maxn, stream);
  if (maxn <= 64) return launch<2, kCtaEigThreads, 2>(d_blocks, nblk, maxn, stream);
  return launch<3, kCtaEigThreads, 1>(d_blocks, nblk, maxn, stream);
}

}  // namespace nrg
