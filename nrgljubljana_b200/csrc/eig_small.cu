// eig_small.cu -- one CTA per block, whole eigenproblem on one SM (n <= kSmallMaxN).
//
// Replaces LAPACK dsyev as called by diagonalise_dsyev (c++/diag.hpp:62-82 of the
// reference) for the small symmetry blocks of an NRG step: the row-major input with its
// upper triangle set is symmetrised into shared memory, reduced to tridiagonal form by
// Householder reflections in registers, solved by divide and conquer, and the reflections are
// applied to the eigenvectors. Eigenvalues are written ascending and
// eigenvectors as rows (the layout of copy_vec, c++/diag.hpp:41-48).
// Measured on B200, nine blocks of order 3-29: 435 us with an implicit QL iteration, 78 us so (order
// 29: reduction 36, divide and conquer 60, back-transform 8 thousand cycles); 16 blocks of order
// 8-64 beside a step's larger ones 1600 and 168 us.
#include "eig_small.cuh"
#include "kernels.h"

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

template <int R>
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
  int bad = 0;
  for (int idx = tid; idx < n * n; idx += kCtaEigThreads) {
    const int i = idx / n, j = idx - i * n;
    if (j >= i) {
      const double h = b.H[idx];
      if (!isfinite(h)) bad = 1;
      Z[i * ld + j] = h;
      Z[j * ld + i] = h;
    }
  }
  int st = __syncthreads_or(bad) ? -2 : 0;
  if (!st) {
    if (n == 1) {
      if (tid == 0) d[0] = Z[0];
    } else {
      cta_tridiagonalise<R>(Z, ld, n, d, e, taus, V, yb, rb, U);
    }
    __syncthreads();
    bad = 0;
    if (tid < n) bad = !isfinite(d[tid]) || (tid < n - 1 && !isfinite(e[tid]));  // overflow on the way
    if (__syncthreads_or(bad)) st = -2;
  }
  if (!st) st = smem_dc<R>(d, e, n, Z, U, ld, scr, ctl);
  if (st) {
    if (tid == 0) *b.info = st;
    for (int r = tid; r < n; r += kCtaEigThreads) b.evals[r] = nan("");
    for (int idx = tid; idx < n * n; idx += kCtaEigThreads) b.evecs[idx] = nan("");
    return;
  }
  cta_apply_q<R>(Z, ld, n, taus, V);
  if (tid < n) {  // ascending order
    const double di = d[tid];
    int rank = 0;
    for (int j = 0; j < n; j++) rank += d[j] < di || (d[j] == di && j < tid);
    perm[rank] = tid;
    b.evals[rank] = di;
  }
  if (tid == 0) *b.info = 0;
  __syncthreads();
  for (int idx = tid; idx < n * n; idx += kCtaEigThreads) {
    const int r = idx / n, j = idx - r * n;
    b.evecs[idx] = Z[perm[r] * ld + j];
  }
}

__global__ void __launch_bounds__(kCtaEigThreads, 1) eig_small_kernel(const EigBlock* __restrict__ blocks) {
  extern __shared__ __align__(16) double sm[];
  const EigBlock b = blocks[blockIdx.x];
  if (b.n <= 32) solve_block<1>(b, sm);
  else if (b.n <= 64) solve_block<2>(b, sm);
  else solve_block<3>(b, sm);
}

}  // namespace

cudaError_t eig_small_launch(const EigBlock* d_blocks, int nblk, int maxn, cudaStream_t stream) {
  if (nblk <= 0) return cudaSuccess;
  const size_t smem = small_smem_bytes(maxn);
  cudaError_t err = cudaFuncSetAttribute(eig_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err != cudaSuccess) return err;
  eig_small_kernel<<<nblk, kCtaEigThreads, smem, stream>>>(d_blocks);
  return cudaGetLastError();
}

}  // namespace nrg
