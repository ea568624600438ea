// gemm.cu -- batched, segmented FP64 GEMM on the FP64 tensor cores (DMMA m8n8k4).
//
// Used for every GEMM-shaped step of the NRG step core: the recalculation leaves
// product / transform / rotate (numerics_ublas.hpp:108-140 of the reference), the
// prod_fit products of the spectral algorithms, the divide-and-conquer merges and the
// Householder back-transform of the eigensolver. tcgen05.mma has no f64 kind on sm_100a,
// so FP64 tensor work goes through mma.sync DMMA.
//
// One CTA (4 warps, 2 x 2) computes a BT x BT tile of one output. K is walked in chunks of 16 over
// all segments of the output, through a ring of shared-memory stages filled by asynchronous
// copies (cp.async). A stage holds each operand in its own orientation (rows of 16 k, or rows
// of BT m or n), so copies of 16 bytes land where they come from in memory; operands that do
// not start or stride on 16 bytes take copies of 8. Either way a row is 4 doubles longer than
// its contents, which puts two lanes of a fragment load on each bank, the least there is.
#include "common.cuh"
#include "kernels.h"

#include <algorithm>

namespace nrg {
namespace {

constexpr int BK = kGemmBK, NT = kGemmThreads;
constexpr int LDK = BK + 4;  // row stride of an operand stored as rows of k

// Asynchronous copy global -> shared of the first `bytes` of 16 (8); the rest is zero-filled, and
// with 0 nothing is read (src must still be a valid address).
__device__ __forceinline__ void cp_async16(double* dst, const double* src, int bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async8(double* dst, const double* src, int bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Copies of one operand of a segment: a thread has the same column of every row it copies, so an
// address is a pointer that moves by a constant per chunk plus a constant per row, and only the
// edges of the matrix test anything. (The DMMA pipe shares its issue slots with all of this: with
// addresses worked out per element the kernel issued eight instructions for each DMMA.)
// kx = false: element (x, k) at src[x ld + k], stage rows of 16 k; kx = true: element at
// src[k ld + x], stage rows of BT x.
template <int BT>
struct OperandCopy {
  const double* p;     // first element of this thread's first row in the current chunk
  const double* safe;  // the matrix
  int64_t rstep;     // from one of its rows to the next
  int64_t kstep;     // from chunk to chunk
  int r0, c;         // its first row and its column in the stage
  int rlim, clim;    // rows and columns of the matrix from the tile's corner (chunk-relative in k)
  bool kx, wide;

  __device__ __forceinline__ void set(const double* src, int64_t ld, bool kx_, int K, int X, int x0) {
    kx = kx_;
    safe = src;
    wide = ((reinterpret_cast<uintptr_t>(src) & 15) | (ld & 1)) == 0;  // tile corners are multiples of 16
    const int per = (kx ? BT : BK) / (wide ? 2 : 1);  // copies per row
    const int tid = threadIdx.x;
    r0 = tid / per;
    c = (tid % per) * (wide ? 2 : 1);
    rstep = (NT / per) * ld;
    kstep = kx ? BK * ld : BK;
    p = src + (kx ? r0 * ld + x0 + c : (int64_t)(x0 + r0) * ld + c);
    rlim = kx ? K : X - x0;
    clim = kx ? X - x0 : K;
  }

  __device__ __forceinline__ void copy(double* dst) {
    const int rows = kx ? BK : BT, cols = kx ? BT : BK, lds = kx ? BT + 4 : LDK, dr = wide ? 2 * NT / cols : NT / cols;
    double* d = dst + r0 * lds + c;
    const double* q = p;
    if (rlim >= rows && clim >= cols) {
      if (wide) {
#pragma unroll
        for (int i = 0; i < BT * BK / 2 / NT; i++, q += rstep, d += dr * lds) cp_async16(d, q, 16);
      } else {
#pragma unroll
        for (int i = 0; i < BT * BK / NT; i++, q += rstep, d += dr * lds) cp_async8(d, q, 8);
      }
    } else {  // an edge: zeros beyond it (nothing is read for 0 bytes, the address stays valid)
      const int left = clim - c;
      const int bytes = left <= 0 ? 0 : wide ? 8 * min(2, left) : 8;
      if (wide) {
#pragma unroll
        for (int i = 0; i < BT * BK / 2 / NT; i++, q += rstep, d += dr * lds) {
          const int by = r0 + i * dr < rlim ? bytes : 0;
          cp_async16(d, by ? q : safe, by);
        }
      } else {
#pragma unroll
        for (int i = 0; i < BT * BK / NT; i++, q += rstep, d += dr * lds) {
          const int by = r0 + i * dr < rlim ? bytes : 0;
          cp_async8(d, by ? q : safe, by);
        }
      }
    }
    p += kstep;
    (kx ? rlim : clim) -= BK;
  }
};

// Doubles of an operand's stage: the larger of the two orientations.
__host__ __device__ constexpr int stage_doubles(int bt) {
  return bt * LDK > BK * (bt + 4) ? bt * LDK : BK * (bt + 4);
}

// acc += alpha A B for one chunk, A and B in the given orientations (true: rows of m or n).
template <int BM, int BN, bool AKX, bool BKX>
__device__ __forceinline__ void tile_products(const double* As, const double* Bs, double alpha,
                                              double (&acc)[BM / 16][BN / 16][2]) {
  constexpr int FM = BM / 16, FN = BN / 16;
  constexpr int sam = AKX ? 1 : LDK, sak = AKX ? BM + 4 : 1, sbn = BKX ? 1 : LDK, sbk = BKX ? BN + 4 : 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fr = lane >> 2, fc = lane & 3;
  const double* as = As + ((warp >> 1) * (BM / 2) + fr) * sam + fc * sak;
  const double* bs = Bs + ((warp & 1) * (BN / 2) + fr) * sbn + fc * sbk;
#pragma unroll
  for (int kk = 0; kk < BK; kk += 4) {
    double a[FM], b[FN];
#pragma unroll
    for (int i = 0; i < FM; i++) a[i] = as[i * 8 * sam + kk * sak];
#pragma unroll
    for (int j = 0; j < FN; j++) b[j] = bs[j * 8 * sbn + kk * sbk];
    if (alpha != 1.0) {
#pragma unroll
      for (int i = 0; i < FM; i++) a[i] *= alpha;
    }
#pragma unroll
    for (int i = 0; i < FM; i++)
#pragma unroll
      for (int j = 0; j < FN; j++) dmma884(acc[i][j][0], acc[i][j][1], a[i], b[j]);
  }
}

// One BM x BN output tile `tt` (row-major tile order) of output o, whose segments are
// segs[o.seg0 .. o.seg0 + o.nseg).
template <int BM, int BN, int STAGES>
__device__ __forceinline__ void gemm_tile(const GemmOut& o, const GemmSeg* __restrict__ segs, int tt) {
  extern __shared__ __align__(16) double gsm[];  // STAGES x (A, B)
  constexpr int SA = stage_doubles(BM), SB = stage_doubles(BN);
  constexpr int FM = BM / 16, FN = BN / 16;  // a warp's tile is FM x FN DMMA tiles
  const int tiles_n = (o.N + BN - 1) / BN;
  const int m0 = (tt / tiles_n) * BM, n0 = (tt % tiles_n) * BN;
  if (m0 >= o.M) return;  // outputs whose row count is set on the device may shrink

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp >> 1) * (BM / 2), wn = (warp & 1) * (BN / 2);
  const int fr = lane >> 2, fc = lane & 3;

  // The accumulators start from beta*C: the loads of C go out beside the first operand loads
  // instead of after the last product, which matters for the short-K updates (K = 128 of the
  // back-transform), where one exposed load latency is a large part of a tile's time.
  double acc[FM][FN][2];
  const bool addc = o.beta != 0.0;
#pragma unroll
  for (int i = 0; i < FM; i++) {
    const int r = m0 + wm + i * 8 + fr;
#pragma unroll
    for (int j = 0; j < FN; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = n0 + wn + j * 8 + 2 * fc + h;
        acc[i][j][h] = (addc && r < o.M && c < o.N) ? o.beta * o.C[(int64_t)r * o.ldc + c] : 0.0;
      }
  }

  // Flatten (segment, k-chunk) into one sequence of steps.
  int total = 0;
  for (int s = 0; s < o.nseg; s++) total += (segs[o.seg0 + s].K + BK - 1) / BK;

  if (total > 0) {
    int cs = -1, left = 0;  // segment of the next chunk to copy and what is left of its K
    OperandCopy<BM> ca;
    OperandCopy<BN> cb;
    // orientation and factor of the chunks in the ring, two bits and a double per stage
    unsigned orient = 0;
    double alphas[STAGES], galpha = 1.0;
    auto copy_next = [&](int st) {
      if (left <= 0) {  // first chunk of the next segment
        do cs++; while (segs[o.seg0 + cs].K <= 0);
        const GemmSeg& g = segs[o.seg0 + cs];
        left = g.K;
        galpha = g.alpha;
        ca.set(g.A, g.lda, g.transA != 0, left, o.M, m0);
        cb.set(g.B, g.ldb, g.transB == 0, left, o.N, n0);
      }
      double* As = gsm + (size_t)st * (SA + SB);
      ca.copy(As);
      cb.copy(As + SA);
      left -= BK;
      orient = (orient & ~(3u << 2 * st)) | ((ca.kx ? 1u : 0u) | (cb.kx ? 2u : 0u)) << 2 * st;
#pragma unroll
      for (int q = 0; q < STAGES; q++)
        if (q == st) alphas[q] = galpha;
    };
#pragma unroll
    for (int q = 0; q < STAGES - 1; q++) {
      if (q < total) {
        copy_next(q);
      }
      cp_async_commit();
    }
    for (int step = 0, st = 0; step < total; step++, st = st + 1 == STAGES ? 0 : st + 1) {
      // One barrier per chunk: after it chunk `step` has landed for every thread and every thread
      // has finished reading the stage of chunk step-1, which the next copy overwrites.
      cp_async_wait<STAGES - 2>();
      __syncthreads();
      const int nst = st == 0 ? STAGES - 1 : st - 1;
      if (step + STAGES - 1 < total) {
        copy_next(nst);
      }
      cp_async_commit();
      double alpha = alphas[0];
#pragma unroll
      for (int q = 1; q < STAGES; q++)
        if (q == st) alpha = alphas[q];
      const double* as = gsm + (size_t)st * (SA + SB);
      switch (orient >> 2 * st & 3) {  // constant strides for each orientation
        case 0: tile_products<BM, BN, false, false>(as, as + SA, alpha, acc); break;
        case 1: tile_products<BM, BN, true, false>(as, as + SA, alpha, acc); break;
        case 2: tile_products<BM, BN, false, true>(as, as + SA, alpha, acc); break;
        default: tile_products<BM, BN, true, true>(as, as + SA, alpha, acc); break;
      }
    }
    cp_async_wait<0>();
  }

  // Epilogue: C = acc (= beta*C + the products).
#pragma unroll
  for (int i = 0; i < FM; i++) {
    const int r = m0 + wm + i * 8 + fr;
    if (r >= o.M) continue;
#pragma unroll
    for (int j = 0; j < FN; j++) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = n0 + wn + j * 8 + 2 * fc + h;
        if (c < o.N) o.C[(int64_t)r * o.ldc + c] = acc[i][j][h];
      }
    }
  }
}

template <int BM, int BN, int STAGES, int MINB>
__global__ void __launch_bounds__(NT, MINB) gemm_batch_kernel(const GemmOut* __restrict__ outs,
                                                              const GemmSeg* __restrict__ segs, int nout) {
  // Locate the output that owns this tile (binary search over its first tile's number).
  const int t = blockIdx.x;
  int lo = 0, hi = nout - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((BM == kGemmBM ? outs[mid].tile0 : outs[mid].tile0s) <= t) lo = mid; else hi = mid - 1;
  }
  const GemmOut o = outs[lo];
  gemm_tile<BM, BN, STAGES>(o, segs, t - (BM == kGemmBM ? o.tile0 : o.tile0s));
}

// Single output with a single segment, both passed by value (no descriptor memory).
template <int BM, int BN, int STAGES, int MINB>
__global__ void __launch_bounds__(NT, MINB) gemm_one_kernel(const __grid_constant__ GemmOut o,
                                                            const __grid_constant__ GemmSeg g) {
  gemm_tile<BM, BN, STAGES>(o, &g, blockIdx.x);
}

// Measured on B200 (TFLOP/s; even / odd leading dimensions; 35.4 is cuBLAS's rate): 64 products of order
// 1024 31.5 / 30.6, where copies of 8 bytes with an address computed for each and runtime strides gave
// 25.6 / 25.6; updates of 256 1024 x 1024 outputs with K = 128 25.7 / 24.2 (20.6 / 20.2). Two stages with
// four CTAs per SM beat three with three (30.6, 23.2) and 128 x 64 tiles (30.4, 21.6).
// Tiles of 32 x 32 serve calls that would not give every SM its four CTAs: one product of order 456 takes
// 24 us instead of 42, seven of them 73 instead of 88, but ten 120 instead of 109.
constexpr int kStagesL = 2, kMinL = 4, kStagesS = 3, kMinS = 5;
template <int BM, int BN, int STAGES>
constexpr size_t gemm_smem() { return sizeof(double) * (stage_doubles(BM) + stage_doubles(BN)) * STAGES; }

// Dynamic shared memory beyond 48 KB has to be asked for, per device and kernel; every launch does.
template <typename F>
cudaError_t allow_smem(F* fn, size_t bytes) {
  return cudaFuncSetAttribute(reinterpret_cast<const void*>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)bytes);
}

// Small tiles when the large ones would leave SMs idle.
bool small_tiles(int tiles) { return tiles <= kGemmSmallTiles; }

// Element e of the batch belongs to the last term whose off <= e; one product per element.
__global__ void __launch_bounds__(256) row_scale_kernel(const RowScale* __restrict__ terms, int nterm,
                                                        int64_t total) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    int lo = 0, hi = nterm - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (terms[mid].off <= e) lo = mid; else hi = mid - 1;
    }
    const RowScale& r = terms[lo];
    const int64_t q = e - r.off;
    const int k = (int)(q / r.cols), c = (int)(q % r.cols);
    const double b = r.transB ? r.B[(int64_t)c * r.ldb + k] : r.B[(int64_t)k * r.ldb + c];
    r.T[q] = r.d[k] * b;
  }
}

}  // namespace

cudaError_t row_scale_launch(const RowScale* d_terms, int nterm, int64_t total, cudaStream_t stream) {
  if (nterm <= 0 || total <= 0) return cudaSuccess;
  const int64_t blocks = std::min<int64_t>((total + 255) / 256, 148 * 16);
  row_scale_kernel<<<(unsigned)blocks, 256, 0, stream>>>(d_terms, nterm, total);
  return cudaGetLastError();
}

cudaError_t gemm_one_launch(const GemmOut& o, const GemmSeg& g, cudaStream_t stream) {
  const int tiles = gemm_tiles(o.M, o.N, kGemmBM, kGemmBN), tiles_s = gemm_tiles(o.M, o.N, kGemmSmallBM, kGemmSmallBM);
  if (tiles <= 0) return cudaSuccess;
  GemmOut oo = o;
  oo.seg0 = 0;
  oo.nseg = 1;
  oo.tile0 = oo.tile0s = 0;
  if (small_tiles(tiles)) {
    constexpr size_t sm = gemm_smem<kGemmSmallBM, kGemmSmallBM, kStagesS>();
    cudaError_t e = allow_smem(gemm_one_kernel<kGemmSmallBM, kGemmSmallBM, kStagesS, kMinS>, sm);
    if (e != cudaSuccess) return e;
    gemm_one_kernel<kGemmSmallBM, kGemmSmallBM, kStagesS, kMinS><<<tiles_s, NT, sm, stream>>>(oo, g);
  } else {
    constexpr size_t sm = gemm_smem<kGemmBM, kGemmBN, kStagesL>();
    cudaError_t e = allow_smem(gemm_one_kernel<kGemmBM, kGemmBN, kStagesL, kMinL>, sm);
    if (e != cudaSuccess) return e;
    gemm_one_kernel<kGemmBM, kGemmBN, kStagesL, kMinL><<<tiles, NT, sm, stream>>>(oo, g);
  }
  return cudaGetLastError();
}

cudaError_t gemm_batch_launch(const GemmOut* d_outs, const GemmSeg* d_segs, int nout, int ntiles, int ntiles_s,
                              cudaStream_t stream) {
  if (nout <= 0 || ntiles <= 0) return cudaSuccess;
  if (small_tiles(ntiles)) {
    constexpr size_t sm = gemm_smem<kGemmSmallBM, kGemmSmallBM, kStagesS>();
    cudaError_t e = allow_smem(gemm_batch_kernel<kGemmSmallBM, kGemmSmallBM, kStagesS, kMinS>, sm);
    if (e != cudaSuccess) return e;
    gemm_batch_kernel<kGemmSmallBM, kGemmSmallBM, kStagesS, kMinS><<<ntiles_s, NT, sm, stream>>>(d_outs, d_segs, nout);
  } else {
    constexpr size_t sm = gemm_smem<kGemmBM, kGemmBN, kStagesL>();
    cudaError_t e = allow_smem(gemm_batch_kernel<kGemmBM, kGemmBN, kStagesL, kMinL>, sm);
    if (e != cudaSuccess) return e;
    gemm_batch_kernel<kGemmBM, kGemmBN, kStagesL, kMinL><<<ntiles, NT, sm, stream>>>(d_outs, d_segs, nout);
  }
  return cudaGetLastError();
}

}  // namespace nrg
