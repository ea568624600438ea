// eig_large.cu -- batched FP64 symmetric eigensolver for blocks larger than kSmallMaxN.
//
// Replaces LAPACK dsyev/dsyevd as called by diagonalise() (c++/diag.hpp:62-115, 261-292
// of the reference) for the large symmetry blocks of an NRG step, with the output layout
// of copy_results (ascending eigenvalues, eigenvectors as rows, c++/diag.hpp:41-58).
//
// Pipeline per chunk of blocks (all blocks of the chunk advance together):
//   1. reduction to tridiagonal form A = Q T Q^T by Householder reflectors, several kernels side by
//      side by order and number of the blocks (reduction_plan): in the shared memory of a CTA or
//      a cluster, by groups of CTAs through L2, in two stages (eig_band.cu), or, in batches of many
//      blocks, one CTA per block streaming the lower triangle once per column (tridiag_kernel).
//   2. divide and conquer on T: leaves (<= kLeaf) by one in shared memory, merges
//      by rank-one tearing (Cuppen), deflation (small z and close poles with Givens
//      rotations), secular-equation roots with a two-pole rational model safeguarded by
//      bisection, Gu-Eisenstat recomputation of z for orthogonal vectors, and the merge
//      products as FP64 tensor-core GEMMs that skip the zero blocks of the children.
//   3. sort of the eigenvalues and row permutation of the eigenvectors.
//   4. back-transform with the compact-WY form of Q, panels of NBT reflectors, as GEMMs.
// Eigenvectors are kept as ROWS throughout (Zt = Z^T), the layout of the output.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <functional>
#include <vector>

#include "common.cuh"
#include "band.h"
#include "eig_large.h"
#include "eig_small.cuh"

namespace nrg {
namespace {

constexpr int kTriThreads = 128;
constexpr int NB = 16;     // tridiagonalisation panel width
constexpr int NBT = 128;   // back-transform panel width
constexpr int kLeaf = 64;  // divide-and-conquer leaves have at most this order
constexpr int kMaxLargeN = 10240;  // the rows that the threads of tridiag_grid_kernel<20> hold
// Merge nodes whose prep arrays exceed this many bytes keep them in global scratch (kPrepGlobalB
// bytes per row of the block) instead of shared memory.
constexpr size_t kPrepSmemMax = 200 * 1024;
constexpr size_t kPrepGlobalB = 80;

// Deflation rotation of the eigenvector rows p and j (rows of the node): (p, j) <- (c p - s j,
// s p + c j). sup: supports of the two rows before it, p's in bits 0-1 and j's in bits 2-3 (1: the
// first child's columns, 2: the second's); outside its support a row is zero (and not stored).
struct DcRot {
  double c, s;
  int p, j, sup, pad;
};

struct LargeBlock {
  double* H;      // input (consumed); then the eigenvector rows of T during divide and
                  // conquer; then the VT factors of the back-transform
  double* evals;
  double* evecs;  // output; scratch for the merge matrices during divide and conquer
  double* W1;     // n x ldp: packed lower triangle being reduced; Householder vectors after
  double* W2;     // n x n: panel W of the reduction; grouped rows of a merge; back-transform W
  double* d;
  double* e;
  double* tau;
  double* lam;    // eigenvalues of the current divide-and-conquer nodes
  double* dsort;  // per node: non-deflated poles, ascending
  double* dgrp;   // per node: non-deflated poles, grouped order
  double* zgrp;   // per node: z in grouped order; then z-hat
  double* rorg;   // per node: root j is rorg[j] + rtau[j], rorg the pole it was measured from
  double* rtau;
  double* GT;     // per back-transform panel of nb reflectors: Gram matrix V^T V then T (nb x nb each)
  int* rank;      // per node: sorted position of grouped entry
  int* perm;      // final eigenvalue order
  char* pscr;     // kPrepGlobalB bytes per row: merge-prep arrays of nodes too large for shared memory
  int2* slot;     // per node row: (grouped slot, support) of the eigenvector row
  DcRot* rot;     // per node: deflation rotations, in order
  double* gx;     // exchange buffers of tridiag_grid_kernel
  int* info;
  int n, npanel;
  int ldp, pad_;  // leading dimension of the packed lower triangle in W1 (multiple of 32)
};

struct DcLeaf {
  int blk, a0, a1, pad;
};

struct DcNode {
  int blk, a, m, b;
  int gout;  // index of the first of its two GEMM outputs in the level's GEMM arrays
  int pad;
};

struct DcState {
  int K, k1, k2, k3;
  double rho;
  int nrot;
  int ex;  // poles, rho and roots of the merge are divided by 2^ex (about the size of the merged matrix)
};

// ---------------------------------------------------------------- tridiagonalisation

// block_sum_1b with warp_sum_mma for both levels (at most 32 warps).
NRG_DEV double block_sum_mma(double x, double* red, int& phase) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  x = warp_sum_mma(x);
  double* b = red + 32 * (phase & 1);
  phase++;
  if (lane == 0) b[wid] = x;
  __syncthreads();
  return warp_sum_mma(lane < nw ? b[lane] : 0.0);
}

// The sum over all lanes of x[c] for c = lane / 4, by DMMAs: a matrix with a one in row c and its product
// with the lanes' x[c] put the sums over the lanes of equal l/4 into row c; a last one sums each row.
NRG_DEV double colsum8_mma(const double (&x)[8], int lane) {
  double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0, e0 = 0.0, e1 = 0.0;
#pragma unroll
  for (int c = 0; c < 8; c += 2) {
    dmma884(a0, a1, lane >> 2 == c ? 1.0 : 0.0, x[c]);
    dmma884(b0, b1, lane >> 2 == c + 1 ? 1.0 : 0.0, x[c + 1]);
  }
  dmma884(e0, e1, (a0 + a1) + (b0 + b1), 1.0);
  return e0;
}

// ---- bulk asynchronous copies (TMA, non-multicast) into the CTA's own shared memory
NRG_DEV unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

NRG_DEV void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

NRG_DEV void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// Orders this thread's earlier generic-proxy global writes before later bulk (async-proxy)
// reads of the same memory.
NRG_DEV void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// Orders this thread's earlier generic-proxy accesses of shared memory before later bulk copies into it.
NRG_DEV void fence_proxy_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

NRG_DEV void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// Acquire a tensor map that lives in global memory and was written by a host copy: orders the
// copy's generic-proxy writes before this thread's tensormap-proxy reads of the 128-byte map,
// so that no descriptor cached from an earlier map at the same address is used. The maps are
// rewritten at the same addresses for every chunk of blocks and every call.
NRG_DEV void tmap_acquire(const CUtensorMap* map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
}

// Bounded wait for phase `parity` of an mbarrier; false if the bound ran out.
NRG_DEV bool mbar_wait(uint64_t* bar, unsigned parity, int bound = (1 << 26)) {
  const unsigned a = smem_u32(bar);
  for (int it = 0; it < bound; it++) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// 2-D bulk tensor copy (TMA, non-multicast) of one box at coordinates (x, y) into this
// CTA's shared memory, completing on an mbarrier, with an L2 eviction-priority hint (an access policy
// from createpolicy): the slabs of a trailing triangle that is streamed once per column and does not
// fit in L2 go first, so that the panel's vectors (read twice per column) stay.
NRG_DEV void tma_load_2d_hint(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, "
      "%3}], [%4], %5;" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}

NRG_DEV uint64_t l2_evict_first_policy() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// Loads and stores of the panel's vectors (V and W columns, re-read twice per column of
// the panel) with an evict-last L2 hint, so that the streamed slabs do not push them out.
NRG_DEV uint64_t l2_evict_last_policy() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
NRG_DEV double ld_keep(const double* a, uint64_t pol) {
  double v;
  asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(a), "l"(pol));
  return v;
}
NRG_DEV void st_keep(double* a, double v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.f64 [%0], %1, %2;" ::"l"(a), "d"(v), "l"(pol) : "memory");
}

constexpr int kTriStages = 3;              // slabs in flight per warp
constexpr int kSlabRows = 64;              // rows of a slab (two per lane)
constexpr int kSlabD = kSlabRows * 8;      // doubles per slab: 64 rows x 8 columns
constexpr int kTriWarps = kTriThreads / 32;

// Length of a vector of the product: the last slab of a column group may end this far below row n-1.
__host__ __device__ inline int tri_pad(int n) { return (n + 7) / 8 * 8 + kSlabRows; }

// y += A(s0:n, s0:n) v, with v(s0) replaced by vs. A is the packed lower triangle (A(i, j) =
// P[j*ld + i] for i >= j, zero above the diagonal and in the padding) behind the 2-D tensor map `tmap`
// (inner extent ld rows, outer extent n columns, box 64 x 8). The triangle is cut into slabs of 64 rows
// x 8 columns, those of a column group from its diagonal down (slabs of aligned rows read a tenth more at
// order 900); the slabs, column group by column group, are split evenly between the warps, and each warp
// streams its slabs through a ring of kTriStages shared-memory buffers, one TMA box copy per slab
// completing on the buffer's mbarrier. A lane owns rows l and l+32 of the slab. A column group's sums stay
// in registers down the group and cross the lanes once at its end; the row sums are added in
// each slab to the warp's own copy of y, which takes no shuffles (walking along the rows instead costs a
// transposed sum of 8 columns and shared-memory atomics in every slab). y has ny copies of vp numbers,
// one per warp or else (large orders) shared by pairs of warps with atomics; v is zero in n .. vp-1.
// Rows of y before s0 take sums that nothing reads.
// `parity` holds the warp's mbarrier phase bits across calls. `between` is called while the first
// copies are under way.
template <typename F>
NRG_DEV void symv_lower(const CUtensorMap* tmap, int n, int s0, const double* v, double vs, double* y, int ny, int vp,
                        double* ring, uint64_t* bars, unsigned& parity, int* err, uint64_t policy, const F& between) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // column groups u = gl - j/8 from the last one (u = 0) to the one of s0; u/8 + 1 slabs each, so that
  // 4 a (a + 1) slabs belong to the 8 a last groups
  const int gl = (n - 1) >> 3, U1 = gl - (s0 >> 3) + 1;
  const int S = 4 * (U1 >> 3) * ((U1 >> 3) + 1) + (U1 & 7) * ((U1 >> 3) + 1);
  const int f0 = (int)((long long)S * warp / kTriWarps), f1 = (int)((long long)S * (warp + 1) / kTriWarps);
  int a8 = 0;
  while (4 * (a8 + 1) * (a8 + 2) < S - f0) a8++;
  const int rem = S - f0 - 4 * a8 * (a8 + 1);  // slabs left in the octet of groups, this one included
  int u = 8 * a8 + (rem - 1) / (a8 + 1), m = (u - 8 * a8 + 1) * (a8 + 1) - rem;
  double* myring = ring + (size_t)warp * kTriStages * kSlabD;
  uint64_t* mybar = bars + warp * kTriStages;
  auto advance = [](int& m_, int& u_) {
    if (m_ < u_ >> 3) {
      m_++;
    } else {
      u_--;
      m_ = 0;
    }
  };
  auto issue = [&](int m_, int u_, int st) {
    if (lane == 0) {
      mbar_expect_tx(mybar + st, (unsigned)(kSlabD * sizeof(double)));
      tma_load_2d_hint(myring + st * kSlabD, tmap, 8 * (gl - u_) + m_ * kSlabRows, 8 * (gl - u_), mybar + st, policy);
    }
  };
  int pm = m, pu = u;
  for (int t = 0; t < min(kTriStages, f1 - f0); t++) {
    issue(pm, pu, t);
    advance(pm, pu);
  }
  between();
  double* yw = y + (size_t)(warp % ny) * vp;
  const bool own = ny == kTriWarps;
  auto value = [&](int i) { return i > s0 ? v[i] : (i == s0 ? vs : 0.0); };
  double vj[8], cp[8];
  bool first = true;
  int st = 0;
  for (int f = f0; f < f1; f++) {
    const int j0 = 8 * (gl - u);
    if (first) {
#pragma unroll
      for (int c = 0; c < 8; c++) {
        vj[c] = value(j0 + c);
        cp[c] = 0.0;
      }
      first = false;
    }
    const int ia = j0 + m * kSlabRows + lane, ib = ia + 32;
    const double va = value(ia), vb = value(ib);
    if (!mbar_wait(mybar + st, (parity >> st) & 1u)) {
      // a copy never completed: flag the block, wait (bounded) for the copies still in
      // flight so that none lands after this call, and stop streaming
      if (lane == 0) atomicExch(err, -5);
      parity ^= 1u << st;
      for (int g = f + 1; g < min(f + kTriStages, f1); g++) {
        st = st + 1 == kTriStages ? 0 : st + 1;
        mbar_wait(mybar + st, (parity >> st) & 1u, 1 << 22);
        parity ^= 1u << st;
      }
      return;
    }
    parity ^= 1u << st;
    const double* buf = myring + st * kSlabD;
    double a0[8], a1[8];
#pragma unroll
    for (int c = 0; c < 8; c++) {
      a0[c] = buf[c * kSlabRows + lane];
      a1[c] = buf[c * kSlabRows + 32 + lane];
    }
    double r0 = 0.0, r1 = 0.0, q0 = 0.0, q1 = 0.0;
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      r0 = fma(a0[c], vj[c], r0);
      r1 = fma(a1[c], vj[c], r1);
      q0 = fma(a0[c + 1], vj[c + 1], q0);
      q1 = fma(a1[c + 1], vj[c + 1], q1);
    }
    if (m > 0) {
#pragma unroll
      for (int c = 0; c < 8; c++) cp[c] = fma(a0[c], va, fma(a1[c], vb, cp[c]));
    } else {  // on the diagonal: its elements count in the row sums only
#pragma unroll
      for (int c = 0; c < 8; c++) {
        cp[c] = fma(a0[c], c == lane ? 0.0 : va, fma(a1[c], vb, cp[c]));
      }
    }
    r0 += q0;
    r1 += q1;
    // the slab's reads by all lanes come before the copy that overwrites it
    fence_proxy_async_shared();
    __syncwarp();
    if (f + kTriStages < f1) {  // refill this stage with the slab kTriStages ahead
      issue(pm, pu, st);
      advance(pm, pu);
    }
    if (own) {
      yw[ia] += r0;
      yw[ib] += r1;
    } else {
      atomicAdd(yw + ia, r0);
      atomicAdd(yw + ib, r1);
    }
    st = st + 1 == kTriStages ? 0 : st + 1;
    if (m == u >> 3 || f + 1 == f1) {  // the end of the group's part here
      const double cs = colsum8_mma(cp, lane);
      __syncwarp();
      if ((lane & 3) == 0) {
        double* yj = yw + j0 + (lane >> 2);
        if (own) *yj += cs;
        else atomicAdd(yj, cs);
      }
      __syncwarp();
      first = true;
    }
    advance(m, u);
  }
}

// A(i, j) -= sum_{q < nbp} V(i,q) W(j,q) + W(i,q) V(j,q) for s0 <= j <= i < n, with
// V(i, q) = P[(p0+q)*ld + i] and W(i, q) = W[q*n + i], on the FP64 tensor cores:
// A -= Y X^T with Y = [V | W] (rows i) and X = [W | V] (rows j), K = 2NB. A warp owns a
// 32 x 32 tile (rows i, columns j) as 4 x 4 DMMA 8x8x4 accumulators whose rows run along
// the contiguous direction of P, so every load and store of the tile and of the operands
// is 8 consecutive doubles per quarter-warp. The row operands Y of a tile row stay in
// registers while the warp walks the columns. The tiles of the trailing lower triangle,
// in tile-row order, are split evenly between the warps.
NRG_DEV void panel_update(double* __restrict__ P, const double* __restrict__ W, int n, int ld, int p0, int nbp,
                          int s0, int gwarp, int gnwarps) {
  const int lane = threadIdx.x & 31;
  const int r = lane >> 2, c4 = lane & 3;
  const int T0 = s0 >> 5, Tn = (n - 1) >> 5;
  const int nt = Tn - T0 + 1;
  const long long S = (long long)nt * (nt + 1) / 2;
  const long long f0 = S * gwarp / gnwarps, f1 = S * (gwarp + 1) / gnwarps;
  if (f0 >= f1) return;
  int I = T0;
  long long acc0 = 0;
  while (acc0 + (I - T0 + 1) <= f0) {
    acc0 += I - T0 + 1;
    I++;
  }
  int J = T0 + (int)(f0 - acc0);
  double ya[4][2 * NB / 4];  // A fragments of Y for the current tile row
  int rowI = -1;
  for (long long f = f0; f < f1; f++) {
    const int i0 = I << 5, j0 = J << 5;
    if (rowI != I) {
      rowI = I;
#pragma unroll
      for (int ks = 0; ks < 2 * NB / 4; ks++) {
        const int q = 4 * ks + c4;
        const bool first = q < NB;
        const int qq = first ? q : q - NB;
        const double* row = first ? P + (size_t)(p0 + qq) * ld : W + (size_t)qq * n;
#pragma unroll
        for (int mi = 0; mi < 4; mi++) {
          const int ii = i0 + 8 * mi + r;
          ya[mi][ks] = (qq < nbp && ii < n) ? -row[ii] : 0.0;
        }
      }
    }
    double acc[4][4][2];
#pragma unroll
    for (int mi = 0; mi < 4; mi++)
#pragma unroll
      for (int ni = 0; ni < 4; ni++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int ii = i0 + 8 * mi + r, jj = j0 + 8 * ni + 2 * c4 + h;
          const bool ok = jj >= s0 && ii < n && ii >= jj;
          acc[mi][ni][h] = ok ? P[(size_t)jj * ld + ii] : 0.0;
        }
#pragma unroll
    for (int ks = 0; ks < 2 * NB / 4; ks++) {
      const int q = 4 * ks + c4;
      const bool first = q < NB;
      const int qq = first ? q : q - NB;
      const double* row = first ? W + (size_t)qq * n : P + (size_t)(p0 + qq) * ld;
      double b[4];
#pragma unroll
      for (int ni = 0; ni < 4; ni++) {
        const int jj = j0 + 8 * ni + r;
        b[ni] = (qq < nbp && jj < n) ? row[jj] : 0.0;
      }
#pragma unroll
      for (int mi = 0; mi < 4; mi++)
#pragma unroll
        for (int ni = 0; ni < 4; ni++) dmma884(acc[mi][ni][0], acc[mi][ni][1], ya[mi][ks], b[ni]);
    }
#pragma unroll
    for (int mi = 0; mi < 4; mi++)
#pragma unroll
      for (int ni = 0; ni < 4; ni++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int ii = i0 + 8 * mi + r, jj = j0 + 8 * ni + 2 * c4 + h;
          if (jj >= s0 && ii < n && ii >= jj) P[(size_t)jj * ld + ii] = acc[mi][ni][h];
        }
    if (J < I) {
      J++;
    } else {
      I++;
      J = T0;
    }
  }
}

// Packs the upper triangle of the row-major input (the lower triangle in column terms)
// into W1 with leading dimension ldp: W1[j*ldp + i] = H[j*n + i] for i >= j, zero for i < j
// and in the padding rows n <= i < ldp. Grid (row chunks of 8, blocks).
__global__ void __launch_bounds__(256) pack_lower_kernel(const LargeBlock* __restrict__ blocks) {
  const LargeBlock B = blocks[blockIdx.y];
  const int n = B.n, ld = B.ldp;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j = blockIdx.x * 8 + warp;
  if (j >= n) return;
  const double* src = B.H + (size_t)j * n;
  double* dst = B.W1 + (size_t)j * ld;
  for (int i = lane; i < ld; i += 32) dst[i] = (i >= j && i < n) ? src[i] : 0.0;
}

// One CTA per block: blocked (NB) Householder reduction of the packed lower triangle in W1
// (leading dimension ldp) to tridiagonal form; d, e, tau out; Householder vector k is left
// in column k (W1[k*ldp + k+1 ..], with a unit at k+1).
// Two CTAs per SM (255 registers, three slabs in flight per warp; three CTAs at 168 registers and two
// slabs took 9% longer). ny: copies of y.
// Many blocks are bound by HBM: 4/3 n^3 bytes of the triangle and a third more for the panel's vectors and
// updates, about 5.5 TB/s over 1400 blocks of order 601-900: 189 ms, from 241 with slabs of aligned
// rows, sums across lanes in every slab and three passes over V and W; 900 of order 380-420 (in L2) 24 ms,
// from 66.
// What bounds it is the chain of a column: its product, then sums that need the whole of a vector. The
// reflector stays unscaled in v (u = v / scale, u(k+1) = u1), so that the product starts right after its
// norm; the sums with the panel's V and W run while the product's first slabs are under way, one warp
// per vector; and one pass over V and W gives both t = tau (A v - V (W^T v) - W (V^T v)) and the next
// column without the terms in t, which follow once K = tau/2 t^T v is known: c -= v w(k+1) + w.
__global__ void __launch_bounds__(kTriThreads, 2) tridiag_kernel(const LargeBlock* __restrict__ blocks,
                                                                 const CUtensorMap* __restrict__ tmaps, int ny) {
  extern __shared__ __align__(16) double sm[];
  __shared__ __align__(8) uint64_t bars[kTriWarps * kTriStages];
  __shared__ double t1;  // t(k+1)
  const LargeBlock B = blocks[blockIdx.x];
  const int n = B.n, ld = B.ldp, tid = threadIdx.x, nt = kTriThreads, vp = tri_pad(n);
  const int lane = tid & 31, warp = tid >> 5;
  double* A = B.W1;
  double* W = B.W2;
  const uint64_t keep = l2_evict_last_policy(), once = l2_evict_first_policy();
  // TMA destinations: 1024-byte aligned ring of kTriStages slabs per warp
  double* ring = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(sm) + 1023) & ~(uintptr_t)1023);
  double* v = ring + kTriWarps * kTriStages * kSlabD;      // vp
  double* y = v + vp;                                  // ny x vp, ny >= 2
  double4* coef = reinterpret_cast<double4*>(y + (size_t)ny * vp);  // NB: W^T u, V^T u, row k+1 of W and V
  double* red = reinterpret_cast<double*>(coef + NB);  // 64 (two halves for block_sum_mma)
  double* vb = y + vp;  // the next column, in the second copy of y between two products
  int phase = 0;
  unsigned parity = 0;
  if (lane == 0) {
    for (int st = 0; st < kTriStages; st++) mbar_init(bars + warp * kTriStages + st, 1);
    fence_mbar_init();
    tmap_acquire(tmaps + blockIdx.x);  // lane 0 issues this warp's bulk copies
  }
  for (int i = tid; i < vp; i += nt) {
    v[i] = 0.0;
    for (int c = 0; c < ny; c++) y[(size_t)c * vp + i] = 0.0;
  }
  __syncthreads();

  for (int p0 = 0; p0 < n - 2; p0 += NB) {
    const int pe = min(p0 + NB, n - 2);
    double ps = 0.0;
    for (int i = p0 + tid; i < n; i += nt) {
      const double a = A[(size_t)p0 * ld + i];
      v[i] = a;
      if (i >= p0 + 2) ps = fma(a, a, ps);
    }
    if (tid < 4 * NB) reinterpret_cast<double*>(coef)[tid] = 0.0;
    double sigma = block_sum_mma(ps, red, phase);  // its barrier also publishes v
    for (int k = p0; k < pe; k++) {
      const int j = k - p0;
      // (1) Householder reflector for rows k+1..n-1 (dlarfg convention, v[k+1] = 1)
      double alpha = v[k + 1], unit = 1.0;
      if (tiny_column(alpha, sigma)) {  // the same in every thread
        alpha *= kTinyUp;
        ps = 0.0;
        for (int i = k + 2 + tid; i < n; i += nt) {
          v[i] *= kTinyUp;
          ps = fma(v[i], v[i], ps);
        }
        sigma = tiny_squares(block_sum_mma(ps, red, phase));
        unit = 1.0 / kTinyUp;
      }
      double tau = 0.0, beta = alpha, scale = 1.0, u1 = 1.0;
      if (sigma > 0.0) {
        beta = -copysign(sqrt(alpha * alpha + sigma), alpha);
        u1 = alpha - beta;
        tau = (beta - alpha) / beta;
        scale = 1.0 / u1;
      }
      if (tid == 0) {
        B.d[k] = v[k];
        B.e[k] = beta * unit;
        B.tau[k] = tau;
      }
      // (2) W^T u and V^T u, four vectors q = warp + 4 c of each per warp; row k+1 of W and V
      auto dots = [&](auto nq) {
        constexpr int Q = decltype(nq)::value;
        double x[8] = {};
        const double *pw[Q], *pv[Q];
#pragma unroll
        for (int c = 0; c < Q; c++) {
          const int q = min(warp + 4 * c, j - 1);
          pw[c] = W + (size_t)q * n;
          pv[c] = A + (size_t)(p0 + q) * ld;
        }
        for (int i = k + 1 + lane; i < n; i += 64) {
          const int i2 = min(i + 32, n - 1);
          double a[Q], b[Q], a2[Q], b2[Q];
#pragma unroll
          for (int c = 0; c < Q; c++) {
            a[c] = ld_keep(pw[c] + i, keep);
            b[c] = ld_keep(pv[c] + i, keep);
            a2[c] = ld_keep(pw[c] + i2, keep);
            b2[c] = ld_keep(pv[c] + i2, keep);
          }
          const double ui = i == k + 1 ? u1 : v[i], ui2 = i + 32 < n ? v[i2] : 0.0;
#pragma unroll
          for (int c = 0; c < Q; c++) {
            x[c] = fma(a[c], ui, fma(a2[c], ui2, x[c]));
            x[4 + c] = fma(b[c], ui, fma(b2[c], ui2, x[4 + c]));
          }
        }
        const double s = colsum8_mma(x, lane);
        const int q = warp + 4 * ((lane >> 2) & 3);
        double* cq = reinterpret_cast<double*>(coef + q);
        if ((lane & 3) == 0 && q < j) cq[lane >> 4] = s;
        if ((lane & 3) == 1 && q < j) cq[2 + (lane >> 4)] = lane < 16 ? W[(size_t)q * n + k + 1] : A[(size_t)(p0 + q) * ld + k + 1];
      };
      auto between = [&] {
        if (j > 12) dots(std::integral_constant<int, 4>{});
        else if (j > 8) dots(std::integral_constant<int, 3>{});
        else if (j > 4) dots(std::integral_constant<int, 2>{});
        else if (j > 0) dots(std::integral_constant<int, 1>{});
      };
      // (3) y = A u, A as it was at the panel's start
      if (tau != 0.0)
        symv_lower(tmaps + blockIdx.x, n, k + 1, v, u1, y, ny, vp, ring, bars, parity, B.info, once, between);
      else
        between();
      __syncthreads();
      // (4) t, the part of K, the next column but for its terms in t; the reflector scaled
      const double f = tau * scale;
      const bool next = k + 1 < pe;
      double pp = 0.0;
      for (int i0 = k + 1 + tid; i0 < n; i0 += 4 * nt) {
        int ii[4];
        double t[4], b[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
          ii[r] = min(i0 + r * nt, n - 1);
          b[r] = next ? A[(size_t)(k + 1) * ld + ii[r]] : 0.0;
          t[r] = y[ii[r]] + vb[ii[r]];
        }
        for (int c = 2; c < ny; c++)
#pragma unroll
          for (int r = 0; r < 4; r++) t[r] += y[(size_t)c * vp + ii[r]];
        for (int q = 0; q < j; q += 4) {  // coefficients beyond j are zero
          double a[4][4], w[4][4];
#pragma unroll
          for (int h = 0; h < 4; h++) {
            const int qq = min(q + h, j - 1);
#pragma unroll
            for (int r = 0; r < 4; r++) {
              a[h][r] = ld_keep(A + (size_t)(p0 + qq) * ld + ii[r], keep);
              w[h][r] = ld_keep(W + (size_t)qq * n + ii[r], keep);
            }
          }
#pragma unroll
          for (int h = 0; h < 4; h++) {
            const double4 cf = coef[q + h];
#pragma unroll
            for (int r = 0; r < 4; r++) {
              t[r] = fma(-a[h][r], cf.x, fma(-w[h][r], cf.y, t[r]));
              b[r] = fma(-a[h][r], cf.z, fma(-w[h][r], cf.w, b[r]));
            }
          }
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
          if (i0 + r * nt < n) {
            const int i = ii[r];
            const double vi = i == k + 1 ? 1.0 : scale * v[i], ti = f * t[r];
            pp = fma(ti, vi, pp);
            v[i] = vi;
            y[i] = ti;
            vb[i] = b[r];
            if (i == k + 1) t1 = ti;
            st_keep(A + (size_t)k * ld + i, vi, keep);
          }
      }
      // column k of W1 now holds v_k below the diagonal; clear its entries above, inside
      // the back-transform panel, so that the panel's V block is exactly unit lower trapezoidal
      for (int i = (k / NBT) * NBT + 1 + tid; i <= k; i += nt) A[(size_t)k * ld + i] = 0.0;
      const double Kc = 0.5 * tau * block_sum_mma(pp, red, phase);  // its barrier also publishes t1
      // (5) w, the next column and its norm
      const double w1 = t1 - Kc;
      ps = 0.0;
      for (int i = k + 1 + tid; i < n; i += nt) {
        const double vi = v[i], wi = y[i] - Kc * vi, ci = vb[i] - vi * w1 - wi;
        st_keep(W + (size_t)j * n + i, wi, keep);
        v[i] = ci;
        for (int c = 0; c < ny; c++) y[(size_t)c * vp + i] = 0.0;
        if (i >= k + 3) ps = fma(ci, ci, ps);
      }
      if (next) sigma = block_sum_mma(ps, red, phase);  // its barrier also publishes v, w and y
    }
    __syncthreads();
    panel_update(A, W, n, ld, p0, pe - p0, pe, warp, kTriWarps);
    fence_proxy_async_global();  // the next symv reads the updated trailing block by bulk copies
    __syncthreads();
  }
  if (tid == 0) {
    B.d[n - 2] = A[(size_t)(n - 2) * ld + n - 2];
    B.e[n - 2] = A[(size_t)(n - 2) * ld + n - 1];
    B.d[n - 1] = A[(size_t)(n - 1) * ld + n - 1];
    B.e[n - 1] = 0.0;
    B.tau[n - 2] = 0.0;
    B.tau[n - 1] = 0.0;
  }
  __syncthreads();
  int bad = 0;
  for (int i = tid; i < n; i += nt) bad |= !(isfinite(B.d[i]) && isfinite(B.e[i]));
  if (__syncthreads_or(bad) && tid == 0) atomicMin(B.info, -2);
}

// ---------------------------------------------------------------- mid-size tridiagonalisation
// Blocks with small_max_n < n <= mid_max_n (nrg_tuning): the whole lower triangle fits in shared memory,
// packed by columns (column j holds rows j..n-1 at pcol(j)), so the unblocked Householder
// reduction runs without touching HBM or L2 after the first read of H. Output as
// tridiag_kernel: d, e, tau, and v_k in row k of W1 (unit at k+1, zeros from the start of
// its back-transform panel up to k).
constexpr int kMidThreads = 512;

NRG_DEV int pcol(int j, int n) { return j * n - (j * (j - 1)) / 2; }

__global__ void __launch_bounds__(kMidThreads) tridiag_smem_kernel(const LargeBlock* __restrict__ blocks) {
  extern __shared__ __align__(16) double sm[];
  const LargeBlock B = blocks[blockIdx.x];
  const int n = B.n, ld = B.ldp, tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
  const int tot = n * (n + 1) / 2;
  double* P = sm;
  double* v = P + tot;
  double* w = v + n;
  double* red = w + n;  // 64 (two halves for block_sum_1b)
  int phase = 0;
  // column j of the lower triangle is row j of H from the diagonal on (row-major upper)
  for (int j = warp; j < n; j += nwarps) {
    const double* src = B.H + (size_t)j * n;
    double* dst = P + pcol(j, n) - j;
    for (int i = j + lane; i < n; i += 32) dst[i] = src[i];
  }
  __syncthreads();
  double* A = B.W1;
  for (int k = 0; k < n - 2; k++) {
    const int ck = pcol(k, n) - k;  // P[ck + i] = A(i, k), i >= k
    double ps = 0.0;
    for (int i = k + 2 + tid; i < n; i += nt) {
      const double x = P[ck + i];
      ps = fma(x, x, ps);
    }
    double sigma = block_sum_1b(ps, red, phase), alpha = P[ck + k + 1], up = 1.0;
    if (tiny_column(alpha, sigma)) {  // the same in every thread
      up = kTinyUp;
      alpha *= up;
      ps = 0.0;
      for (int i = k + 2 + tid; i < n; i += nt) ps = fma(up * P[ck + i], up * P[ck + i], ps);
      sigma = tiny_squares(block_sum_1b(ps, red, phase));
    }
    double tau = 0.0, beta = alpha, scale = 1.0;
    if (sigma > 0.0) {
      beta = -copysign(sqrt(alpha * alpha + sigma), alpha);
      tau = (beta - alpha) / beta;
      scale = up / (alpha - beta);
    }
    for (int i = k + 1 + tid; i < n; i += nt) {
      const double vi = (i == k + 1) ? 1.0 : P[ck + i] * scale;
      v[i] = vi;
      A[(size_t)k * ld + i] = vi;
    }
    const int kb0 = (k / NBT) * NBT;
    for (int i = kb0 + 1 + tid; i <= k; i += nt) A[(size_t)k * ld + i] = 0.0;
    if (tid == 0) {
      B.d[k] = P[ck + k];
      B.e[k] = beta / up;
      B.tau[k] = tau;
    }
    __syncthreads();
    if (sigma == 0.0) continue;  // uniform; with a sigma that is not a number the update has to spread it
    // w = tau * A22 v over rows/columns k+1..n-1; thread i reads row i left of the
    // diagonal and column i from the diagonal down: n-k-1 entries for every i
    for (int i = k + 1 + tid; i < n; i += nt) {
      double s0 = 0.0, s1 = 0.0;
      int addr = pcol(k + 1, n) + (i - (k + 1));  // A(i, k+1)
      for (int c = k + 1; c < i; c++) {
        s0 = fma(P[addr], v[c], s0);
        addr += n - c - 1;
      }
      const int ci = pcol(i, n) - i;
      for (int r = i; r < n; r++) s1 = fma(P[ci + r], v[r], s1);
      w[i] = tau * (s0 + s1);
    }
    __syncthreads();
    double pp = 0.0;
    for (int i = k + 1 + tid; i < n; i += nt) pp = fma(w[i], v[i], pp);
    const double Kc = 0.5 * tau * block_sum_1b(pp, red, phase);
    for (int i = k + 1 + tid; i < n; i += nt) w[i] -= Kc * v[i];
    __syncthreads();
    // rank-2 update of the trailing triangle, contiguous from pcol(k+1) to the end
    {
      int j = k + 1, off = tid;
      while (j < n && off >= n - j) {
        off -= n - j;
        j++;
      }
      int p = pcol(k + 1, n) + tid;
      while (j < n) {
        const int i = j + off;
        P[p] -= v[i] * w[j] + w[i] * v[j];
        p += nt;
        off += nt;
        while (j < n && off >= n - j) {
          off -= n - j;
          j++;
        }
      }
    }
    __syncthreads();
  }
  if (tid == 0) {
    const int c2 = pcol(n - 2, n);
    B.d[n - 2] = P[c2];
    B.e[n - 2] = P[c2 + 1];
    B.d[n - 1] = P[pcol(n - 1, n)];
    B.e[n - 1] = 0.0;
    B.tau[n - 2] = 0.0;
    B.tau[n - 1] = 0.0;
  }
  __syncthreads();
  int bad = 0;
  for (int i = tid; i < n; i += nt) bad |= !(isfinite(B.d[i]) && isfinite(B.e[i]));
  if (__syncthreads_or(bad) && tid == 0) atomicMin(B.info, -2);
}

// ---------------------------------------------------------------- tridiagonalisation in shared memory
// Blocks with small_max_n < n <= cluster_max_n (nrg_tuning): the full symmetric matrix is spread
// by columns over the shared memory of a cluster of C CTAs (column j lives in CTA j mod C; C = 1
// for the smallest), and the unblocked Householder reduction runs there. It is bound by the
// chain of n columns, so a column costs one exchange between the CTAs:
//   each CTA holds the previous reflector v, its w and the whole column k, and builds the new
//   reflector itself (the same arithmetic in every CTA, so all agree to the last bit);
//   it applies the previous rank-2 update to its columns and in the same pass forms their
//   products with the new reflector -- with both triangles stored a column's product is complete
//   in its CTA, so no partial sums cross the cluster, at 1.5 times the arithmetic of one triangle;
//   for each of its columns it sends the product and the element of row k+1 (the next column,
//   by symmetry) to every CTA by st.async, and waits on its own mbarrier for these pairs.
// Pair buffers alternate between consecutive columns: a CTA can send pairs of column k+2 only
// after it received all of column k+1's, which each other CTA sends after reading column k's. For this
// every CTA has to send something: in the last C columns those that own none of the rest send an empty
// pair to a slot that nobody reads any more.
// The reflector is kept unscaled (u = v / scale, so that the product does not wait for the
// scaling). The rows of a column are summed in the same order whatever C is.
// Pairs are stored by their sender, so that a warp's stores go to consecutive slots of one CTA at a time
// (to 32 slots C apart in as many CTAs they cost a further 0.25 us per column).
// Measured on B200 (one block, us per column): n = 456 in 16 CTAs 2.2 (5.4 with two cluster barriers
// per column over one triangle), n = 300 1.8 in 16, n = 224 1.55 and n = 128 1.4; with the stores apart
// n = 300 2.3 in 8, n = 224 1.6 in 16, 1.9 in 8, 2.5 in 4, 3.7 in 2, n = 128 1.5 in 16, 1.8 in 4, 3.1
// in 1. 256 threads are 8% faster than 512. At n = 456 the products take 1900 cycles of a column, the
// two sums 740, the reflector 250, the exchange the rest.
// Output as tridiag_kernel: d, e, tau, and v_k in row k of W1 (unit at k+1, zeros from the start
// of its back-transform panel up to k).
constexpr int kDsmThreads = 256;
constexpr int kDsmWarps = kDsmThreads / 32;
constexpr int kDsmMaxN = 640;                        // the largest cluster_max_n; 16 CTAs hold orders up to 624
constexpr int kDsmRows = (kDsmMaxN + kDsmThreads - 1) / kDsmThreads;  // rows of the vectors per thread
constexpr int kRowSplit = 4, kColSplit = kDsmWarps / kRowSplit;

__host__ __device__ inline int dsm_cols(int n, int C) { return (n + C - 1) / C; }

// Pairs of a CTA's columns in a pair buffer, odd: neighbouring rows of it lie on different banks.
__host__ __device__ inline int dsm_slot(int n, int C) { return dsm_cols(n, C) | 1; }

// Doubles of shared memory of one CTA of a C-cluster for a block of order n: pairs (2 buffers), v,
// w, u, partial products, row k+1, reduction scratch, columns.
__host__ __device__ inline size_t dsm_smem_doubles(int n, int C) {
  const size_t T = dsm_cols(n, C), Tp = (T + 7) / 8 * 8;
  return 4 * (size_t)C * dsm_slot(n, C) + 3 * (size_t)n + (kRowSplit + 1) * Tp + 64 + T * n;
}

inline bool dsm_fits(int n, int C) {
  return n <= kDsmMaxN && sizeof(double) * dsm_smem_doubles(n, C) + 512 <= 232448;
}

// Pairs that each CTA receives after column k: one for each of the n-k-1 columns left, whose owners are
// min(C, n-k-1) of the CTAs, and an empty one from each other CTA.
__host__ __device__ inline int dsm_pairs(int n, int C, int k) { return n - k - 1 > C ? n - k - 1 : C; }

NRG_DEV unsigned cluster_addr(unsigned smem_addr, unsigned rank) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  return a;
}

// Stores the pair (x, y) to shared memory of a CTA of the cluster and counts 16 bytes on that
// CTA's mbarrier.
NRG_DEV void st_async_pair(unsigned addr, double x, double y, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "l"(__double_as_longlong(x)), "l"(__double_as_longlong(y)), "r"(bar)
               : "memory");
}

// mbar_wait with acquire at cluster scope (the data come from other CTAs).
NRG_DEV bool mbar_wait_cluster(uint64_t* bar, unsigned parity, int bound = (1 << 22)) {
  const unsigned a = smem_u32(bar);
  for (int it = 0; it < bound; it++) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, "
        "p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

template <int C>
__global__ void __launch_bounds__(kDsmThreads, 1) tridiag_dsm_kernel(const LargeBlock* __restrict__ blocks) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) double sm[];
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ double sc[4];  // tau and scale of a reflector, by the parity of the next column
  const int r = blockIdx.x % C;  // rank in the cluster
  const LargeBlock B = blocks[blockIdx.x / C];
  const int n = B.n, ld = B.ldp, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int T = (n - r + C - 1) / C, Tp = (dsm_cols(n, C) + 7) / 8 * 8, Tm = dsm_slot(n, C);  // owned columns
  double2* buf = reinterpret_cast<double2*>(sm);  // 2 x C x Tm pairs (product, column element), by sender
  auto slot = [Tm](int i) { return (i % C) * Tm + i / C; };
  double* v = sm + 4 * C * Tm;                    // previous reflector
  double* w = v + n;                              // and its w
  double* u = w + n;                              // new reflector, unscaled, before the shift of u[k+1]
  double* part = u + n;                           // kRowSplit x Tp
  double* rowk = part + kRowSplit * Tp;           // Tp: row k+1 of the owned columns
  double* red = rowk + Tp;                        // 64
  double* M = red + 64;                           // T columns of n
  double* A = B.W1;
  int phase = 0;
  bool dead = false;  // a wait ran out: the block is flagged and nothing is waited for any more

  for (int t = warp; t < T; t += kDsmWarps) {  // column j: row j of H from the diagonal, column j above it
    const int j = r + t * C;
    double* dst = M + (size_t)t * n;
    for (int i = j + lane; i < n; i += 32) dst[i] = B.H[(size_t)j * n + i];
  }
  for (int i = warp; i < n; i += kDsmWarps)
    for (int t = lane; t < T; t += 32)
      if (r + t * C > i) M[(size_t)t * n + i] = B.H[(size_t)i * n + r + t * C];
  for (int i = tid; i < n; i += kDsmThreads) {
    buf[slot(i)] = make_double2(0.0, B.H[i]);
    v[i] = w[i] = 0.0;
  }
  if (tid == 0) {
    sc[0] = 0.0;
    sc[1] = 1.0;
  }
  if constexpr (C > 1) {
    if (tid == 0) {
      mbar_init(bars, 1);
      mbar_init(bars + 1, 1);
      fence_mbar_init();
    }
    cg::this_cluster().sync();
  } else {
    __syncthreads();
  }

  double ur[kDsmRows] = {};             // u of this thread's rows (of the previous column)
  double ek = 0.0;                      // e of the previous column
  for (int k = 0; k < n - 1; k++) {
    const double2* pb = buf + (k & 1) * C * Tm;
    const double tau = sc[2 * (k & 1)], scale = sc[2 * (k & 1) + 1], f = tau * scale;
    double vr[kDsmRows];
#pragma unroll
    for (int q = 0; q < kDsmRows; q++) {
      const int i = tid + q * kDsmThreads;
      vr[q] = 0.0;
      if (k > 0 && i >= k && i < n) {
        vr[q] = i == k ? 1.0 : scale * ur[q];
        if (C == 1 || (i >> 5) % C == r) A[(size_t)(k - 1) * ld + i] = vr[q];
      }
    }
    if (k > 0) {
      if (r == k % C)
        for (int i = ((k - 1) / NBT) * NBT + 1 + tid; i < k; i += kDsmThreads) A[(size_t)(k - 1) * ld + i] = 0.0;
      if (tid == 0 && r == 0) {
        B.e[k - 1] = ek;
        B.tau[k - 1] = tau;
      }
    }
    if constexpr (C > 1) {
      if (k > 0 && !dead && !mbar_wait_cluster(bars + (k & 1), ((k - 1) >> 1) & 1)) {
        dead = true;
        if (tid == 0) atomicExch(B.info, -5);
      }
    }
    // (1) previous reflector: w = f y - K v with f = tau scale
    double y[kDsmRows], cc[kDsmRows], pd = 0.0;
#pragma unroll
    for (int q = 0; q < kDsmRows; q++) {
      const int i = tid + q * kDsmThreads;
      y[q] = cc[q] = 0.0;
      if (i >= k && i < n) {
        const double2 p = pb[slot(i)];
        y[q] = f * p.x;
        cc[q] = p.y;
        pd = fma(y[q], vr[q], pd);
      }
    }
    const double yk = f * pb[slot(k)].x;
    const double Kc = 0.5 * tau * block_sum_mma(pd, red, phase);
    // (2) column k after that update; reflector for rows k+1..n-1 (dlarfg convention)
    const double wk = k > 0 ? yk - Kc : 0.0;
    double ps = 0.0;
#pragma unroll
    for (int q = 0; q < kDsmRows; q++) {
      const int i = tid + q * kDsmThreads;
      if (i >= k && i < n) {
        const double wi = y[q] - Kc * vr[q];
        const double ai = k > 0 ? cc[q] - vr[q] * wk - wi : cc[q];
        v[i] = vr[q];
        w[i] = wi;
        u[i] = ai;
        ur[q] = ai;
        if (i >= k + 2) ps = fma(ai, ai, ps);
      }
    }
    double sigma = block_sum_mma(ps, red, phase);  // its barrier also publishes v, w and u
    double alpha = u[k + 1], unit = 1.0;
    if (tid == 0 && r == 0) B.d[k] = u[k];
    if (k == n - 2) {
      if (tid == 0 && r == 0) {
        B.e[k] = alpha;
        B.tau[k] = 0.0;
      }
      if (tid == 0 && r == (n - 1) % C) {
        B.d[n - 1] = M[(size_t)((n - 1) / C) * n + n - 1] - 2.0 * v[n - 1] * w[n - 1];
        B.e[n - 1] = 0.0;
        B.tau[n - 1] = 0.0;
      }
      break;
    }
    if (tiny_column(alpha, sigma)) {  // the same in every thread of the cluster
      alpha *= kTinyUp;
      ps = 0.0;
#pragma unroll
      for (int q = 0; q < kDsmRows; q++) {
        const int i = tid + q * kDsmThreads;
        if (i >= k + 2 && i < n) {  // u[k+1] may still be read for alpha
          ur[q] *= kTinyUp;
          u[i] = ur[q];
          ps = fma(ur[q], ur[q], ps);
        }
      }
      sigma = tiny_squares(block_sum_mma(ps, red, phase));
      unit = 1.0 / kTinyUp;
    }
    const double beta = sigma > 0.0 ? -copysign(sqrt(alpha * alpha + sigma), alpha) : alpha;
    const double u1 = alpha - beta;  // u[k+1]
    ek = beta * unit;
#pragma unroll
    for (int q = 0; q < kDsmRows; q++)
      if (tid + q * kDsmThreads == k + 1) ur[q] = u1;
    // the two divisions of the reflector are needed for the next column only: the warp with the
    // least work makes them beside the products
    if (tid == kDsmThreads - 1) {
      double tau1 = 0.0, scale1 = 1.0;
      if (sigma > 0.0) {
        tau1 = (beta - alpha) / beta;
        scale1 = 1.0 / u1;
      }
      sc[2 * ((k + 1) & 1)] = tau1;
      sc[2 * ((k + 1) & 1) + 1] = scale1;
    }
    // (3) previous update of the owned columns j > k and their products with u
    const int t0 = (k + 1 - r > 0) ? (k + 1 - r + C - 1) / C : 0;
    const int wr = warp % kRowSplit, wc = warp / kRowSplit;
    const int s0 = (k + 1) >> 5, s1 = (n - 1) >> 5;
    for (int tg = t0 + 8 * wc; tg < T; tg += 8 * kColSplit) {
      const int nv = min(8, T - tg);
      double vj[8], wj[8], cs[8];
#pragma unroll
      for (int c = 0; c < 8; c++) {
        const int j = r + (tg + (c < nv ? c : 0)) * C;
        vj[c] = v[j];
        wj[c] = w[j];
        cs[c] = 0.0;
      }
      // row chunks s with s mod kRowSplit = wr, whatever k and C are; lanes above row k+1 or below
      // row n-1 and columns beyond the last read something finite and store nothing
      for (int s = s0 + ((wr - s0) & (kRowSplit - 1)); s <= s1; s += kRowSplit) {
        const int i = min(32 * s + lane, n - 1);
        const bool act = i > k && 32 * s + lane < n;
        const double vi = v[i], wi = w[i], ui = act ? (i == k + 1 ? u1 : u[i]) : 0.0;
        double* col = M + (size_t)tg * n + i;
        double x[8];
#pragma unroll
        for (int c = 0; c < 8; c++) x[c] = col[(size_t)(c < nv ? c : 0) * n];
#pragma unroll
        for (int c = 0; c < 8; c++) x[c] = fma(-vi, wj[c], x[c]);
#pragma unroll
        for (int c = 0; c < 8; c++) x[c] = fma(-wi, vj[c], x[c]);
#pragma unroll
        for (int c = 0; c < 8; c++) {
          cs[c] = fma(x[c], ui, cs[c]);
          if (act && c < nv) col[(size_t)c * n] = x[c];
        }
        if (act && i == k + 1) {
#pragma unroll
          for (int c = 0; c < 8; c++)
            if (c < nv) rowk[tg + c] = x[c];
        }
      }
      __syncwarp();
      const double sum = colsum8_mma(cs, lane);
      const int c = lane >> 2;
      if ((lane & 3) == 0 && c < nv) part[wr * Tp + tg + c] = sum;
    }
    __syncthreads();
    // (4) each owned column's product and element of row k+1 to every CTA
    double2* nb = buf + ((k + 1) & 1) * C * Tm;
    if constexpr (C > 1) {
      uint64_t* bar = bars + ((k + 1) & 1);
      if (tid == 0) mbar_expect_tx(bar, 16u * (unsigned)dsm_pairs(n, C, k));
      // a warp sends its columns' pairs to one CTA at a time, to consecutive slots there
      constexpr int kPer = C < kDsmWarps ? kDsmWarps / C : 1;  // warps per destination
      static_assert(kRowSplit == 4, "pairwise sum of the row parts");
      // (without a column left: an empty pair to the slot of its first one, which is reduced)
      const bool some = t0 < T;
      const int end = some ? T : 1;
      for (int t = (some ? t0 : 0) + lane + 32 * (warp / C); t < end; t += 32 * kPer) {
        const double yj = some ? (part[t] + part[Tp + t]) + (part[2 * Tp + t] + part[3 * Tp + t]) : 0.0;
        const double xj = some ? rowk[t] : 0.0;
#pragma unroll
        for (int dst = warp % C; dst < C; dst += kDsmWarps)
          st_async_pair(cluster_addr(smem_u32(nb + r * Tm + t), dst), yj, xj, cluster_addr(smem_u32(bar), dst));
      }
    } else {
      for (int t = t0 + tid; t < T; t += kDsmThreads)
        nb[t] = make_double2((part[t] + part[Tp + t]) + (part[2 * Tp + t] + part[3 * Tp + t]), rowk[t]);
      __syncthreads();
    }
  }
  if constexpr (C > 1) cg::this_cluster().sync();  // d and e are complete; no CTA leaves while pairs are under way
  else __syncthreads();
  if (r == 0) {
    int bad = 0;
    for (int i = tid; i < n; i += kDsmThreads) bad |= !(isfinite(B.d[i]) && isfinite(B.e[i]));
    if (__syncthreads_or(bad) && tid == 0) atomicMin(B.info, -2);
  }
}

// ---------------------------------------------------------------- large blocks, few of them
// The blocked reduction of one block by a group of G CTAs (one per SM, all of them resident: one
// cooperative launch for every group). What bounds it is the chain of n columns, two exchanges
// through L2 per column, and for the largest blocks the bytes of the trailing matrix per column.
//   The full symmetric matrix is kept (W1[j ld + i] = A(i, j)), twice the triangle's bytes: then
//   CTA r's columns j = r + t G give complete products A(:, j) v -- no partial vectors to add up over
//   the group -- by plain 16-byte loads with v in shared memory, and the CTA is the only one that
//   reads or updates its columns.
//   Per column k of a panel of kGNB every CTA has the whole column in shared memory and builds the
//   reflector v itself. It publishes its part of W^T v and V^T v, forms the products of its columns
//   (which cover that exchange), then its rows of t = tau (A v - V (W^T v) - W (V^T v)) and of the
//   next column without the terms in K = tau/2 t^T v and t(k+1), and publishes these beside its part
//   of K: the one exchange that is waited for. The next column is b + (2 K - t(k+1)) v, W = t - K v.
//   At the panel's end, after a barrier, each CTA updates its columns by V W^T + W V^T on the FP64
//   tensor cores.
// An exchanged number travels in 16 bytes with the column it belongs to, and its readers poll it: a
// barrier (fence, counter, poll, and the loads behind it) took 2 us, twice per column. Each buffer
// is written again only after its writer has received what every reader sends after reading it.
constexpr int kGridThreads = 512;
constexpr int kGridWarps = kGridThreads / 32;
constexpr int kGNB = 16;           // panel width
constexpr int kGridMaxT = 256;     // columns per CTA
constexpr int kGridSeg = 8;        // most row segments of a product
constexpr int kGridMaxG = 160;     // most CTAs of a group

struct GridGroup {
  int cta0, G;        // its CTAs
  int job0, njob;     // its blocks, one after another: jobs[job0 ..]
};


// Doubles of global scratch per block (pairs: number, tag): next column, parts of K, parts of the dot
// products, then t(k+1) and row k+1 of V and W.
__host__ __device__ inline size_t grid_scratch_doubles(int n) {
  return 2 * ((size_t)n + kGridMaxG + (size_t)kGridMaxG * 2 * kGNB + 2 * kGNB + 1);
}
__host__ __device__ inline size_t grid_smem_doubles(int ldp, int T) {
  return (size_t)ldp + 64 + (2 * kGNB + 2 + kGridSeg) * (size_t)T + 4 * kGNB + 64 + 32;
}

// Barrier over the group's CTAs: the counter reaches `target` when all have arrived. False if the
// bounded wait ran out (the block is flagged, and the caller stops waiting).
NRG_DEV bool group_barrier(unsigned* ctr, unsigned target, bool wait) {
  __syncthreads();
  int ok = 1;
  if (threadIdx.x == 0) {
    __threadfence();
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
    if (wait) {
      ok = 0;
      for (int it = 0; it < (1 << 24); it++) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
        if ((int)(v - target) >= 0) {
          ok = 1;
          break;
        }
      }
      __threadfence();
    }
  }
  return __syncthreads_and(threadIdx.x != 0 || ok) != 0;
}

// One 16-byte access each, so number and tag are always of the same store.
NRG_DEV void tag_store(double2* p, double x, unsigned tag) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p),
               "l"(__double_as_longlong(x)), "l"((long long)tag)
               : "memory");
}
NRG_DEV bool tag_load(const double2* p, unsigned tag, double& x) {
  long long a, b;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
               : "=l"(a), "=l"(b)
               : "l"(p)
               : "memory");
  x = __longlong_as_double(a);
  return b == (long long)tag;
}
// Bounded poll of one number; live turns false when the bound runs out (the caller flags the block and
// no later poll waits).
NRG_DEV double tag_wait(const double2* p, unsigned tag, bool& live) {
  double x = 0.0;
  bool ok = tag_load(p, tag, x);
  for (int it = 0; !ok && live; it++) {
    ok = tag_load(p, tag, x);
    if (it >= 1 << 24) live = false;
  }
  return x;
}

// Lower-triangle input (rows of H from the diagonal on) to the full symmetric W1, 32 x 32 tiles.
__global__ void __launch_bounds__(256) pack_full_kernel(const LargeBlock* __restrict__ blocks) {
  __shared__ double tile[32][33];
  const LargeBlock B = blocks[blockIdx.z];
  const int n = B.n, ld = B.ldp, i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;  // j0 <= i0: H(j, i), i >= j
  if (j0 == 0)  // no tag of an earlier reduction is left in the exchange buffers
    for (size_t q = blockIdx.x * 256 + threadIdx.x; q < grid_scratch_doubles(n); q += (size_t)gridDim.x * 256) B.gx[q] = 0.0;
  if (i0 >= ld || j0 >= n || j0 > i0) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int r = ty; r < 32; r += 8) {
    const int j = j0 + r, i = i0 + tx;
    tile[r][tx] = j < n && i < n && i >= j ? B.H[(size_t)j * n + i] : 0.0;
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int j = j0 + r, i = i0 + tx;  // column j, rows i: below the diagonal
    if (j < n) {
      const double x = i0 != j0 || tx >= r ? tile[r][tx] : tile[tx][r];
      B.W1[(size_t)j * ld + i] = x;
    }
    if (i0 != j0) {  // column i, rows j: above it
      const int jj = i0 + r, ii = j0 + tx;
      if (jj < n) B.W1[(size_t)jj * ld + ii] = tile[tx][r];
    }
  }
}

// Sum over the lanes of x[c] for c = (lane >> 3) & 3, in every lane.
NRG_DEV double colsum4(double (&x)[4], int lane) {
#pragma unroll
  for (int s = 2, o = 16; s >= 1; s >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int q = 0; q < s; q++) {
      const double send = up ? x[q] : x[q + s];
      const double keep = up ? x[q + s] : x[q];
      x[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
  return x[0];
}

// Products of a CTA's columns t0 .. T-1 with the vector vf: items of four columns x a segment of the rows
// (S of them, chunks of 64 rows from `base`), parts of the sums in yp.
__device__ __forceinline__ void grid_products(const double* A, int yp_off, int ld, int r, int G, int T, int Tm, int t0,
                                           int ng, int S, int base, int nch) {
  extern __shared__ __align__(16) double sm[];
  const double* vf = sm;
  double* yp = sm + yp_off;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int it = warp; it < ng * S; it += kGridWarps) {
    const int tg = t0 + 4 * (it / S), s = it % S, c0 = nch * s / S, c1 = nch * (s + 1) / S;
    const double* col[4];
#pragma unroll
    for (int c = 0; c < 4; c++) col[c] = A + (size_t)(r + (tg + c < T ? tg + c : tg) * G) * ld + base + 2 * lane;
    const double2* vp = reinterpret_cast<const double2*>(vf + base + 2 * lane);
    double sum[4] = {};
    const int cf = min(c1, (ld - base) / 64);  // a last chunk may have 32 rows only
    int ch = c0;
    for (; ch + 4 <= cf; ch += 4) {  // sixteen loads a lane before the first is used
      double2 x[4][4], v[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int c = 0; c < 4; c++) x[u][c] = __ldcg(reinterpret_cast<const double2*>(col[c] + 64 * (ch + u)));
#pragma unroll
      for (int u = 0; u < 4; u++) v[u] = vp[32 * (ch + u)];
#pragma unroll
      for (int u = 0; u < 4; u++)
#pragma unroll
        for (int c = 0; c < 4; c++) sum[c] = fma(x[u][c].x, v[u].x, fma(x[u][c].y, v[u].y, sum[c]));
    }
    for (; ch < cf; ch++) {
      const double2 v = vp[32 * ch];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const double2 x = __ldcg(reinterpret_cast<const double2*>(col[c] + 64 * ch));
        sum[c] = fma(x.x, v.x, fma(x.y, v.y, sum[c]));
      }
    }
    if (ch < c1 && lane < 16) {
      const double2 v = vp[32 * ch];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const double2 x = __ldcg(reinterpret_cast<const double2*>(col[c] + 64 * ch));
        sum[c] = fma(x.x, v.x, fma(x.y, v.y, sum[c]));
      }
    }
    __syncwarp();
    const double y = colsum4(sum, lane);
    const int c = lane >> 3;
    if ((lane & 7) == 0 && tg + c < T) yp[s * Tm + tg + c] = y;
  }
}

// A(i, j) -= V(i, :) W(j, :)^T + W(i, :) V(j, :)^T for a CTA's columns j = r + t G >= pe and the rows i >= pe.
__device__ __forceinline__ void grid_panel_update(double* A, const double* W, int vo_off, int n, int ld, int r, int G,
                                               int T, int Tm, int t0, int p0, int pe, int nbp) {
  extern __shared__ __align__(16) double sm[];
  const double* Vo = sm + vo_off;
  const double* Wo = Vo + kGNB * Tm;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fr = lane >> 2, fc = lane & 3;
  for (int i0 = (pe & ~31) + 32 * warp; i0 < n; i0 += 32 * kGridWarps) {
    double bf[2 * kGNB / 4][4];  // [V; W] rows q of the 32 rows i
#pragma unroll
    for (int ks = 0; ks < 2 * kGNB / 4; ks++) {
      const int q = 4 * ks + fc, qq = q < kGNB ? q : q - kGNB;
      const double* row = q < kGNB ? A + (size_t)(p0 + qq) * ld : W + (size_t)qq * n;
#pragma unroll
      for (int ni = 0; ni < 4; ni++) {
        const int i = i0 + 8 * ni + fr;
        bf[ks][ni] = qq < nbp && i >= pe && i < n ? __ldcg(row + i) : 0.0;
      }
    }
    for (int tg = t0; tg < T; tg += 8) {
      const int t = tg + fr;
      double* col = A + (size_t)(r + (t < T ? t : t0) * G) * ld + i0 + 2 * fc;
      double acc[4][2];
#pragma unroll
      for (int ni = 0; ni < 4; ni++) {
        const double2 x = __ldcg(reinterpret_cast<const double2*>(col + 8 * ni));
        acc[ni][0] = x.x;
        acc[ni][1] = x.y;
      }
#pragma unroll
      for (int ks = 0; ks < 2 * kGNB / 4; ks++) {
        const int q = 4 * ks + fc, qq = q < kGNB ? q : q - kGNB;
        const double a = t < T && qq < nbp ? -(q < kGNB ? Wo : Vo)[qq * Tm + t] : 0.0;
#pragma unroll
        for (int ni = 0; ni < 4; ni++) dmma884(acc[ni][0], acc[ni][1], a, bf[ks][ni]);
      }
      if (t < T) {
#pragma unroll
        for (int ni = 0; ni < 4; ni++)
          __stcg(reinterpret_cast<double2*>(col + 8 * ni), make_double2(acc[ni][0], acc[ni][1]));
      }
    }
  }
}

// ROWS: rows of a column per thread (8: orders up to 4096, 20: up to 10240).
template <int ROWS>
__global__ void __launch_bounds__(kGridThreads, 1) tridiag_grid_kernel(const LargeBlock* __restrict__ blocks,
                                                                       const GridGroup* __restrict__ groups, int ngroup,
                                                                       const int* __restrict__ jobs, unsigned* ctrs) {
  extern __shared__ __align__(16) double sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int g = 0;
  while (g + 1 < ngroup && groups[g + 1].cta0 <= (int)blockIdx.x) g++;
  const GridGroup gr = groups[g];
  const int G = gr.G, r = (int)blockIdx.x - gr.cta0;
  if (r >= G) return;
  unsigned* ctr = ctrs + 32 * g;
  unsigned epoch = 0;
  bool live = true;
  int phase = 0;
  for (int jb = 0; jb < gr.njob; jb++) {
    const LargeBlock B = blocks[jobs[gr.job0 + jb]];
    const int n = B.n, ld = B.ldp, T = (n - r + G - 1) / G, Tm = (n + G - 1) / G;
    double* A = B.W1;
    double* W = B.W2;
    double* vf = sm;                    // ld + 64: current reflector, zero outside k+1 .. n-1
    double* Vo = vf + ld + 64;          // kGNB x Tm: the panel's reflectors at this CTA's rows
    double* Wo = Vo + kGNB * Tm;
    double* to = Wo + kGNB * Tm;        // Tm: t
    double* co = to + Tm;               // Tm: elements of row k+1
    double* yp = co + Tm;               // kGridSeg x Tm
    double* cd = yp + kGridSeg * Tm;    // 2 kGNB: W^T v, V^T v
    double* k1 = cd + 2 * kGNB;         // 2 kGNB: row k+1 of V and W
    double* red = k1 + 2 * kGNB;        // 64
    double* sc = red + 64;              // t(k) of the previous reflector; parts of K by warp from 8 on
    double2* gb = reinterpret_cast<double2*>(B.gx);  // next column
    double2* gk = gb + n;                            // parts of K
    double2* gd = gk + kGridMaxG;                    // parts of the dot products
    double2* gy = gd + kGridMaxG * 2 * kGNB;         // t(k+1), row k+1 of V, of W
    // parts of K of reflector k, from every CTA (all threads call it; sum in every thread)
    auto sum_k = [&](int k) {
      if (warp <= (G - 1) >> 5) {
        const double s = warp_sum_mma(tid < G ? tag_wait(gk + tid, k + 1, live) : 0.0);
        if (lane == 0) sc[8 + warp] = s;
      }
    };
    auto k_of = [&]() {
      double s = 0.0;
      for (int q = 0; q <= (G - 1) >> 5; q++) s += sc[8 + q];
      return s;
    };
    auto publish_column = [&](int c) {  // column c of the updated matrix, by rows of this CTA's columns
      for (int t = tid; t < T; t += kGridThreads)
        if (r + t * G >= c) tag_store(gb + r + t * G, __ldcg(A + (size_t)(r + t * G) * ld + c), c + 1);
    };
    for (int i = tid; i < ld + 64; i += kGridThreads) vf[i] = 0.0;
    publish_column(0);
    int p0 = 0;
    double tau = 0.0, scale = 1.0;
    for (int k = 0; k < n - 2; k++) {
      const int j = k - p0;
      const int t0 = k + 1 - r > 0 ? (k + 1 - r + G - 1) / G : 0;  // its first column beyond k
      // (1) this column: b and K from the group; the previous column's W (own rows); its reflector
      double b[ROWS];
      unsigned pending = 0;  // every load goes out before the first is looked at
#pragma unroll
      for (int q = 0; q < ROWS; q++) {
        const int i = k + tid + q * kGridThreads;
        if (k + q * kGridThreads >= n) break;  // uniform
        b[q] = 0.0;
        if (i < n && !tag_load(gb + i, k + 1, b[q])) pending |= 1u << q;
      }
      while (pending && live) {
#pragma unroll
        for (int q = 0; q < ROWS; q++)
          if (pending >> q & 1) {
            b[q] = tag_wait(gb + k + tid + q * kGridThreads, k + 1, live);
            pending &= ~(1u << q);
          }
      }
      if (j > 0) {
        sum_k(k - 1);
        if (tid == kGridThreads - 1) sc[0] = tag_wait(gy, k, live);
      }
      __syncthreads();
      const double Kc = j > 0 ? k_of() : 0.0, vc = j > 0 ? 2.0 * Kc - sc[0] : 0.0, vs = vc * scale;
      double ps = 0.0;
#pragma unroll
      for (int q = 0; q < ROWS; q++) {
        const int i = k + tid + q * kGridThreads;
        if (k + q * kGridThreads >= n) break;  // uniform
        if (i < n) {
          // the previous reflector is 1 at k and scale u beyond
          const double a = i == k ? b[q] + vc : fma(vs, vf[i], b[q]);
          vf[i] = a;
          if (i >= k + 2) ps = fma(a, a, ps);
        }
      }
      double sigma = block_sum_mma(ps, red, phase), alpha = vf[k + 1], unit = 1.0;
      const double dk = vf[k];
      if (tiny_column(alpha, sigma)) {  // the same in every thread of the group
        alpha *= kTinyUp;
        ps = 0.0;
        for (int i = k + 2 + tid; i < n; i += kGridThreads) {
          vf[i] *= kTinyUp;
          ps = fma(vf[i], vf[i], ps);
        }
        sigma = tiny_squares(block_sum_mma(ps, red, phase));
        unit = 1.0 / kTinyUp;
      }
      const double beta = sigma > 0.0 ? -copysign(sqrt(alpha * alpha + sigma), alpha) : alpha;
      const double u1 = alpha - beta;
      if (j > 0)
        for (int t = tid; t < T; t += kGridThreads) {
          const int i = r + t * G;
          if (i >= k) {
            const double vi = Vo[(j - 1) * Tm + t], wi = to[t] - Kc * vi;
            Wo[(j - 1) * Tm + t] = wi;
            __stcg(A + (size_t)(k - 1) * ld + i, vi);
            __stcg(W + (size_t)(j - 1) * n + i, wi);
          }
        }
      __syncthreads();  // alpha is read, W is complete
      if (tid == 0) {
        vf[k] = 0.0;
        vf[k + 1] = u1;
      }
      if (r == k % G)  // zeros from the start of its back-transform panel down to the diagonal
        for (int i = (k / NBT) * NBT + 1 + tid; i <= k; i += kGridThreads) A[(size_t)k * ld + i] = 0.0;
      // elements of row k+1 of the own columns, for the next column; T <= kGridMaxT < kGridThreads
      const bool last = j == kGNB - 1 || k == n - 3;
      const double ck1 = !last && t0 + tid < T ? __ldcg(A + (size_t)(r + (t0 + tid) * G) * ld + k + 1) : 0.0;
      // the owner of row k+1 publishes its V and W
      if ((k + 1) % G == r && tid < 2 * j) {
        const int q = tid < j ? tid : tid - j;
        tag_store(gy + 1 + (tid < j ? q : kGNB + q), (tid < j ? Vo : Wo)[q * Tm + t0], k + 1);
      }
      __syncthreads();
      // parts of W^T u and V^T u over the own rows
      // (the first column of a panel has none, but the exchange has to take place: one dummy)
      const int nd = max(2 * j, 1);
      for (int q = warp; q < nd; q += kGridWarps) {
        const double* x = q < j ? Wo + q * Tm : Vo + (q - j) * Tm;
        double s = 0.0;
        if (j > 0)
          for (int t = t0 + lane; t < T; t += 32) s = fma(x[t], vf[r + t * G], s);
        s = warp_sum_mma(s);
        if (lane == 0) tag_store(gd + (size_t)(q < j || j == 0 ? q : kGNB + q - j) * kGridMaxG + r, s, k + 1);
      }
      // (2) products of the own columns with u: items of four columns x a segment of the rows
      const int ng = (T - t0 + 3) / 4, S = ng > 0 ? max(1, min(kGridSeg, kGridWarps / ng)) : 1;
      const int base = (k + 1) & ~63, nch = (n - base + 63) / 64;
      grid_products(A, (int)(yp - sm), ld, r, G, T, Tm, t0, ng, S, base, nch);
      // the reflector's divisions, beside the slower warps' products
      tau = 0.0;
      scale = 1.0;
      if (sigma > 0.0) {
        tau = (beta - alpha) / beta;
        scale = 1.0 / u1;
      }
      if (tid == 0 && r == 0) {
        B.d[k] = dk;
        B.e[k] = beta * unit;
        B.tau[k] = tau;
      }
      if (t0 + tid < T) co[t0 + tid] = ck1;
      // (3) the sums of the dot products, row k+1 of V and W; t and the next column at the own rows
      for (int q = warp; q < nd; q += kGridWarps) {
        const double2* row = gd + (size_t)(q < j || j == 0 ? q : kGNB + q - j) * kGridMaxG;
        constexpr int kL = (kGridMaxG + 31) / 32;
        double x[kL], s = 0.0;
        bool ok[kL];
#pragma unroll
        for (int c = 0; c < kL; c++) {
          x[c] = 0.0;
          ok[c] = lane + 32 * c >= G || tag_load(row + lane + 32 * c, k + 1, x[c]);
        }
#pragma unroll
        for (int c = 0; c < kL; c++) {
          if (!ok[c]) x[c] = tag_wait(row + lane + 32 * c, k + 1, live);
          s += x[c];
        }
        s = warp_sum_mma(s);
        if (lane == 0) cd[q < j || j == 0 ? q : kGNB + q - j] = scale * s;
      }
      if (tid < 2 * j) {
        const int q = tid < j ? tid : kGNB + tid - j;
        k1[q] = tag_wait(gy + 1 + q, k + 1, live);
      }
      __syncthreads();
      // lanes per row: the sums over the panel are chains
      const int left = T - t0, L = left <= kGridThreads / 8 ? 8 : left <= kGridThreads / 4 ? 4 : 2;
      const int tl = tid % L;
      double pk = 0.0;
      for (int u = tid / L; u < (left + 31) / 32 * 32; u += kGridThreads / L) {  // whole warps
        const bool in = u < left;
        const int t = t0 + (in ? u : 0), i = r + t * G;
        double y = 0.0, c = 0.0;
        if (in)
          for (int q = tl; q < j; q += L) {
            const double vq = Vo[q * Tm + t], wq = Wo[q * Tm + t];
            y = fma(vq, cd[q], fma(wq, cd[kGNB + q], y));
            c = fma(vq, k1[kGNB + q], fma(wq, k1[q], c));
          }
        for (int o = L >> 1; o > 0; o >>= 1) {
          y += __shfl_xor_sync(0xffffffffu, y, o);
          c += __shfl_xor_sync(0xffffffffu, c, o);
        }
        if (in && tl == 0) {
          double a = yp[t];
          for (int s = 1; s < S; s++) a += yp[s * Tm + t];
          y = tau * (scale * a - y);
          to[t] = y;
          const double vi = i == k + 1 ? 1.0 : scale * vf[i];
          Vo[j * Tm + t] = vi;
          pk = fma(y, vi, pk);
          if (!last) tag_store(gb + i, co[t] - c - y, k + 2);
          if (i == k + 1) tag_store(gy, y, k + 1);
        }
      }
      pk = block_sum_mma(pk, red, phase);
      if (tid == 0) tag_store(gk + r, 0.5 * tau * pk, k + 1);
      if (!last) continue;
      // (4) end of the panel: its last W, then the update of the own columns
      sum_k(k);
      __syncthreads();
      const double Kl = k_of();
      const int pe = k + 1, nbp = j + 1;
      for (int t = t0 + tid; t < T; t += kGridThreads) {
        const int i = r + t * G;
        const double vi = Vo[j * Tm + t], wi = to[t] - Kl * vi;
        Wo[j * Tm + t] = wi;
        __stcg(A + (size_t)k * ld + i, vi);
        __stcg(W + (size_t)j * n + i, wi);
      }
      epoch++;
      if (!group_barrier(ctr, epoch * (unsigned)G, live)) live = false;
      grid_panel_update(A, W, (int)(Vo - sm), n, ld, r, G, T, Tm, t0, p0, pe, nbp);
      __syncthreads();
      p0 = pe;
      if (k < n - 3) publish_column(pe);
    }
    if (!live) atomicExch(B.info, -5);  // a wait ran out (any thread's)
    // the last 2 x 2, by its columns' owners
    __syncthreads();
    if (tid == 0) {
      if (r == (n - 2) % G) {
        B.d[n - 2] = __ldcg(A + (size_t)(n - 2) * ld + n - 2);
        B.e[n - 2] = __ldcg(A + (size_t)(n - 2) * ld + n - 1);
        B.tau[n - 2] = 0.0;
      }
      if (r == (n - 1) % G) {
        B.d[n - 1] = __ldcg(A + (size_t)(n - 1) * ld + n - 1);
        B.e[n - 1] = 0.0;
        B.tau[n - 1] = 0.0;
      }
    }
    epoch++;
    if (!group_barrier(ctr, epoch * (unsigned)G, live)) live = false;
    if (r == 0) {
      int bad = 0;
      for (int i = tid; i < n; i += kGridThreads) bad |= !(isfinite(__ldcg(B.d + i)) && isfinite(__ldcg(B.e + i)));
      if (__syncthreads_or(bad) && tid == 0) atomicMin(B.info, -2);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- divide and conquer: leaves
// One CTA per leaf of order <= 64: the leaf is itself solved by divide and conquer in shared memory
// (smem_dc). Measured on B200: leaves of order 32 by implicit QL took 0.40 ms of a step of 40 blocks up to
// order 480, these 0.10 ms, with a merge level less to follow (0.1 ms).
constexpr int kLeafLd = kLeaf + 1;

__global__ void __launch_bounds__(kCtaEigThreads) dc_leaf_kernel(const LargeBlock* __restrict__ blocks,
                                                                 const DcLeaf* __restrict__ leaves) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int ctl[12];
  const DcLeaf L = leaves[blockIdx.x];
  const LargeBlock B = blocks[L.blk];
  const int n = B.n, a0 = L.a0, nl = L.a1 - L.a0, tid = threadIdx.x;
  double* Z = sm;
  double* U = Z + kLeaf * kLeafLd;
  double* d = U + kLeaf * kLeafLd;
  double* e = d + kLeaf;
  int bad = 0;
  if (tid < nl) {
    double di = B.d[a0 + tid];
    if (tid == 0 && a0 > 0) di -= fabs(B.e[a0 - 1]);             // rank-one tearing at the left cut
    if (tid == nl - 1 && L.a1 < n) di -= fabs(B.e[L.a1 - 1]);    // and at the right cut
    d[tid] = di;
    e[tid] = (tid < nl - 1) ? B.e[a0 + tid] : 0.0;
    bad = !(isfinite(di) && isfinite(e[tid]));
  }
  if (__syncthreads_or(bad)) {  // the reduction has flagged the block; anything finite will do
    if (tid < nl) {
      d[tid] = 0.0;
      e[tid] = 0.0;
    }
    __syncthreads();
  }
  const int st = smem_dc<kLeaf / 32>(d, e, nl, Z, U, kLeafLd, e + kLeaf, ctl);
  if (st && tid == 0) atomicMax(B.info, st);
  if (tid < nl) B.lam[a0 + tid] = d[tid];
  for (int idx = tid; idx < nl * nl; idx += kCtaEigThreads) {
    const int r = idx / nl, c = idx % nl;
    B.H[(size_t)(a0 + r) * n + a0 + c] = Z[r * kLeafLd + c];
  }
}

// ---------------------------------------------------------------- divide and conquer: merge prep
// Shared-memory layout for a node of order N (P = next power of two >= N).
struct PrepLayout {
  size_t key, sidx, zs, lst, flg, fl, total;
};

__host__ __device__ inline size_t r16(size_t x) { return (x + 15) & ~(size_t)15; }

__host__ __device__ inline PrepLayout prep_layout(int N) {
  int P = 1;
  while (P < N) P <<= 1;
  PrepLayout L;
  size_t o = 0;
  L.key = o;  o += r16(sizeof(double) * (size_t)P);   // pole values, sorted
  L.sidx = o; o += r16(sizeof(int) * (size_t)P);      // original position
  L.zs = o;   o += r16(sizeof(double) * (size_t)N);   // z in sorted order
  L.lst = o;  o += r16(sizeof(int) * (size_t)N);      // sorted positions with a coupling above the tolerance
  L.flg = o;  o += r16(sizeof(int) * (size_t)N);      // those of them that are close to their successor
  L.fl = o;   o += r16((size_t)N);                    // support per sorted position; 0x80: deflated
  L.total = o;
  return L;
}

// Exclusive scan over the block of one 64-bit count per thread; `total` gets the sum. `red` holds
// one word per warp; every thread takes part.
NRG_DEV unsigned long long block_scan(unsigned long long v, unsigned long long* red, unsigned long long& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unsigned long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  __syncthreads();  // the previous call's reads of red
  if (lane == 31) red[wid] = x;
  __syncthreads();
  unsigned long long before = 0;
  total = 0;
  for (int w = 0; w < nw; w++) {
    if (w < wid) before += red[w];
    total += red[w];
  }
  return before + x - v;
}

// Poles and z of a merge, deflation, grouping of the rows by support. Everything that moves
// eigenvector rows is left to dc_secular_kernel's row CTAs, which spread over the chip; this
// kernel, one CTA per node, keeps to O(N) data. The deflation of close poles is a serial
// recurrence, but only where neighbours are close: whether a pair is close before any rotation
// is tested for all pairs at once, and one thread follows the recurrence from each such pair to
// its end. Measured on B200, 40 blocks up to order 480 (4 levels): 0.73 ms with the scan, the
// grouping and the row copies in one CTA, 0.09 ms so.
__global__ void __launch_bounds__(512) dc_prep_kernel(const LargeBlock* __restrict__ blocks,
                                                      const DcNode* __restrict__ nodes, DcState* __restrict__ states,
                                                      GemmOut* __restrict__ gouts, GemmSeg* __restrict__ gsegs,
                                                      size_t smem_bytes) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double red[32];
  __shared__ unsigned long long sred[32];
  __shared__ int s_nrot;
  const DcNode nd = nodes[blockIdx.x];
  const LargeBlock B = blocks[nd.blk];
  const int n = B.n, a = nd.a, m = nd.m, b = nd.b, N = b - a;
  const int tid = threadIdx.x, nt = blockDim.x;
  int P = 1;
  while (P < N) P <<= 1;
  const PrepLayout PL = prep_layout(N);
  // a node whose arrays do not fit the shared memory of the launch uses its rows' slice of the
  // block's global scratch (nodes of one level cover disjoint rows)
  char* smc = PL.total <= smem_bytes ? reinterpret_cast<char*>(sm) : B.pscr + kPrepGlobalB * (size_t)a;
  double* key = reinterpret_cast<double*>(smc + PL.key);
  int* sidx = reinterpret_cast<int*>(smc + PL.sidx);
  double* zs = reinterpret_cast<double*>(smc + PL.zs);
  int* lst = reinterpret_cast<int*>(smc + PL.lst);
  int* flg = reinterpret_cast<int*>(smc + PL.flg);
  unsigned char* fl = reinterpret_cast<unsigned char*>(smc + PL.fl);
  const double* Z = B.H;
  DcRot* rot = B.rot + a;

  // 1. poles and the rank-one vector z = [last row of child 1; sign(beta) first row of child 2] / sqrt(2)
  const double beta = B.e[m - 1];
  const double rho = 2.0 * fabs(beta);
  const double sg = beta >= 0.0 ? 1.0 : -1.0;
  for (int s = tid; s < P; s += nt) {
    key[s] = (s < N) ? B.lam[a + s] : INFINITY;
    sidx[s] = s;
  }
  __syncthreads();
  // 2. bitonic sort (key, sidx) ascending
  for (int k = 2; k <= P; k <<= 1) {
    for (int jb = k >> 1; jb > 0; jb >>= 1) {
      for (int i = tid; i < P; i += nt) {
        const int ixj = i ^ jb;
        if (ixj > i) {
          const bool asc = (i & k) == 0;
          const double ki = key[i], kj = key[ixj];
          const bool sw = asc ? (ki > kj || (ki == kj && sidx[i] > sidx[ixj])) : (ki < kj || (ki == kj && sidx[i] < sidx[ixj]));
          if (sw) {
            key[i] = kj;
            key[ixj] = ki;
            const int t = sidx[i];
            sidx[i] = sidx[ixj];
            sidx[ixj] = t;
          }
        }
      }
      __syncthreads();
    }
  }
  // A non-finite pole (the block was already flagged) could move a padding slot forward:
  // merge nothing at such a node rather than index outside it (its rows stay where they are).
  int badidx = 0;
  for (int s = tid; s < N; s += nt) badidx |= (sidx[s] >= N);
  if (__syncthreads_or(badidx)) {
    for (int s = tid; s < N; s += nt) B.slot[a + s] = make_int2(s, a + s < m ? 1 : 2);
    if (tid == 0) {
      atomicCAS(B.info, 0, -3);
      DcState st{};
      st.rho = rho;
      states[blockIdx.x] = st;
      for (int q = 0; q < 2; q++) {
        gouts[nd.gout + q].M = 0;
        gsegs[nd.gout + q].K = 0;
      }
    }
    return;
  }
  double dmx = 0.0, zmx = 0.0;
  for (int s = tid; s < N; s += nt) {
    const int c = a + sidx[s];
    const double z = (c < m ? Z[(size_t)c * n + (m - 1)] : sg * Z[(size_t)c * n + m]) * 0.70710678118654752440;
    zs[s] = z;
    fl[s] = (c < m) ? 1 : 2;
    dmx = fmax(dmx, fabs(key[s]));
    zmx = fmax(zmx, fabs(z));
  }
  dmx = block_max(dmx, red);
  zmx = block_max(zmx, red);
  const double tol = 8.0 * kEps * fmax(dmx, rho * zmx);  // relative to the merged matrix
  const bool none = rho * zmx <= tol;  // nothing couples the children
  // the secular equation in units in which squares neither overflow nor underflow
  const int ex = min(1000, max(-1000, ilogb(fmax(dmx, rho))));
  const double sc = scalbn(1.0, -ex);
  // 3. deflation of small couplings; the rest in order. Thread t has the positions [s0, s1).
  const int per = (N + nt - 1) / nt, s0 = min(N, tid * per), s1 = min(N, s0 + per);
  unsigned long long total;
  int cnt = 0;
  for (int s = s0; s < s1; s++) {
    if (none || rho * fabs(zs[s]) <= tol) fl[s] |= 0x80;
    else cnt++;
  }
  int o = (int)block_scan(cnt, sred, total);
  for (int s = s0; s < s1; s++)
    if (!(fl[s] & 0x80)) lst[o++] = s;
  const int L0 = (int)total;
  __syncthreads();
  // 4. close neighbours: for p, s = lst[q], lst[q+1] the rotation that zeroes z_p couples the two
  //    poles by (d_s - d_p) c sn
  auto close_pair = [&](int p, int s, double& t, double& c, double& sn) {
    const double zp = zs[p], zj = zs[s];
    t = hypot(zp, zj);
    c = zj / t;
    sn = zp / t;
    return fabs((key[s] - key[p]) * c * sn) <= tol;
  };
  const int perl = (L0 + nt - 1) / nt, q0 = min(L0, tid * perl), q1 = min(L0, q0 + perl);
  cnt = 0;
  unsigned cl = 0;  // one bit per position: perl <= 20 (the launch's thread count grows with N)
  for (int q = q0; q < q1; q++) {
    double t, c, sn;
    if (q + 1 < L0 && close_pair(lst[q], lst[q + 1], t, c, sn)) {
      cl |= 1u << (q - q0);
      cnt++;
    }
  }
  o = (int)block_scan(cnt, sred, total);
  for (int q = q0; q < q1; q++)
    if (cl >> (q - q0) & 1) flg[o++] = q;
  const int F = (int)total;
  __syncthreads();
  // 5. the chains of rotations (p, s): z_p -> 0, z_s -> t; p deflates, and s goes on with its new
  //    pole and coupling
  if (tid == 0) {
    int nrot = 0, done = 0;  // list positions below `done` are settled
    for (int f = 0; f < F; f++) {
      int q = flg[f];
      if (q < done) continue;
      while (q + 1 < L0) {
        const int p = lst[q], s = lst[q + 1];
        double t, c, sn;
        if (!close_pair(p, s, t, c, sn)) break;
        DcRot R;
        R.c = c;
        R.s = sn;
        R.p = sidx[p];
        R.j = sidx[s];
        R.sup = fl[p] | fl[s] << 2;
        R.pad = 0;
        rot[nrot++] = R;
        const double dp = key[p], ds = key[s];
        key[p] = c * c * dp + sn * sn * ds;
        key[s] = sn * sn * dp + c * c * ds;
        zs[s] = t;
        zs[p] = 0.0;
        const unsigned char u = fl[p] | fl[s];
        fl[s] = u;
        fl[p] = u | 0x80;
        q++;
      }
      done = q;
    }
    s_nrot = nrot;
  }
  __syncthreads();
  // 6. the non-deflated entries grouped by support: child 1 only, both, child 2 only (counts
  //    packed in one word: types 1, 3, 2 in 16 bits each, deflated entries in the top 16)
  unsigned long long w = 0;
  for (int s = s0; s < s1; s++) {
    const int f = fl[s];
    w += 1ull << ((f & 0x80) ? 48 : f == 1 ? 0 : f == 3 ? 16 : 32);
  }
  w = block_scan(w, sred, total);
  const int k1 = (int)(total & 0xffff), k2 = (int)(total >> 16 & 0xffff), k3 = (int)(total >> 32 & 0xffff);
  const int K = k1 + k2 + k3;
  int g1 = (int)(w & 0xffff), g2 = (int)(w >> 16 & 0xffff), g3 = (int)(w >> 32 & 0xffff), gd = (int)(w >> 48);
  for (int s = s0; s < s1; s++) {
    const int f = fl[s];
    int g;
    if (f & 0x80) {
      g = K + gd++;
      B.lam[a + g] = key[s];
    } else {
      const int t = g1 + g2 + g3;  // rank among the non-deflated poles
      g = f == 1 ? g1++ : f == 3 ? k1 + g2++ : k1 + k2 + g3++;
      B.rank[a + g] = t;
      B.dgrp[a + g] = key[s] * sc;
      B.zgrp[a + g] = zs[s];
      B.dsort[a + t] = key[s] * sc;
    }
    B.slot[a + sidx[s]] = make_int2(g, f & 3);
  }
  if (tid == 0) {
    DcState st;
    st.K = K;
    st.k1 = k1;
    st.k2 = k2;
    st.k3 = k3;
    st.rho = rho * sc;
    st.nrot = s_nrot;
    st.ex = ex;
    states[blockIdx.x] = st;
    // the two merge GEMMs: rows of child-1 columns from types 1+2, child-2 columns from 2+3
    gouts[nd.gout].M = K;
    gouts[nd.gout + 1].M = K;
    gsegs[nd.gout].K = k1 + k2;
    gsegs[nd.gout + 1].K = k2 + k3;
    gsegs[nd.gout + 1].A = B.evecs + (size_t)a * n + a + k1;
    gsegs[nd.gout + 1].B = B.W2 + (size_t)(a + k1) * n + m;
  }
}

// ---------------------------------------------------------------- divide and conquer: row moves
constexpr int kMoveCols = 32;  // columns of a row CTA's slab

// The node's eigenvector rows with the deflation rotations applied, in grouped order
// (non-deflated first, then deflated) in W2. One CTA owns a slab of 32 columns of all rows, so
// the rotations of a slab need no other CTA. A child's rows are stored for its own columns
// only; what the merge GEMMs read of a grouped row is its support, and only deflated rows are
// written out to the full width.
NRG_DEV void dc_move_rows(const LargeBlock& B, const DcNode& nd, const DcState& st, int slab) {
  const int n = B.n, a = nd.a, b = nd.b, N = b - a, c0 = a + slab * kMoveCols;
  if (c0 >= b) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int col = c0 + lane;
  const bool act = col < b;
  const int half = col < nd.m ? 1 : 2;
  if (st.nrot > 0) {  // uniform over the CTA
    if (warp == 0) {
      const DcRot* rot = B.rot + a;
      int lastj = -1;
      double zl = 0.0;
      constexpr int U = 8;  // rotations whose rows are loaded together: a row that an earlier
                            // rotation changed is always the one before's j, held in zl
      for (int r0 = 0; r0 < st.nrot; r0 += U) {
        DcRot R[U];
        double zp[U], zj[U];
#pragma unroll
        for (int u = 0; u < U; u++)
          if (r0 + u < st.nrot) R[u] = rot[r0 + u];
#pragma unroll
        for (int u = 0; u < U; u++) {
          zp[u] = zj[u] = 0.0;
          if (r0 + u < st.nrot && act) {
            const int before = u ? R[u - 1].j : lastj;
            if (R[u].p != before && (R[u].sup & half)) zp[u] = B.H[(size_t)(a + R[u].p) * n + col];
            if (R[u].sup >> 2 & half) zj[u] = B.H[(size_t)(a + R[u].j) * n + col];
          }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          if (r0 + u < st.nrot) {
            const double x = R[u].p == lastj ? zl : zp[u];
            zl = R[u].s * x + R[u].c * zj[u];
            lastj = R[u].j;
            if (act && ((R[u].sup | R[u].sup >> 2) & half)) {
              B.H[(size_t)(a + R[u].p) * n + col] = R[u].c * x - R[u].s * zj[u];
              B.H[(size_t)(a + R[u].j) * n + col] = zl;
            }
          }
        }
      }
    }
    __syncthreads();
  }
  constexpr int R = 4;  // rows in flight per warp
  for (int s = warp * R; s < N; s += nw * R) {
    int2 sl[R];
    double x[R];
#pragma unroll
    for (int u = 0; u < R; u++) {
      sl[u] = s + u < N ? B.slot[a + s + u] : make_int2(0, 0);
      x[u] = (s + u < N && act && (sl[u].y & half)) ? B.H[(size_t)(a + s + u) * n + col] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < R; u++)
      if (s + u < N && act && ((sl[u].y & half) || sl[u].x >= st.K)) B.W2[(size_t)(a + sl[u].x) * n + col] = x[u];
  }
}

// ---------------------------------------------------------------- divide and conquer: secular equation
// Root j of 1 + rho sum_i z_i^2 / (d_i - lambda) = 0 with poles d ascending. One warp per
// root, lanes over i. The root is left as the pole it was measured from and the distance, which
// give d_g - lambda_j without cancellation wherever it is needed. The CTAs blockIdx.y >= ysec move
// the node's eigenvector rows beside it (dc_move_rows).
// The iteration starts from the root of the two-pole model that the midpoint's values give, and
// the last root, which lies right of every pole, takes the model's root on that side: the other
// one is outside the bracket, and bisection in its place took 45-100 steps (the longest warp of
// the launch) where now every root takes at most ten.
// The divisions bound it, two per pole and step, so warps in flight count: four CTAs per SM.
// Measured on B200 with the row moves in it: 40 blocks up to order 480 (4 levels) 0.095 ms, from 0.59
// with bisections and 0.104 with two CTAs per SM and the K x K matrix of d_g - lambda_j written
// for the kernels below; 1400 blocks of order 601-900 21.6 ms, from 37.6 (one CTA per SM: 56).
__global__ void __launch_bounds__(256, 4) dc_secular_kernel(const LargeBlock* __restrict__ blocks,
                                                            const DcNode* __restrict__ nodes,
                                                            const DcState* __restrict__ states, int ysec) {
  const DcNode nd = nodes[blockIdx.x];
  const DcState st = states[blockIdx.x];
  const LargeBlock B = blocks[nd.blk];
  if ((int)blockIdx.y >= ysec) {
    dc_move_rows(B, nd, st, blockIdx.y - ysec);
    return;
  }
  const int K = st.K;
  if (K == 0) return;
  const int a = nd.a;
  const double rho = st.rho;
  const int lane = threadIdx.x & 31;
  const int wg = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int wstride = ysec * (blockDim.x >> 5);
  const double* ds = B.dsort + a;
  const double* dg = B.dgrp + a;
  const double* zg = B.zgrp + a;
  const int* rk = B.rank + a;
  for (int j = wg; j < K; j += wstride) {
    double dorg, lo, hi, tau;
    int p1, p2;
    if (K == 1) {
      const double z = zg[0];
      if (lane == 0) {
        B.rorg[a] = ds[0];
        B.rtau[a] = rho * z * z;
        B.lam[a] = scalbn(ds[0] + rho * z * z, st.ex);
      }
      continue;
    }
    const bool last = j == K - 1;
    if (!last) {
      p1 = j;
      p2 = j + 1;
      const double dj = ds[j], gap = ds[j + 1] - dj, mid = 0.5 * gap;
      double s = 0.0, z1 = 0.0, z2 = 0.0;  // the function at the midpoint; the two poles' residues
      for (int i = lane; i < K; i += 32) {
        const double z = zg[i];
        const int r = rk[i];
        if (r == p1) z1 = z * z;
        if (r == p2) z2 = z * z;
        s += z * z / ((dg[i] - dj) - mid);
      }
      const double f = 1.0 + rho * warp_sum(s);
      z1 = rho * warp_sum(z1);
      z2 = rho * warp_sum(z2);
      if (f >= 0.0) {
        dorg = dj;
        lo = 0.0;
        hi = mid;
      } else {
        dorg = ds[j + 1];
        lo = -mid;
        hi = 0.0;
      }
      tau = secular_start(f, f + (z1 - z2) / mid, gap, z1, z2);
      if (!(tau > lo && tau < hi)) tau = 0.5 * (lo + hi);
    } else {
      double s = 0.0;
      for (int i = lane; i < K; i += 32) s += zg[i] * zg[i];
      dorg = ds[K - 1];
      lo = 0.0;
      hi = rho * warp_sum(s);
      p1 = K - 2;
      p2 = K - 1;
      tau = 0.5 * hi;
    }
    const double d1 = ds[p1] - dorg, d2 = ds[p2] - dorg;
    for (int it = 0; it < 100; it++) {
      double psi = 0.0, dpsi = 0.0, phi = 0.0, dphi = 0.0;
#pragma unroll 4
      for (int i = lane; i < K; i += 32) {
        const double z = zg[i], t = z / ((dg[i] - dorg) - tau);
        const bool left = rk[i] <= p1;
        const double zl = left ? z : 0.0, tl = left ? t : 0.0, zr = left ? 0.0 : z, tr = left ? 0.0 : t;
        psi = fma(zl, t, psi);
        dpsi = fma(tl, t, dpsi);
        phi = fma(zr, t, phi);
        dphi = fma(tr, t, dphi);
      }
      psi = rho * warp_sum(psi);
      dpsi = rho * warp_sum(dpsi);
      phi = rho * warp_sum(phi);
      dphi = rho * warp_sum(dphi);
      const double f = 1.0 + psi + phi;
      const double err = 8.0 * (fabs(psi) + fabs(phi)) + 2.0 + 3.0 * fabs(tau) * (dpsi + dphi);
      if (fabs(f) <= kEps * err) break;
      if (f < 0.0) lo = tau; else hi = tau;
      double tn = tau + secular_step(f, dpsi, dphi, d1 - tau, d2 - tau, last);
      if (!(tn > lo && tn < hi)) tn = 0.5 * (lo + hi);
      if (tn == tau) break;
      tau = tn;
    }
    if (lane == 0) {
      B.rorg[a + j] = dorg;
      B.rtau[a + j] = tau;
      B.lam[a + j] = scalbn(dorg + tau, st.ex);
    }
  }
}

// ---------------------------------------------------------------- divide and conquer: vectors
// z-hat by the Gu-Eisenstat product formula (into zgrp, free after the secular solve), then
// u_j(g) = zhat_g / (d_g - lambda_j), normalised, in grouped column order. Both kernels spread a
// node over gridDim.y CTAs, and form d_g - lambda_j from the poles and (rorg, rtau): that they need no
// matrix of these, and one division per entry, brought 1400 blocks of order 601-900 from 16.2 to
// 12.0 ms.
// A CTA takes 32 columns g and splits the product over the roots between its eight warps (the
// chain of K dependent multiplications and divisions was the whole time of small batches: 0.52 ms
// of a step of 40 blocks up to order 480 with one thread per column, both kernels, 0.077 ms now).
__global__ void __launch_bounds__(256) dc_zhat_kernel(const LargeBlock* __restrict__ blocks,
                                                      const DcNode* __restrict__ nodes,
                                                      const DcState* __restrict__ states) {
  __shared__ double part[8][32];
  const DcNode nd = nodes[blockIdx.x];
  const DcState st = states[blockIdx.x];
  const int K = st.K, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = blockIdx.y * 32 + lane;
  if ((int)blockIdx.y * 32 >= K) return;  // uniform over the CTA
  const LargeBlock B = blocks[nd.blk];
  const int a = nd.a;
  const double* ds = B.dsort + a;
  const double* og = B.rorg + a;
  const double* rt = B.rtau + a;
  double p = 1.0;
  if (g < K) {
    const int i = B.rank[a + g];
    const double di = ds[i];
#pragma unroll 4
    for (int j = warp; j < K - 1; j += 8) p *= -((di - og[j]) - rt[j]) / (ds[j < i ? j : j + 1] - di);
    if (warp == 0) p *= -((di - og[K - 1]) - rt[K - 1]) / st.rho;
  }
  part[warp][lane] = p;
  __syncthreads();
  if (warp == 0 && g < K) {
    double q = 1.0;
#pragma unroll
    for (int v = 0; v < 8; v++) q *= part[v][lane];
    B.zgrp[a + g] = copysign(sqrt(fabs(q)), B.zgrp[a + g]);
  }
}

__global__ void __launch_bounds__(256) dc_vectors_kernel(const LargeBlock* __restrict__ blocks,
                                                         const DcNode* __restrict__ nodes,
                                                         const DcState* __restrict__ states) {
  const DcNode nd = nodes[blockIdx.x];
  const DcState st = states[blockIdx.x];
  const LargeBlock B = blocks[nd.blk];
  const int K = st.K;
  const int n = B.n, a = nd.a, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int wg = blockIdx.y * (blockDim.x >> 5) + warp, wstride = gridDim.y * (blockDim.x >> 5);
  // deflated rows are final: grouped copy (W2) back to the node's rows a+K.. (H)
  for (int r = a + K + wg; r < nd.b; r += wstride)
    for (int col = a + lane; col < nd.b; col += 32) B.H[(size_t)r * n + col] = B.W2[(size_t)r * n + col];
  const double* zh = B.zgrp + a;
  const double* dg = B.dgrp + a;
  for (int j = wg; j < K; j += wstride) {
    double* row = B.evecs + (size_t)(a + j) * n + a;
    const double og = B.rorg[a + j], rt = B.rtau[a + j];
    constexpr int U = 16;  // entries a lane keeps between the norm and the scaled store
    double u[U], ss = 0.0;
#pragma unroll
    for (int q = 0; q < U; q++) {
      if (32 * q >= K) break;
      const int g = lane + 32 * q;
      u[q] = g < K ? zh[g] / ((dg[g] - og) - rt) : 0.0;
      ss = fma(u[q], u[q], ss);
    }
#pragma unroll 4
    for (int g = lane + 32 * U; g < K; g += 32) {
      const double x = zh[g] / ((dg[g] - og) - rt);
      ss = fma(x, x, ss);
    }
    const double inv = 1.0 / sqrt(warp_sum(ss));
#pragma unroll
    for (int q = 0; q < U; q++) {
      if (32 * q >= K) break;
      const int g = lane + 32 * q;
      if (g < K) row[g] = u[q] * inv;
    }
#pragma unroll 4
    for (int g = lane + 32 * U; g < K; g += 32) row[g] = zh[g] / ((dg[g] - og) - rt) * inv;
  }
}

// ---------------------------------------------------------------- final order
__global__ void __launch_bounds__(1024) sort_final_kernel(const LargeBlock* __restrict__ blocks) {
  extern __shared__ __align__(16) double key[];
  const LargeBlock B = blocks[blockIdx.x];
  const int n = B.n, tid = threadIdx.x, nt = blockDim.x;
  int P = 1;
  while (P < n) P <<= 1;
  int* idx = reinterpret_cast<int*>(key + P);
  for (int s = tid; s < P; s += nt) {
    key[s] = (s < n) ? B.lam[s] : INFINITY;
    idx[s] = s;
  }
  __syncthreads();
  for (int k = 2; k <= P; k <<= 1) {
    for (int jb = k >> 1; jb > 0; jb >>= 1) {
      for (int i = tid; i < P; i += nt) {
        const int ixj = i ^ jb;
        if (ixj > i) {
          const bool asc = (i & k) == 0;
          const double ki = key[i], kj = key[ixj];
          const bool sw = asc ? (ki > kj || (ki == kj && idx[i] > idx[ixj])) : (ki < kj || (ki == kj && idx[i] < idx[ixj]));
          if (sw) {
            key[i] = kj;
            key[ixj] = ki;
            const int t = idx[i];
            idx[i] = idx[ixj];
            idx[ixj] = t;
          }
        }
      }
      __syncthreads();
    }
  }
  for (int s = tid; s < n; s += nt) {
    B.evals[s] = key[s];
    B.perm[s] = idx[s];
  }
}

// evecs[r][:] = W1[perm[r]][:]; grid (rows / 8, blocks)
__global__ void __launch_bounds__(256) permute_rows_kernel(const LargeBlock* __restrict__ blocks) {
  const LargeBlock B = blocks[blockIdx.y];
  const int n = B.n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.x * 8 + warp;
  if (r >= n) return;
  int pr = B.perm[r];
  if (pr < 0 || pr >= n) pr = r;  // only after a flagged non-finite block
  const double* src = B.H + (size_t)pr * n;
  double* dst = B.evecs + (size_t)r * n;
  for (int c = lane; c < n; c += 32) dst[c] = src[c];
}

// ---------------------------------------------------------------- back-transform factors
// T of the compact-WY form H_k0 ... H_k0+nb-1 = I - V T V^T (forward, columnwise), from
// the Gram matrix G = V^T V (nb x nb) at GT + gt_off, written to GT + gt_off + nb^2.
struct PanelRef {
  int blk, k0, nb, pad;
  long long gt_off;
};

// The columns of T depend on one another, but T = [T1, -T1 G12 T2; 0, T2] for any split: the 16 x 16
// diagonal blocks come from the recurrence, one warp each, and are merged 16 -> 32 -> 64 -> 128 by
// two small DMMA products per merge, in place of G in shared memory. A reflector with tau = 0
// has a zero row and column in T, which the products keep. Measured on B200: 40 blocks up to
// order 480 (66 panels) 226 us with the 128-step recurrence in one CTA, 39 us now; 1400 blocks of
// order 601-900 13.3 and 2.1 ms.
constexpr int kTfThreads = 256;
constexpr int kTfLd = NBT + 4, kTfLx = NBT / 2 + 4;

// Tile of 8 x 8 of A B (A rows m0.., B columns n0.., inner index k0 <= k < k1, multiples of 4).
NRG_DEV void tf_tile(const double* A, int lda, const double* Bm, int ldb, int m0, int n0, int k0, int k1, double& d0,
                     double& d1) {
  const int lane = threadIdx.x & 31, fr = lane >> 2, fc = lane & 3;
  d0 = d1 = 0.0;
  for (int k = k0; k < k1; k += 4) dmma884(d0, d1, A[(m0 + fr) * lda + k + fc], Bm[(k + fc) * ldb + n0 + fr]);
}

__global__ void __launch_bounds__(kTfThreads) tfactor_kernel(const LargeBlock* __restrict__ blocks,
                                                             const PanelRef* __restrict__ panels) {
  extern __shared__ __align__(16) double tsm[];
  const PanelRef P = panels[blockIdx.x];
  const LargeBlock B = blocks[P.blk];
  const int nb = P.nb, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* Ts = tsm;                // NBT x kTfLd: G above the diagonal, then T
  double* X = tsm + NBT * kTfLd;   // G12 T2 of the merges of one level
  const double* G = B.GT + P.gt_off;
  double* T = B.GT + P.gt_off + (size_t)nb * nb;
  const int nbr = (nb + 15) / 16 * 16;
  for (int r = warp; r < nbr; r += kTfThreads / 32)
    for (int c = lane; c < nbr; c += 32) Ts[r * kTfLd + c] = (c > r && c < nb) ? G[(size_t)r * nb + c] : 0.0;
  __syncthreads();
  if (16 * warp < nbr) {  // diagonal block of 16: lane t holds row t
    const int o = 16 * warp;
    double row[16];
#pragma unroll
    for (int q = 0; q < 16; q++) {
      const double tq = (o + q < nb) ? B.tau[P.k0 + o + q] : 0.0;
      double s = 0.0;
#pragma unroll
      for (int r = 0; r < q; r++) {
        const double w = -tq * Ts[(o + r) * kTfLd + o + q];
        if (r >= lane) s += row[r] * w;
      }
      row[q] = lane == q ? tq : lane < q ? s : 0.0;
    }
    __syncwarp();
    if (lane < 16) {
#pragma unroll
      for (int q = 0; q < 16; q++) Ts[(o + lane) * kTfLd + o + q] = row[q];
    }
  }
  __syncthreads();
  const int fr = lane >> 2, fc = lane & 3;
  for (int h = 16; h < nbr; h *= 2) {  // merge neighbours of order h (the last one may be shorter)
    const int q8 = h / 8, per = q8 * q8, nm = (nbr + 2 * h - 1) / (2 * h);
    for (int u = warp; u < nm * per; u += kTfThreads / 32) {
      const int o = (u / per) * 2 * h, i = (u % per) / q8 * 8, j = (u % per) % q8 * 8;
      if (o + h + j >= nbr) continue;
      double d0, d1;
      tf_tile(Ts + o * kTfLd + o + h, kTfLd, Ts + (o + h) * kTfLd + o + h, kTfLd, i, j, 0, j + 8, d0, d1);
      double* x = X + ((u / per) * h + i + fr) * kTfLx + j + 2 * fc;
      x[0] = d0;
      x[1] = d1;
    }
    __syncthreads();
    for (int u = warp; u < nm * per; u += kTfThreads / 32) {
      const int o = (u / per) * 2 * h, i = (u % per) / q8 * 8, j = (u % per) % q8 * 8;
      if (o + h + j >= nbr) continue;
      double d0, d1;
      tf_tile(Ts + o * kTfLd + o, kTfLd, X + (u / per) * h * kTfLx, kTfLx, i, j, i, h, d0, d1);
      double* y = Ts + (o + i + fr) * kTfLd + o + h + j + 2 * fc;
      y[0] = -d0;
      y[1] = -d1;
    }
    __syncthreads();
  }
  for (int r = warp; r < nb; r += kTfThreads / 32)
    for (int c = lane; c < nb; c += 32) T[(size_t)r * nb + c] = Ts[r * kTfLd + c];
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    else
      cudaGetLastError();
  }
  return fn;
}

size_t large_block_doubles(int n, bool two_stage) {
  const size_t ldp = (size_t)(n + 31) / 32 * 32;
  return (size_t)n * ldp + (size_t)n * n + 8 * (size_t)n + 2 * (size_t)NBT * n + 9 * (size_t)n + 64 * 18 + grid_scratch_doubles(n) +
         (prep_layout(n).total > kPrepSmemMax ? (kPrepGlobalB * (size_t)n + 7) / 8 : 0) +
         (two_stage ? band_extra_doubles(n) + 4 * 64 : 0);
}

// Largest order that a cluster of 16 holds.
int dsm_max_order() {
  static const int n = [] {
    int k = kDsmMaxN;
    while (!dsm_fits(k, 16)) k--;
    return k;
  }();
  return n;
}

// Microseconds of a block's reduction in a C-cluster (B200, see tridiag_dsm_kernel).
double dsm_us(int n, int C) { return n * (1.42 + 7.5e-5 * n * n / C); }

// Microseconds of a block's reduction by a group of G CTAs (B200, see tridiag_grid_kernel): the chain of
// columns and the bytes an SM streams, 75 GB/s from L2; 45 when the chip streams from HBM, and 30 where it is
// the largest blocks that count.
constexpr double kGroupL2 = 75.0, kGroupHbm = 45.0, kGroupHbmLow = 30.0;
double grid_us(int n, int G, double gbs) { return n * (5.2 + 8.0 / 3.0 * n * n / (1e3 * gbs * G)); }
int grid_min_ctas(int n) { return (n + kGridMaxT - 1) / kGridMaxT; }
int grid_max_ctas(int n) { return std::min(kGridMaxG, std::max(grid_min_ctas(n), n / 16)); }

// Shared memory of a CTA of tridiag_kernel for blocks up to order n with ny copies of the product.
size_t tri_smem(int n, int ny) {
  return 1024 + sizeof(double) * ((size_t)kTriWarps * kTriStages * kSlabD + (size_t)(1 + ny) * tri_pad(n) +
                                  4 * NB + 64);
}
// Copies of the product: one per warp, or two where that leaves no room for two CTAs in an SM's smsm
// bytes (1 KB is reserved per CTA), or 0 if two do not fit either.
int tri_copies(int n, int smsm) {
  for (int ny : {kTriWarps, 2})
    if (2 * (tri_smem(n, ny) + 1024 + 256) <= (size_t)smsm) return ny;
  return 0;
}

// ... in a CTA of tridiag_kernel, two per SM (alone on the chip 10 n + 5e-5 n^3), and in
// tridiag_smem_kernel.
double stream_us(int n) { return n * (10.0 + 7.2e-5 * n * n); }
double smem_us(int n) { return n * (2.0 + 1.4e-4 * n * n); }

// How blocks sorted by falling order are reduced: [0, ngrid) by groups of CTAs, [ngrid, cut) and
// [mid, nb) by clusters of C[q] (C = 0: tridiag_smem_kernel), [cut, mid) by the streaming kernel.
// While the least clusters and groups of all blocks fit the SMs at once the longest chain bounds the
// call: no block streams, and clusters double, the slowest block first, as long as they fit. Otherwise
// the SMs' time does. Of that the streaming kernel takes least from order mid_max_n on (SM ms of a block
// of order 250 / 500 / 850: 1.9 / 7 / 26; clusters 2.7 / 21, groups - / 9 / 45), but its blocks take longest: so
// the shortest span is sought, in steps of 5%, in which the blocks that stream within it do, groups take
// the larger ones, and the SMs (85% of them) have time for all. It has to be 7% below what clusters
// and groups alone take. (Clusters beside streamed blocks starve: those take each SM that falls free.)
// Measured on B200, reductions in ms by clusters and groups alone / all streamed / this plan: 300 blocks
// of order 225-300 6.9 / 4.3 / 4.3, 100 of 400-600 17 / 16.5 / 9.7, 300 of 400-600 50 / 19 / 17, 1400 of 601-900
// 489 / 189 / 189, 300 of 225-1000 46 / 66 / 33, 1500 of 8-2048 569 / 656 / 384, 500 of 1200-1500 667 / 363 / 377, 160
// of 1800-2200 670 / 770 / 683, 300 of 8-1024 13.9 / 74 / 13.9; 12 of order 800-2000 16 by groups, 93 by one
// cluster of 8 or 16 CTAs each; one of order 7049 263 by a group, 623 in two stages (band_min_n).
struct ReductionPlan {
  int ngrid = 0, cut = 0, mid = 0;
  int nsm_grid = 0;  // SMs for the groups
  std::vector<int> C;
};

ReductionPlan reduction_plan(const LargeBlock* b, int nb, int cluster_max_n, int mid_max_n, int nsm, int smsm,
                             bool may_stream) {
  ReductionPlan p;
  p.C.assign(nb, 0);
  // SM time of the first q blocks: by clusters or groups; by groups; streamed
  std::vector<double> wl(nb + 1, 0.0), wg(nb + 1, 0.0), ws(nb + 1, 0.0);
  double foot = 0.0;
  for (; p.ngrid < nb && b[p.ngrid].n > cluster_max_n; p.ngrid++) foot += 8.0 * b[p.ngrid].n * b[p.ngrid].n;
  const double gbs = foot > 1e8 ? kGroupHbm : kGroupL2;
  int sum = 0;
  for (int q = 0; q < nb; q++) {
    const int n = b[q].n, G = grid_min_ctas(n);
    const double group = G * grid_us(n, G, gbs);
    if (q < p.ngrid) {
      sum += G;
      wl[q + 1] = wl[q] + group;
    } else {
      int C = 1;
      while (!dsm_fits(n, C)) C *= 2;
      p.C[q] = C;
      sum += C;
      wl[q + 1] = wl[q] + (n > mid_max_n ? C * dsm_us(n, C) : smem_us(n));
    }
    if (n > mid_max_n) p.mid = q + 1;
    wg[q + 1] = wg[q] + group;
    ws[q + 1] = ws[q] + 0.5 * stream_us(n);
  }
  p.cut = p.mid;
  const double wmid = wl[nb] - wl[p.mid];
  if (sum > nsm && p.mid > 0 && may_stream) {
    const double chain = p.ngrid > 0 ? grid_us(b[0].n, grid_max_ctas(b[0].n), gbs) : dsm_us(b[0].n, 16);
    const double most = 0.93 * std::max(chain, wl[nb] / (0.95 * nsm));
    for (double span = chain; span < most; span *= 1.05) {
      const int cut = (int)(std::partition_point(b, b + p.mid, [&](const LargeBlock& x) {
                              return stream_us(x.n) > span || !tri_copies(x.n, smsm);
                            }) - b);
      if (wg[cut] + (ws[p.mid] - ws[cut]) + wmid > 0.85 * nsm * span) continue;
      if (cut < p.mid) p.ngrid = p.cut = cut;
      break;
    }
  }
  int most = 1, clusters = 0;
  double wrest = ws[p.mid] - ws[p.cut], wgrid = 0.0;
  foot = 0.0;
  for (int q = 0; q < p.ngrid; q++) foot += 8.0 * b[q].n * b[q].n;
  for (int q = 0; q < nb; q++) {
    const int n = b[q].n, G = grid_min_ctas(n);
    if (q < p.ngrid) {
      wgrid += G * grid_us(n, G, foot < 1e8 ? kGroupL2 : p.cut < p.mid ? kGroupHbm : kGroupHbmLow);
    } else if (q < p.cut || q >= p.mid) {
      most = std::max(most, p.C[q]);
      clusters += p.C[q];
      wrest += p.C[q] * dsm_us(n, p.C[q]);
    }
  }
  if (p.ngrid > 0)  // SMs in proportion to the work
    p.nsm_grid = p.ngrid == nb ? nsm
                               : nsm - std::min(nsm - grid_min_ctas(b[0].n),
                                                std::max(most, (int)(nsm * wrest / (wgrid + wrest))));
  if (p.cut == p.mid && clusters <= nsm - p.nsm_grid) {
    for (;;) {
      int best = -1;
      double tb = 0.0;
      for (int q = p.ngrid; q < nb; q++)
        if (dsm_us(b[q].n, p.C[q]) > tb) tb = dsm_us(b[q].n, p.C[best = q]);
      if (best < 0 || p.C[best] == 16 || clusters + p.C[best] > nsm - p.nsm_grid) return p;
      clusters += p.C[best];
      p.C[best] *= 2;
    }
  }
  // Blocks that fit one CTA's packed triangle stay in one CTA (two would take 1.3 times the SM time of
  // that kernel from order 160 on, and it half as much again as the full square below).
  for (int q = p.mid; q < nb; q++)
    if (p.C[q] > 1) p.C[q] = 0;
  return p;
}

struct GridPlan {
  std::vector<GridGroup> groups;
  std::vector<int> jobs;
  int ctas = 0;
  size_t smem = 0;
  double us = 0.0;  // of the slowest group
};

// Groups for the blocks [0, count) (sorted by falling order) on nsm SMs: the shortest makespan, in steps of
// 5%, for which the blocks fit, each the first group that still has time for it or else a new one of
// the least size that is fast enough; what SMs are left go to the slowest groups.
GridPlan grid_plan(const LargeBlock* b, int count, int nsm) {
  double foot = 0.0;
  for (int q = 0; q < count; q++) foot += 8.0 * b[q].n * b[q].n;
  const double gbs = foot > 1e8 ? kGroupHbmLow : kGroupL2;
  struct Group { int G, cap; double us; std::vector<int> list; };
  std::vector<Group> gs;
  double span = grid_us(b[0].n, std::min(nsm, grid_max_ctas(b[0].n)), gbs);
  for (;; span *= 1.05) {
    gs.clear();
    int used = 0;
    bool ok = true;
    for (int q = 0; q < count && ok; q++) {
      const int n = b[q].n, lo = grid_min_ctas(n);
      Group* to = nullptr;
      for (Group& g : gs)
        if (!to && g.G >= lo && g.us + grid_us(n, std::min(g.G, grid_max_ctas(n)), gbs) <= span) to = &g;
      if (!to) {
        int G = lo;
        while (G < grid_max_ctas(n) && grid_us(n, G, gbs) > span) G++;
        ok = grid_us(n, G, gbs) <= span * 1.0001 && used + G <= nsm;
        if (!ok) break;
        used += G;
        gs.push_back(Group{G, grid_max_ctas(n), 0.0, {}});
        to = &gs.back();
      }
      to->us += grid_us(n, to->G, gbs);
      to->list.push_back(q);
    }
    if (!ok) continue;
    while (used < nsm) {  // the rest
      Group* slow = nullptr;
      for (Group& g : gs)
        if (g.G < g.cap && (!slow || g.us > slow->us)) slow = &g;
      if (!slow) break;
      slow->G++;
      used++;
      slow->us = 0.0;
      for (int q : slow->list) slow->us += grid_us(b[q].n, slow->G, gbs);
    }
    break;
  }
  GridPlan p;
  for (const Group& g : gs) {
    p.groups.push_back(GridGroup{p.ctas, g.G, (int)p.jobs.size(), (int)g.list.size()});
    p.jobs.insert(p.jobs.end(), g.list.begin(), g.list.end());
    p.ctas += g.G;
    p.us = std::max(p.us, g.us);
    for (int q : g.list)
      p.smem = std::max(p.smem, sizeof(double) * grid_smem_doubles(b[q].ldp, (b[q].n + g.G - 1) / g.G));
  }
  return p;
}

cudaError_t reduce_in_smem_launch(const LargeBlock* d_blk, int maxn, int count, int C, cudaStream_t s) {
  if (C == 0) {
    const size_t smem = sizeof(double) * ((size_t)maxn * (maxn + 1) / 2 + 2 * (size_t)maxn + 64);
    cudaError_t e = cudaFuncSetAttribute(tridiag_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    tridiag_smem_kernel<<<count, kMidThreads, smem, s>>>(d_blk);
    return cudaGetLastError();
  }
  const void* fn = C == 16 ? (const void*)tridiag_dsm_kernel<16> : C == 8 ? (const void*)tridiag_dsm_kernel<8>
                   : C == 4 ? (const void*)tridiag_dsm_kernel<4> : C == 2 ? (const void*)tridiag_dsm_kernel<2>
                                                                          : (const void*)tridiag_dsm_kernel<1>;
  const size_t smem = sizeof(double) * dsm_smem_doubles(maxn, C);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess && C == 16) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(count * C));
  cfg.blockDim = dim3(kDsmThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  void* kargs[] = {(void*)&d_blk};
  return cudaLaunchKernelExC(&cfg, fn, kargs);
}

int tri_streams(nrg_ctx* c) {
  if (c->tri_fork) return NRG_OK;
  for (int i = 0; i < nrg_ctx::kTriStreams; i++) {
    if (!c->tri[i]) NRG_CK(cudaStreamCreateWithFlags(&c->tri[i], cudaStreamNonBlocking));
    if (!c->tri_join[i]) NRG_CK(cudaEventCreateWithFlags(&c->tri_join[i], cudaEventDisableTiming));
  }
  NRG_CK(cudaEventCreateWithFlags(&c->tri_fork, cudaEventDisableTiming));
  return NRG_OK;
}

}  // namespace

int eig_large_run(nrg_ctx* c, const std::vector<int>& which, const int* n, double* const* H, double* const* evals,
                  double* const* evecs, int* info_dev, cudaStream_t s, const std::function<int()>& beside) {
  std::vector<int> ord(which);
  std::stable_sort(ord.begin(), ord.end(), [n](int x, int y) { return n[x] > n[y]; });
  const int mid_max_n = c->tune.mid_max_n, cluster_max_n = c->tune.cluster_max_n;
  // Two-stage reduction for the largest blocks when they are few (the first nts of `ord`).
  int nts_all = 0;
  if (c->tune.band_min_n > 0) {
    while (nts_all < (int)ord.size() && n[ord[nts_all]] >= c->tune.band_min_n) nts_all++;
    if (nts_all > c->tune.band_max_blocks) nts_all = 0;
  }
  for (int b : ord)
    if (n[b] > kMaxLargeN)
      return fail(NRG_ERR_ARG, "block %d: order %d exceeds the supported maximum %d", b, n[b], kMaxLargeN);
  // Chunk the blocks so that their workspaces fit in the context limit.
  size_t all_bytes = 0;
  for (size_t t = 0; t < ord.size(); t++)
    all_bytes += align_up(sizeof(double) * large_block_doubles(n[ord[t]], (int)t < nts_all), 256);
  // Chunks fit what the arena can grow to now; a call that fits the arena as it is asks the device
  // for nothing (cudaMemGetInfo now and then stalls the host for milliseconds).
  const size_t limit = all_bytes <= c->ws_size ? c->ws_size : ws_available(c);
  size_t pos = 0;
  while (pos < ord.size()) {
    size_t bytes = 0, end = pos;
    while (end < ord.size()) {
      const size_t bb = align_up(sizeof(double) * large_block_doubles(n[ord[end]], (int)end < nts_all), 256);
      if (end > pos && bytes + bb > limit) break;
      bytes += bb;
      end++;
    }
    int rc = ensure_ws(c, bytes);
    if (rc) return rc;
    // ---- per-block descriptors
    std::vector<LargeBlock> blk;
    std::vector<BandBlock> bblk;  // the chunk's two-stage blocks (its first nts, the largest)
    std::vector<int> shift;       // row offset of each block's reflectors: 1, or kBand (two-stage)
    char* base = static_cast<char*>(c->ws);
    size_t off = 0;
    int maxn = 0, maxpanel = 0;
    const int nts = std::max(0, std::min((int)end, nts_all) - (int)pos);
    for (size_t t = pos; t < end; t++) {
      const int b = ord[t], nb_ = n[b];
      LargeBlock L{};
      auto take = [&](size_t nd) {
        double* p = reinterpret_cast<double*>(base + off);
        off += align_up(sizeof(double) * nd, 256);
        return p;
      };
      L.H = H[b];
      L.evals = evals[b];
      L.evecs = evecs[b];
      L.ldp = (nb_ + 31) / 32 * 32;
      L.W1 = take((size_t)nb_ * L.ldp);
      L.W2 = take((size_t)nb_ * nb_);
      L.d = take(nb_);
      L.e = take(nb_);
      L.tau = take(nb_);
      L.lam = take(nb_);
      L.dsort = take(nb_);
      L.dgrp = take(nb_);
      L.zgrp = take(nb_);
      L.rorg = take(nb_);
      L.rtau = take(nb_);
      L.npanel = (nb_ - 2 + NBT - 1) / NBT;
      L.GT = take(2 * (size_t)NBT * nb_);  // >= sum over panels of 2 nb^2
      int* ip = reinterpret_cast<int*>(take(nb_));
      L.rank = ip;
      L.perm = ip + nb_;
      L.pscr = prep_layout(nb_).total > kPrepSmemMax
                   ? reinterpret_cast<char*>(take((kPrepGlobalB * (size_t)nb_ + 7) / 8)) : nullptr;
      L.slot = reinterpret_cast<int2*>(take(nb_));
      L.rot = reinterpret_cast<DcRot*>(take(4 * (size_t)nb_));
      L.gx = take(grid_scratch_doubles(nb_));
      L.info = info_dev + b;
      L.n = nb_;
      if ((int)(t - pos) < nts) {
        // two-stage: reflectors of stage 1 at rows k, unit at k + kBand; n - 1 - kBand of them
        const int K1 = std::max(0, nb_ - 1 - kBand);
        L.npanel = (K1 + NBT - 1) / NBT;
        BandBlock Bb{};
        Bb.S = L.W1;
        Bb.H = L.H;
        Bb.lds = L.ldp;
        Bb.n = nb_;
        Bb.J = band_nsteps(nb_, 0);
        int jf = 0;
        while (nb_ - jf - kBand > 1) jf += kBand;
        Bb.jfin = jf;
        Bb.BND = take((size_t)nb_ * kLDB);
        Bb.V2 = take((size_t)band_nsweeps(nb_) * Bb.J * kBand);
        Bb.tau2 = take((size_t)band_nsweeps(nb_) * Bb.J);
        Bb.T2 = take((size_t)band_ngroups(nb_) * Bb.J * kGrp * kGrp);
        Bb.tau1 = L.tau;
        Bb.scr = L.W2;
        Bb.d = L.d;
        Bb.e = L.e;
        Bb.evecs = L.evecs;
        Bb.info = L.info;
        bblk.push_back(Bb);
        shift.push_back(kBand);
      } else {
        shift.push_back(1);
      }
      blk.push_back(L);
      maxn = std::max(maxn, nb_);
      maxpanel = std::max(maxpanel, L.npanel);
    }
    const int nb = (int)blk.size();
    if (off > c->ws_size) return fail(NRG_ERR_ARG, "internal: chunk workspace %zu > %zu", off, c->ws_size);
    // ---- 2-D tensor maps over each block's packed lower triangle (box 64 rows x 8 columns)
    std::vector<CUtensorMap> tmaps(nb);
    {
      auto encode = tensor_map_encoder();
      if (!encode) return fail(NRG_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
      for (int bi = nts; bi < nb; bi++) {
        const LargeBlock& L = blk[bi];
        if (L.n <= mid_max_n) continue;  // reduced in the shared memory of one CTA, no bulk copies
        const cuuint64_t dims[2] = {(cuuint64_t)L.ldp, (cuuint64_t)L.n};
        const cuuint64_t strides[1] = {(cuuint64_t)L.ldp * sizeof(double)};
        const cuuint32_t box[2] = {(cuuint32_t)kSlabRows, 8u};
        const cuuint32_t estr[2] = {1u, 1u};
        const CUresult r = encode(&tmaps[bi], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, L.W1, dims, strides, box, estr,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(NRG_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) for n=%d", (int)r, L.n);
      }
    }
    // ---- divide-and-conquer tree (leaves and merge levels by height)
    std::vector<DcLeaf> leaves;
    std::vector<std::vector<DcNode>> levels;
    std::function<int(int, int, int)> build = [&](int bi, int lo, int hi) -> int {
      if (hi - lo <= kLeaf) {
        leaves.push_back(DcLeaf{bi, lo, hi, 0});
        return 0;
      }
      const int mid = lo + (hi - lo) / 2;
      const int h = 1 + std::max(build(bi, lo, mid), build(bi, mid, hi));
      if ((int)levels.size() < h) levels.resize(h);
      DcNode nd{};
      nd.blk = bi;
      nd.a = lo;
      nd.m = mid;
      nd.b = hi;
      levels[h - 1].push_back(nd);
      return h;
    };
    for (int bi = 0; bi < nb; bi++) build(bi, 0, blk[bi].n);
    // ---- one staging image for the whole chunk
    std::vector<char> img;
    const size_t blk_off = push(img, blk);
    const size_t tmap_off = push(img, tmaps);
    const size_t leaf_off = push(img, leaves);
    std::vector<size_t> node_off(levels.size()), st_off(levels.size());
    std::vector<StagedGemm> lvl_gemm(levels.size());
    for (size_t h = 0; h < levels.size(); h++) {
      GemmPlan gp;
      for (auto& nd : levels[h]) {
        const LargeBlock& L = blk[nd.blk];
        const int N = nd.b - nd.a, nn = L.n;
        nd.gout = (int)gp.outs.size();
        // child-1 columns: C = Zt[a:a+K, a:m] = U[:, 0:k1+k2] * G[a:a+k1+k2, a:m]
        gp.add_out(L.H + (size_t)nd.a * nn + nd.a, nn, N, nd.m - nd.a, 0.0);
        gp.add_seg(L.evecs + (size_t)nd.a * nn + nd.a, nn, 0, L.W2 + (size_t)nd.a * nn + nd.a, nn, 0, N, 1.0);
        // child-2 columns: C = Zt[a:a+K, m:b] = U[:, k1:K] * G[a+k1:a+K, m:b] (pointers set on device)
        gp.add_out(L.H + (size_t)nd.a * nn + nd.m, nn, N, nd.b - nd.m, 0.0);
        gp.add_seg(L.evecs + (size_t)nd.a * nn + nd.a, nn, 0, L.W2 + (size_t)nd.a * nn + nd.m, nn, 0, N, 1.0);
      }
      node_off[h] = push(img, levels[h]);
      st_off[h] = push(img, std::vector<DcState>(levels[h].size()));
      lvl_gemm[h] = stage_gemm(img, gp);
    }
    // back-transform: Gram, T, VT, then per panel step two GEMMs
    std::vector<PanelRef> panels;
    GemmPlan gram, vt;
    std::vector<GemmPlan> bsteps(maxpanel * 2);
    for (int bi = 0; bi < nb; bi++) {
      const LargeBlock& L = blk[bi];
      const int nn = L.n;
      size_t vt_off = 0, gt_off = 0;
      // reflector k has its unit at row k + sh: k + 1 after the one-stage reduction, k + kBand
      // after the first stage of the two-stage one; nn - 1 - sh reflectors
      const int sh = shift[bi], nrefl = nn - 1 - sh;
      for (int p = 0; p < L.npanel; p++) {
        const int k0 = p * NBT, pnb = std::min(NBT, nrefl - k0), K = nn - k0 - sh;
        panels.push_back(PanelRef{bi, k0, pnb, 0, (long long)gt_off});
        double* Gp = L.GT + gt_off;                 // pnb x pnb
        double* Tp = Gp + (size_t)pnb * pnb;        // pnb x pnb
        gt_off += 2 * (size_t)pnb * pnb;
        const double* Vrows = L.W1 + (size_t)k0 * L.ldp + k0 + sh;  // pnb x K, row q = v_{k0+q}
        gram.add_out(Gp, pnb, pnb, pnb, 0.0);
        gram.add_seg(Vrows, L.ldp, 0, Vrows, L.ldp, 1, K, 1.0);
        double* VTp = L.H + vt_off;  // K x pnb (H is free after the final row permutation)
        vt_off += (size_t)K * pnb;
        if (vt_off > (size_t)nn * nn) return fail(NRG_ERR_ARG, "internal: VT factors exceed H for n=%d", nn);
        vt.add_out(VTp, pnb, K, pnb, 0.0);
        vt.add_seg(Vrows, L.ldp, 1, Tp, pnb, 0, pnb, 1.0);
        // step index counts from the last panel of each block
        const int stp = L.npanel - 1 - p;
        GemmPlan& g1 = bsteps[2 * stp];
        GemmPlan& g2 = bsteps[2 * stp + 1];
        double* Wb = L.W2;  // n x pnb
        g1.add_out(Wb, pnb, nn, pnb, 0.0);
        g1.add_seg(L.evecs + k0 + sh, nn, 0, Vrows, L.ldp, 1, K, 1.0);
        g2.add_out(L.evecs + k0 + sh, nn, nn, K, 1.0);
        g2.add_seg(Wb, pnb, 0, VTp, pnb, 1, pnb, -1.0);
      }
    }
    const size_t pan_off = push(img, panels);
    // two-stage blocks: per stage-1 panel j0 = p kBand, the blocks with more than one row below
    // the band (a prefix: sorted by order), six GEMMs of the trailing update in compact-WY form
    //   X = S22 V, Y = X T1, Z = V^T Y, U = T1^T Z, W = Y - V U / 2, S22 -= V W^T + W V^T
    const size_t bblk_off = push(img, bblk);
    int npan1 = 0;
    for (const BandBlock& Bb : bblk) npan1 = std::max(npan1, Bb.jfin / kBand);
    std::vector<int> pan_active(npan1, 0);
    std::vector<StagedGemm> s1_g((size_t)npan1 * 6);
    for (int p = 0; p < npan1; p++) {
      const int j0 = p * kBand;
      GemmPlan ga, gb, gc, gd, ge, gf;
      for (const BandBlock& Bb : bblk) {
        const int nn = Bb.n, m = nn - j0 - kBand;
        if (m <= 1) break;
        pan_active[p]++;
        const int kb = std::min(kBand, m - 1);
        double* S22 = Bb.S + (size_t)(j0 + kBand) * Bb.lds + j0 + kBand;
        const double* Vt = Bb.S + (size_t)j0 * Bb.lds + j0 + kBand;  // kb x m
        double* Y = Bb.scr + band_scr_y(nn);
        double* T1 = Bb.scr + band_scr_t(nn);
        double* U = Bb.scr + band_scr_u(nn);
        const int ns = band_split(m), chunk = (m + ns - 1) / ns;
        // X = S22 V and Z = V^T Y in parts along m (rows k0 .. k1 of V), summed as segments
        for (int q = 0; q < ns; q++) {
          const int k0 = q * chunk, k1 = std::min(m, k0 + chunk);
          if (k1 <= k0) break;
          double* Xq = Bb.scr + band_scr_x(nn, q);
          ga.add_out(Xq, kBand, m, kb, 0.0);
          ga.add_seg(S22 + k0, Bb.lds, 0, Vt + k0, Bb.lds, 1, k1 - k0, 1.0);
        }
        gb.add_out(Y, kBand, m, kb, 0.0);
        for (int q = 0; q < ns; q++) {
          if (q * chunk >= m) break;
          gb.add_seg(Bb.scr + band_scr_x(nn, q), kBand, 0, T1, kBand, 0, kb, 1.0);
        }
        for (int q = 0; q < ns; q++) {
          const int k0 = q * chunk, k1 = std::min(m, k0 + chunk);
          if (k1 <= k0) break;
          gc.add_out(Bb.scr + band_scr_z(nn, q), kBand, kb, kb, 0.0);
          gc.add_seg(Vt + k0, Bb.lds, 0, Y + (size_t)k0 * kBand, kBand, 0, k1 - k0, 1.0);
        }
        gd.add_out(U, kBand, kb, kb, 0.0);
        for (int q = 0; q < ns; q++) {
          if (q * chunk >= m) break;
          gd.add_seg(T1, kBand, 1, Bb.scr + band_scr_z(nn, q), kBand, 0, kb, 1.0);
        }
        ge.add_out(Y, kBand, m, kb, 1.0);
        ge.add_seg(Vt, Bb.lds, 1, U, kBand, 0, kb, -0.5);
        gf.add_out(S22, Bb.lds, m, m, 1.0);
        gf.add_seg(Vt, Bb.lds, 1, Y, kBand, 1, kb, -1.0);
        gf.add_seg(Y, kBand, 0, Vt, Bb.lds, 0, kb, -1.0);
      }
      s1_g[6 * p + 0] = stage_gemm(img, ga);
      s1_g[6 * p + 1] = stage_gemm(img, gb);
      s1_g[6 * p + 2] = stage_gemm(img, gc);
      s1_g[6 * p + 3] = stage_gemm(img, gd);
      s1_g[6 * p + 4] = stage_gemm(img, ge);
      s1_g[6 * p + 5] = stage_gemm(img, gf);
    }
    const StagedGemm gram_g = stage_gemm(img, gram), vt_g = stage_gemm(img, vt);
    std::vector<StagedGemm> bs_g(bsteps.size());
    for (size_t t = 0; t < bsteps.size(); t++) bs_g[t] = stage_gemm(img, bsteps[t]);
    // room for the grid reduction's groups, jobs and barrier counters (filled when planned)
    const size_t grid_off = push(img, std::vector<char>(160 * (sizeof(GridGroup) + 128) + sizeof(int) * (size_t)nb + 1024));
    rc = stage_desc(c, img, s);
    if (rc) return rc;
    char* dbase = static_cast<char*>(c->desc);
    const LargeBlock* dblk = reinterpret_cast<const LargeBlock*>(dbase + blk_off);
    const BandBlock* dbb = reinterpret_cast<const BandBlock*>(dbase + bblk_off);

    // ---- 1a. two-stage reduction of the largest blocks (when few): symmetric copy, stage-1
    //          panels and their GEMMs, bulge chasing, the T factors of its back-transform.
    //          With one-stage blocks beside them it runs on the context's fourth stream, so
    //          that the one-stage reductions fill the SMs its clusters leave idle.
    const bool fork3 = nts > 0 && nts < nb;
    cudaStream_t s3 = s;
    SideStreams two_stage(s);
    if (fork3) {
      if (!c->side3) {
        NRG_CK(cudaStreamCreateWithFlags(&c->side3, cudaStreamNonBlocking));
        NRG_CK(cudaEventCreateWithFlags(&c->fork3_ev, cudaEventDisableTiming));
        NRG_CK(cudaEventCreateWithFlags(&c->join3_ev, cudaEventDisableTiming));
      }
      NRG_CK(cudaEventRecord(c->fork3_ev, s));
      NRG_CK(cudaStreamWaitEvent(c->side3, c->fork3_ev, 0));
      s3 = c->side3;
      two_stage.add(s3, c->join3_ev);
    }
    if (nts > 0) {
      for (const BandBlock& Bb : bblk)
        NRG_CK(cudaMemsetAsync(Bb.BND, 0, sizeof(double) * (size_t)Bb.n * kLDB, s3));
      {
        PhaseScope ps(c, kPhBandReduce, s3);
        NRG_CK(band_sym_launch(dbb, nts, blk[0].n, s3));
      }
      for (int p = 0; p < npan1; p++) {
        {
          PhaseScope ps(c, kPhBandPanel, s3);
          NRG_CK(band_panel_launch(dbb, pan_active[p], p * kBand, bblk[0].n - p * kBand - kBand, s3));
        }
        for (int q = 0; q < 6; q++) {
          rc = launch_staged_gemm(c, s1_g[6 * p + q], s3, kPhBandReduce);
          if (rc) return rc;
        }
      }
      {
        PhaseScope ps(c, kPhBulgeChase, s3, 2);
        NRG_CK(band_chase_launch(dbb, nts, s3));
        NRG_CK(band_q2_tfactor_launch(dbb, nts, blk[0].n, s3));
      }
    }

    // ---- 1. tridiagonalisation, split by reduction_plan: blocks sorted by falling order go to the groups
    //         of CTAs, then to the clusters, the streaming kernel and the one-CTA kernel
    {
      int nsm = 148;
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device);
      // the one-stage reductions: the blocks after the two-stage ones
      const LargeBlock* b1 = blk.data() + nts;
      const LargeBlock* d1 = dblk + nts;
      const int nb1 = nb - nts;
      int smsm = 0;
      NRG_CK(cudaDeviceGetAttribute(&smsm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, c->device));
      const ReductionPlan rp = reduction_plan(b1, nb1, std::min(cluster_max_n, dsm_max_order()), mid_max_n, nsm, smsm,
                                              c->tune.reduction_ctas_per_sm > 1);
      const int ngrid = rp.ngrid, nstream = rp.mid - rp.cut;
      // Launches that can run side by side go to streams of their own: the groups of the largest blocks on
      // s, then each cluster size, the streaming kernel and the one-CTA kernels beside them,
      // largest first (clusters need SMs of one GPC free at once).
      struct Launch { int C, q0, q1; };  // C = 0: tridiag_smem_kernel, -1: tridiag_kernel
      std::vector<Launch> ls;
      for (int C = 16; C >= 0; C = C > 1 ? C / 2 : C - 1) {
        if (C == 1 && nstream > 0) ls.push_back({-1, rp.cut, rp.mid});
        for (int q0 = ngrid, q1; q0 < nb1; q0 = q1) {
          if (q0 >= rp.cut && q0 < rp.mid) {
            q1 = rp.mid;
            continue;
          }
          for (q1 = q0 + 1; q1 < nb1 && q1 != rp.cut && rp.C[q1] == rp.C[q0]; q1++) {}
          if (rp.C[q0] == C) ls.push_back({C, q0, q1});
        }
      }
      const bool fork = ls.size() + (ngrid > 0) > 1;
      if (fork) {
        rc = tri_streams(c);
        if (rc) return rc;
        NRG_CK(cudaEventRecord(c->tri_fork, s));
      }
      PhaseScope ps(c, kPhTridiag, s, (ngrid > 0 ? 2 : 0) + (nstream > 0 ? 1 : 0) + (int)ls.size());
      unsigned used = 0;  // side streams with a launch
      SideStreams sides(s);
      if (ngrid > 0) {
        const GridPlan gp = grid_plan(b1, ngrid, rp.nsm_grid);
        pack_full_kernel<<<dim3((b1[0].ldp + 31) / 32, (b1[0].n + 31) / 32, ngrid), 256, 0, s>>>(d1);
        NRG_CK(cudaGetLastError());
        std::vector<char> gi;
        const size_t go = push(gi, gp.groups), jo = push(gi, gp.jobs),
                     co = push(gi, std::vector<unsigned>(32 * gp.groups.size(), 0u));
        if (grid_off + gi.size() > c->desc_size) return fail(NRG_ERR_ARG, "internal: grid descriptors");
        char* gb = dbase + grid_off;
        NRG_CK(cudaMemcpyAsync(gb, gi.data(), gi.size(), cudaMemcpyHostToDevice, s));
        const void* fn = b1[0].n <= 8 * kGridThreads ? (const void*)tridiag_grid_kernel<8> : (const void*)tridiag_grid_kernel<20>;
        NRG_CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gp.smem));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)gp.ctas);
        cfg.blockDim = dim3(kGridThreads);
        cfg.dynamicSmemBytes = gp.smem;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;  // the groups' barriers need all CTAs resident
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        const LargeBlock* db = d1;
        const GridGroup* dg = reinterpret_cast<const GridGroup*>(gb + go);
        int ng = (int)gp.groups.size();
        const int* dj = reinterpret_cast<const int*>(gb + jo);
        unsigned* dc = reinterpret_cast<unsigned*>(gb + co);
        void* kargs[] = {(void*)&db, (void*)&dg, (void*)&ng, (void*)&dj, (void*)&dc};
        NRG_CK(cudaLaunchKernelExC(&cfg, fn, kargs));
      }
      for (size_t q = 0; q < ls.size(); q++) {
        cudaStream_t ss = s;
        const size_t side = q + (ngrid > 0);  // 0: stream s
        if (side > 0) {
          const int i = (int)(side - 1) % nrg_ctx::kTriStreams;
          ss = c->tri[i];
          if (!(used >> i & 1)) {
            NRG_CK(cudaStreamWaitEvent(ss, c->tri_fork, 0));
            sides.add(ss, c->tri_join[i]);
          }
          used |= 1u << i;
        }
        const LargeBlock* dq = d1 + ls[q].q0;
        const int nq = b1[ls[q].q0].n, count = ls[q].q1 - ls[q].q0;
        if (ls[q].C < 0) {
          const int ny = tri_copies(nq, smsm);
          const size_t smem = tri_smem(nq, ny);
          pack_lower_kernel<<<dim3((nq + 7) / 8, count), 256, 0, ss>>>(dq);
          NRG_CK(cudaGetLastError());
          NRG_CK(cudaFuncSetAttribute(tridiag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
          tridiag_kernel<<<count, kTriThreads, smem, ss>>>(
              dq, reinterpret_cast<const CUtensorMap*>(dbase + tmap_off) + nts + ls[q].q0, ny);
          NRG_CK(cudaGetLastError());
        } else {
          NRG_CK(reduce_in_smem_launch(dq, nq, count, ls[q].C, ss));
        }
      }
      if (beside && pos == 0) {  // the small-block solver takes what SMs are left
        rc = beside();
        if (rc) return rc;
      }
      NRG_CK(sides.join());
    }
    NRG_CK(two_stage.join());  // all blocks are tridiagonal
    // ---- 2. divide and conquer
    {
      PhaseScope ps(c, kPhDcLeaf, s);
      const size_t ls = sizeof(double) * 2 * (kLeaf * kLeafLd + kLeaf) + dc_scratch_bytes(kLeaf);
      NRG_CK(cudaFuncSetAttribute(dc_leaf_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ls));
      dc_leaf_kernel<<<(int)leaves.size(), kCtaEigThreads, ls, s>>>(dblk, reinterpret_cast<const DcLeaf*>(dbase + leaf_off));
      NRG_CK(cudaGetLastError());
    }
    for (size_t h = 0; h < levels.size(); h++) {
      int maxN = 0;
      for (auto& nd : levels[h]) maxN = std::max(maxN, nd.b - nd.a);
      const int nn = (int)levels[h].size();
      const DcNode* dn = reinterpret_cast<const DcNode*>(dbase + node_off[h]);
      DcState* dst = reinterpret_cast<DcState*>(dbase + st_off[h]);
      GemmOut* go = reinterpret_cast<GemmOut*>(dbase + lvl_gemm[h].outs_off);
      GemmSeg* gs = reinterpret_cast<GemmSeg*>(dbase + lvl_gemm[h].segs_off);
      // shared memory for the largest node that fits it; larger nodes use global scratch
      size_t ps = 16;
      for (auto& nd : levels[h]) {
        const size_t t = prep_layout(nd.b - nd.a).total;
        if (t <= kPrepSmemMax) ps = std::max(ps, t);
      }
      NRG_CK(cudaFuncSetAttribute(dc_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ps));
      {
        PhaseScope sc(c, kPhDcPrep, s);
        dc_prep_kernel<<<nn, maxN <= 128 ? 128 : maxN <= 512 ? 256 : 512, ps, s>>>(dblk, dn, dst, go, gs, ps);
        NRG_CK(cudaGetLastError());
      }
      // one warp per root (8 per CTA), at most 256 CTAs per node, and a CTA per slab of the rows
      const int ysec = std::max(1, std::min(256, (maxN + 7) / 8)), ymove = (maxN + kMoveCols - 1) / kMoveCols;
      {
        PhaseScope sc(c, kPhDcSecular, s);
        dc_secular_kernel<<<dim3(nn, ysec + ymove), 256, 0, s>>>(dblk, dn, dst, ysec);
        NRG_CK(cudaGetLastError());
      }
      {
        PhaseScope sc(c, kPhDcVectors, s, 2);
        dc_zhat_kernel<<<dim3(nn, (maxN + 31) / 32), 256, 0, s>>>(dblk, dn, dst);
        NRG_CK(cudaGetLastError());
        dc_vectors_kernel<<<dim3(nn, ysec), 256, 0, s>>>(dblk, dn, dst);
        NRG_CK(cudaGetLastError());
      }
      rc = launch_staged_gemm(c, lvl_gemm[h], s, kPhDcGemm);
      if (rc) return rc;
    }
    // ---- 3. order
    {
      int P = 1;
      while (P < maxn) P <<= 1;
      const size_t ss = (sizeof(double) + sizeof(int)) * (size_t)P;
      NRG_CK(cudaFuncSetAttribute(sort_final_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ss));
      PhaseScope sc(c, kPhSort, s, 2);
      sort_final_kernel<<<nb, 1024, ss, s>>>(dblk);
      NRG_CK(cudaGetLastError());
      permute_rows_kernel<<<dim3((maxn + 7) / 8, nb), 256, 0, s>>>(dblk);
      NRG_CK(cudaGetLastError());
    }
    // ---- 3a. two-stage blocks: the bulge-chasing reflectors applied to the eigenvector rows
    if (nts > 0) {
      PhaseScope sc(c, kPhBtBand, s);
      NRG_CK(band_q2_apply_launch(dbb, nts, blk[0].n, s));
    }
    // ---- 4. back-transform
    rc = launch_staged_gemm(c, gram_g, s, kPhBtGemm);
    if (rc) return rc;
    if (!panels.empty()) {
      PhaseScope sc(c, kPhBtTfactor, s);
      const size_t ts = sizeof(double) * ((size_t)NBT * kTfLd + (size_t)(NBT / 2) * kTfLx);
      NRG_CK(cudaFuncSetAttribute(tfactor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ts));
      tfactor_kernel<<<(int)panels.size(), kTfThreads, ts, s>>>(dblk, reinterpret_cast<const PanelRef*>(dbase + pan_off));
      NRG_CK(cudaGetLastError());
    }
    rc = launch_staged_gemm(c, vt_g, s, kPhBtGemm);
    if (rc) return rc;
    for (size_t t = 0; t < bs_g.size(); t++) {
      rc = launch_staged_gemm(c, bs_g[t], s, kPhBtGemm);
      if (rc) return rc;
    }
    pos = end;
    if (pos < ord.size()) NRG_CK(cudaStreamSynchronize(s));  // the next chunk reuses the workspace
  }
  return NRG_OK;
}

}  // namespace nrg
