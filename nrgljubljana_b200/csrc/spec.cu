// spec.cu -- fused spectral-weight + log-grid binning kernel, and the Matsubara sums.
//
// Replaces the per-term loops of Algo_DMNRG::calc (c++/algo_DMNRG.hpp:29-52) and
// Algo_FDMgt/Algo_FDMls::calc (c++/algo_FDM.hpp:84-114, 30-60) together with
// ChainBinning::add (c++/spectrum.hpp:19-28) and Bins::add/add_std (c++/bins.hpp:103-132).
// The O(k^3) inner sums of the DM-NRG loop and the prod_fit products of FDM are computed
// beforehand as GEMMs (X, Y); these kernels only form the weights and scatter them.
#include "common.cuh"
#include "spec.h"

#include <algorithm>

namespace nrg {
namespace {

constexpr int kThreads = 256;

struct Hist {
  double* pos;
  double* neg;
};

// The region that owns work item t (binary search over tile0).
NRG_DEV int find_region(const SpecRegion* __restrict__ regs, int nreg, int64_t t) {
  int lo = 0, hi = nreg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (regs[mid].tile0 <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// A lane's running sum of consecutive terms that fall between the same two bins.
struct Run {
  int key = -1;  // bin index, + nbins for the negative half; -1: nothing pending
  double lo = 0.0, hi = 0.0;
};

NRG_DEV void run_flush(Run& a, const Hist& h, int nbins) {
  if (a.key >= 0) {
    double* b = a.key < nbins ? h.pos + a.key : h.neg + (a.key - nbins);
    if (a.lo != 0.0) atomicAdd(b, a.lo);
    if (a.hi != 0.0) atomicAdd(b + 1, a.hi);
  }
  a.key = -1;
}

// Bins::add (bins.hpp:103-110) + add_std (bins.hpp:112-132) + ChainBinning::add
// (spectrum.hpp:19-24), for a real weight, into the lane's running sum.
NRG_DEV void bin_add(Run& a, const Hist& h, const BinParams& bp, double energy, double w) {
  if (w == 0.0) return;  // adding an exact zero changes no bin
  const double e = fabs(energy);
  if (fabs(w) < bp.discard_immediately * e) return;
  int idx = 0;
  double lo = w, hi = 0.0;
  if (!(e < 1e-14)) {
    const double x = (log10(e) - bp.log10emin) * bp.bins;
    const double ip = floor(x);
    if (ip < 0.0) {
      idx = 0;
    } else if (ip >= (double)(bp.nbins - 1)) {
      idx = bp.nbins - 1;
    } else {
      idx = (int)ip;
      const double rem = x - ip;
      lo = (1.0 - rem) * w;
      hi = rem * w;
    }
  }
  const int key = (energy >= 0.0) ? idx : idx + bp.nbins;
  if (key == a.key) {
    a.lo += lo;
    a.hi += hi;
    return;
  }
  run_flush(a, h, bp.nbins);
  a.key = key;
  a.lo = lo;
  a.hi = hi;
}

// One warp tile: columns i0 + 32 ti .., `rows` rows from j0 + rows tj. A lane keeps one column
// and walks down the rows, U of whose operands it loads together.
template <int KIND, int U>
NRG_DEV void bin_tile(const SpecRegion& r, const Hist& h, const BinParams& bp, int ib, int jb, int jn) {
  const int lane = threadIdx.x & 31;
  const int i = ib + lane;
  const bool act = i < r.i1;
  const double ei = act ? r.Ei[i] : 0.0;
  const double xi = (KIND == kSpecExpI && act) ? exp(-ei / r.T) : 0.0;
  Run run;
  const bool XY = KIND == kSpecDMNRG || KIND == kSpecGemmX;
  const double* p1 = r.op1 + (int64_t)jb * r.ld1 + i;
  const double* p2 = KIND != kSpecGemmX ? r.op2 + (int64_t)jb * r.ld2 + i : nullptr;
  const double* px = XY ? r.X + (int64_t)(jb - r.j0) * r.ldx + (i - r.i0) : nullptr;
  const double* py = KIND == kSpecDMNRG ? r.Y + (int64_t)(jb - r.j0) * r.ldy + (i - r.i0) : nullptr;
  for (int g = 0; g < jn; g += 32) {
    const int cnt = min(32, jn - g);
    const double ejl = lane < cnt ? r.Ej[jb + g + lane] : 0.0;
    const double xjl = (KIND == kSpecExpJ && lane < cnt) ? exp(-ejl / r.T) : 0.0;
    for (int q = 0; q < cnt; q += U) {
      double en[U], o1[U], o2[U], x[U], y[U], xj[U];
      bool ok[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int row = min(q + u, 31);
        en[u] = __shfl_sync(0xffffffffu, ejl, row) - ei;
        xj[u] = KIND == kSpecExpJ ? __shfl_sync(0xffffffffu, xjl, row) : 0.0;
        ok[u] = act && q + u < cnt;
        if (KIND == kSpecDMNRG) ok[u] = ok[u] && !(fabs(en[u]) < r.Emin || fabs(en[u]) > r.Emax);
        o1[u] = ok[u] ? p1[u * r.ld1] : 0.0;
        o2[u] = (KIND != kSpecGemmX && ok[u]) ? p2[u * r.ld2] : 0.0;
        if (XY) x[u] = ok[u] ? px[u * r.ldx] : 0.0;
        if (KIND == kSpecDMNRG) y[u] = ok[u] ? py[u * r.ldy] : 0.0;
      }
      p1 += U * r.ld1;
      if (KIND != kSpecGemmX) p2 += U * r.ld2;
      if (XY) px += U * r.ldx;
      if (KIND == kSpecDMNRG) py += U * r.ldy;
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (!ok[u]) continue;
        double w;
        if (KIND == kSpecDMNRG) w = x[u] * o1[u] + (double)(-r.sign) * (y[u] * o2[u]);
        else if (KIND == kSpecExpI) w = o1[u] * o2[u] * r.coef * xi;
        else if (KIND == kSpecExpJ) w = o1[u] * o2[u] * r.coef * xj[u];
        else w = o1[u] * x[u] * r.coef;
        bin_add(run, h, bp, en[u], r.factor * w);
      }
    }
  }
  // The lanes' last runs, summed across the warp for the bins that many lanes share (coarse
  // grids: neighbouring columns have neighbouring energies), one by one for the rest.
#pragma unroll 1
  for (int it = 0; it < 3; it++) {
    const unsigned live = __ballot_sync(0xffffffffu, run.key >= 0);
    if (live == 0) return;
    const int key = __shfl_sync(0xffffffffu, run.key, __ffs(live) - 1);
    const bool mine = run.key == key;
    if (__popc(__ballot_sync(0xffffffffu, mine)) < 4) break;
    const double lo = warp_sum(mine ? run.lo : 0.0), hi = warp_sum(mine ? run.hi : 0.0);
    if (mine) run.key = -1;
    if (lane == 0) {
      Run s;
      s.key = key;
      s.lo = lo;
      s.hi = hi;
      run_flush(s, h, bp.nbins);
    }
  }
  run_flush(run, h, bp.nbins);
}

// FP64 atomics on shared memory are compare-and-swap loops, so what bounds a scatter kernel is
// the number of atomics and how many lanes meet at one bin, not the operands' bytes. A lane
// walks down a column: its energies Ej - Ei grow with j (both sorted), so consecutive terms
// mostly fall between the same two bins and are summed in registers; an atomic goes out when
// the bin changes. exp(-E/T) is taken once per row or column of a tile, not per term. Every CTA
// keeps both halves of the histogram in shared memory when they fit and stays for many tiles
// (one flush of its non-zero bins at the end); larger grids take FP64 atomics in L2.
// Measured on B200, both FDM parts of 12 subspaces of order 800-2000 (36 million terms, 10 bins a
// decade, whole call with its GEMMs): 2643 us with one atomic pair per term and a 64-bit division
// for the indices, 628 us so; a DM-NRG call of 40 subspaces up to order 192 on 1000 bins a decade
// 76 and 36 us. What is left is the latency of a term's chain (a logarithm, 200 instructions): the FDM
// kernel runs at four CTAs per SM with two rows loaded together (its launches 0.38 ms, 0.50 at two
// CTAs and four rows, 0.42 at four and four), DM-NRG's short launch at two and four (16 us, 19).
// DM: all regions are of DM-NRG (kSpecDMNRG), otherwise none is.
template <bool DM>
__global__ void __launch_bounds__(kThreads, DM ? 2 : 4) spec_bin_kernel(const SpecRegion* __restrict__ regs, int nreg,
                                                                        int64_t ntiles, int rows, BinParams bp,
                                                                        double* gpos, double* gneg, int use_smem) {
  extern __shared__ __align__(16) double sh[];
  Hist h{gpos, gneg};
  if (use_smem) {
    for (int i = threadIdx.x; i < 2 * bp.nbins; i += blockDim.x) sh[i] = 0.0;
    __syncthreads();
    h.pos = sh;
    h.neg = sh + bp.nbins;
  }
  const int nw = kThreads / 32;
  for (int64_t t = (int64_t)blockIdx.x * nw + (threadIdx.x >> 5); t < ntiles; t += (int64_t)gridDim.x * nw) {
    const SpecRegion r = regs[find_region(regs, nreg, t)];
    const int lt = (int)(t - r.tile0), ti = (r.i1 - r.i0 + 31) / 32;
    const int ib = r.i0 + 32 * (lt % ti), jb = r.j0 + rows * (lt / ti), jn = min(rows, r.j1 - jb);
    if (DM) {
      bin_tile<kSpecDMNRG, 4>(r, h, bp, ib, jb, jn);
    } else {
      switch (r.kind) {
        case kSpecExpI: bin_tile<kSpecExpI, 2>(r, h, bp, ib, jb, jn); break;
        case kSpecExpJ: bin_tile<kSpecExpJ, 2>(r, h, bp, ib, jb, jn); break;
        default: bin_tile<kSpecGemmX, 2>(r, h, bp, ib, jb, jn); break;
      }
    }
    __syncwarp();
  }
  if (use_smem) {
    __syncthreads();
    for (int i = threadIdx.x; i < bp.nbins; i += blockDim.x) {
      if (sh[i] != 0.0) atomicAdd(gpos + i, sh[i]);
      if (sh[bp.nbins + i] != 0.0) atomicAdd(gneg + i, sh[bp.nbins + i]);
    }
  }
}

// ---------------------------------------------------------------- Matsubara sums
// Algo_FDMmats, Algo_FTmats, Algo_DMNRGmats (c++/algo_FDM.hpp:167-217, c++/algo_FT.hpp:63-85,
// c++/algo_DMNRG.hpp:76-100) into ChainMatsubara (c++/spectrum.hpp:34-42): every
// term adds factor w / (i w_n - E) = factor w (-E - i w_n) / (E^2 + w_n^2) to point n, n < mats.
constexpr int kMatsTerms = kMatsChunk / kThreads;  // terms of a thread

// The weight of term (i, j) without `factor`, and the value that replaces it at n = 0 (see
// MatsSpecial); false for a DM-NRG term outside the energy window.
NRG_DEV bool mats_weight(const SpecRegion& r, int i, int j, double energy, double& w, double& v0) {
  const double o1 = r.op1[(int64_t)j * r.ld1 + i];
  const double o2 = r.kind != kSpecGemmX ? r.op2[(int64_t)j * r.ld2 + i] : 0.0;
  const int64_t xo = (int64_t)(j - r.j0) * r.ldx + (i - r.i0);
  v0 = 0.0;
  switch (r.kind) {
    case kSpecDMNRG: {
      if (fabs(energy) < r.Emin || fabs(energy) > r.Emax) return false;
      const double a = r.X[xo] * o1;
      w = a + (double)(-r.sign) * (r.Y[(int64_t)(j - r.j0) * r.ldy + (i - r.i0)] * o2);
      v0 = -a / r.T;
      return true;
    }
    case kSpecExpIJ: {
      const double a = o1 * o2 * r.coef * exp(-r.Ei[i] / r.T), b = o1 * o2 * r.coef2 * exp(-r.Ej[j] / r.T);
      w = a + b;
      v0 = (r.mspecial == kMatsFtB ? b : -a) / r.T;
      return true;
    }
    case kSpecExpIX:
      w = o1 * o2 * r.coef * exp(-r.Ei[i] / r.T) + o1 * r.X[xo] * r.coef2;
      return true;
    default:  // kSpecXExpJ
      w = o1 * r.X[xo] * r.coef + o1 * o2 * r.coef2 * exp(-r.Ej[j] / r.T);
      return true;
  }
}

// Sum over the warp of x[c] for c = (lane >> 2) & 7, in every lane (9 shuffles).
NRG_DEV double warp_sum8(double (&x)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 4, o = 16; s >= 1; s >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int q = 0; q < s; q++) {
      const double send = up ? x[q] : x[q + s];
      const double keep = up ? x[q + s] : x[q];
      x[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  x[0] += __shfl_xor_sync(0xffffffffu, x[0], 2);
  x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
  return x[0];
}

// FP64-bound: about ten FP64 instructions per (term, point), one reciprocal among them. A thread
// holds its terms (E, w) in registers and walks over the points four at a time, so a point's
// sum is formed in registers over a thread's terms, then across the warp by shuffles; only that
// warp sum goes to the CTA's copy of the points by an atomic (8 lanes, 8 addresses), and the
// copy to memory at the end. The two exponential parts of a term are added before the
// division. Measured on B200 (40 subspaces up to order 480, 100 points, whole call): 165 us;
// with one pair of shared-memory atomics per (term, point), all threads of a CTA at the same
// address, 8330 us.
__global__ void __launch_bounds__(kThreads) spec_mats_kernel(const SpecRegion* __restrict__ regs, int nreg,
                                                             int64_t nchunks, MatsParams mp, double* gre,
                                                             double* gim) {
  extern __shared__ __align__(16) double sh[];
  double* re = sh;
  double* im = sh + mp.mats;
  for (int n = threadIdx.x; n < 2 * mp.mats; n += blockDim.x) sh[n] = 0.0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const double pt = 3.14159265358979323846 * mp.T;
  for (int64_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
    const SpecRegion r = regs[find_region(regs, nreg, ch)];
    const int wi = r.i1 - r.i0;
    const int64_t t0 = (ch - r.tile0) * (int64_t)kMatsChunk, tn = (int64_t)wi * (r.j1 - r.j0);
    const int jq = (int)(t0 / wi);
    const unsigned iq = (unsigned)(t0 % wi);
    double e[kMatsTerms], w[kMatsTerms], v0[kMatsTerms];
#pragma unroll
    for (int k = 0; k < kMatsTerms; k++) {
      const unsigned o = (unsigned)threadIdx.x + (unsigned)k * kThreads;
      e[k] = 1.0;  // no term: adds zero to every point
      w[k] = v0[k] = 0.0;
      if (t0 + o < tn) {
        const int j = r.j0 + jq + (int)((iq + o) / (unsigned)wi), i = r.i0 + (int)((iq + o) % (unsigned)wi);
        const double energy = r.Ej[j] - r.Ei[i];
        double wk, vk;
        if (mats_weight(r, i, j, energy, wk, vk)) {
          e[k] = energy;
          w[k] = r.factor * wk;
          v0[k] = r.factor * vk;
        }
      }
    }
    for (int n0 = 0; n0 < mp.mats; n0 += 4) {
      double acc[8];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int n = n0 + q;
        const double wn = pt * (double)(mp.bosonic ? 2 * n : 2 * n + 1);
        double sr = 0.0, si = 0.0;
        if (n == 0 && mp.bosonic) {  // w_0 = 0: the denominator is E^2, whose reciprocal E may put out of range
#pragma unroll
          for (int k = 0; k < kMatsTerms; k++) {
            if (r.mspecial != kMatsPlain && fabs(e[k]) <= 1e-8) {
              sr += v0[k];
            } else {
              const double d = e[k] * e[k];
              sr -= w[k] * e[k] / d;
              si -= w[k] * wn / d;
            }
          }
        } else {
#pragma unroll
          for (int k = 0; k < kMatsTerms; k++) {
            const double t = w[k] * (1.0 / fma(e[k], e[k], wn * wn));
            sr = fma(-t, e[k], sr);
            si = fma(-t, wn, si);
          }
        }
        acc[2 * q] = sr;
        acc[2 * q + 1] = si;
      }
      const double s = warp_sum8(acc);
      const int c = lane >> 2, n = n0 + (c >> 1);
      if ((lane & 3) == 0 && n < mp.mats && s != 0.0) atomicAdd((c & 1 ? im : re) + n, s);
    }
  }
  __syncthreads();
  for (int n = threadIdx.x; n < mp.mats; n += blockDim.x) {
    if (re[n] != 0.0) atomicAdd(gre + n, re[n]);
    if (im[n] != 0.0) atomicAdd(gim + n, im[n]);
  }
}

}  // namespace

cudaError_t spec_mats_launch(const SpecRegion* d_regs, int nreg, int64_t nchunks, const MatsParams& mp, double* re,
                             double* im, cudaStream_t stream) {
  if (nreg <= 0 || nchunks <= 0 || mp.mats <= 0) return cudaSuccess;
  const size_t smem = 2 * sizeof(double) * (size_t)mp.mats;
  if (smem > kSpecSmemMax) return cudaErrorInvalidValue;
  cudaError_t err =
      cudaFuncSetAttribute(spec_mats_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSpecSmemMax);
  if (err != cudaSuccess) return err;
  const int64_t grid = std::min<int64_t>(nchunks, 148 * 8);
  spec_mats_kernel<<<(unsigned)grid, kThreads, smem, stream>>>(d_regs, nreg, nchunks, mp, re, im);
  return cudaGetLastError();
}

// Long tiles make long runs (few atomics); short ones keep every SM busy: about 32 warps per
// SM over the call, between 8 and 64 rows.
int spec_tile_rows(int64_t terms) {
  const int64_t rows = terms / (32 * 148 * 32);
  return (int)std::min<int64_t>(64, std::max<int64_t>(8, (rows + 7) / 8 * 8));
}

cudaError_t spec_bin_launch(const SpecRegion* d_regs, int nreg, int64_t ntiles, int rows, const BinParams& bp,
                            double* pos, double* neg, bool dmnrg, cudaStream_t stream) {
  if (nreg <= 0 || ntiles <= 0) return cudaSuccess;
  const size_t smem = 2 * sizeof(double) * (size_t)bp.nbins;
  const int use_smem = smem <= kSpecSmemMax ? 1 : 0;
  const auto kernel = dmnrg ? spec_bin_kernel<true> : spec_bin_kernel<false>;
  if (use_smem) {
    cudaError_t err =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSpecSmemMax);
    if (err != cudaSuccess) return err;
  }
  const int64_t grid = std::min<int64_t>((ntiles + kThreads / 32 - 1) / (kThreads / 32), 148 * 6);
  kernel<<<(unsigned)grid, kThreads, use_smem ? smem : 0, stream>>>(d_regs, nreg, ntiles, rows, bp, pos, neg, use_smem);
  return cudaGetLastError();
}

}  // namespace nrg
