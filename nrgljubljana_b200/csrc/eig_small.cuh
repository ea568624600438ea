// eig_small.cuh -- the symmetric eigenproblem of one CTA: Householder tridiagonalisation of a matrix held
// in registers, divide and conquer of a tridiagonal matrix in shared memory (also the leaves of
// the large blocks' divide and conquer), and the back-transform of its eigenvectors.
//
// Everything here is bound by latency (orders up to 96, one CTA each), so the steps are laid out
// to have few barriers and short dependent chains: no chain like the implicit QL iteration's (order^2
// rotations of a square root and a division each, one after another), no loop whose loads wait
// for a branch.
#pragma once
#include "common.cuh"

namespace nrg {

// Threads T of a CTA, a template parameter: 256 for orders up to 96, or 64 for orders up to 16, in whose merges at
// most two nodes share a CTA (a node has whole warps).
constexpr int kCtaEigThreads = 256, kTinyEigThreads = 64, kTinyEigN = 16;
// The largest order for R and T.
__host__ __device__ constexpr int cta_eig_max(int R, int T) { return T == kTinyEigThreads ? kTinyEigN : 32 * R; }

// Scratch of smem_dc for order N: ten doubles and five ints per row.
__host__ __device__ inline size_t dc_scratch_bytes(int N) { return (10 * sizeof(double) + 5 * sizeof(int)) * (size_t)N; }

// Tangent of the rotation that zeroes the coupling apq of two diagonals whose difference is df, the smaller root:
// 2 a_pq / (df + sgn(df) sqrt(df^2 + 4 a_pq^2)). Couplings between equal diagonals may be of any size, down to
// the smallest denormal: the squares are formed in units in which they stay in range.
__host__ __device__ __forceinline__ double jacobi_tangent(double df, double apq) {
  const double up = fmax(fabs(df), fabs(apq)) < 1e-150 ? 0x1p1000 : 1.0, x = up * df, y = 2.0 * (up * apq);
  return copysign(y, copysign(1.0, df) * apq) / (fabs(x) + sqrt(fma(x, x, y * y)));
}

// Eigenvalues a[i][i] and eigenvectors (rows of v) of a symmetric matrix of order 4 by cyclic Jacobi
// rotations, one thread; of smaller orders with zero rows and columns (zero couplings are
// skipped). False if 30 sweeps did not converge (five or so do). A sweep begins with whether it has anything to
// do: the last one does not.
__host__ __device__ __forceinline__ bool jacobi4(double (&a)[4][4], double (&v)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) v[i][j] = i == j ? 1.0 : 0.0;
  auto active = [&](int p, int q) { return fabs(a[p][q]) > 0.5 * kEps * (fabs(a[p][p]) + fabs(a[q][q])); };
#pragma unroll 1
  for (int sweep = 0; sweep <= 30; sweep++) {
    if (!(active(0, 1) || active(2, 3) || active(0, 2) || active(1, 3) || active(0, 3) || active(1, 2))) return true;
#pragma unroll
    for (int g = 0; g < 6; g++) {  // (0,1) (2,3) (0,2) (1,3) (0,3) (1,2): pairs that overlap, without branches
      constexpr int P[6] = {0, 2, 0, 1, 0, 1}, Q[6] = {1, 3, 2, 3, 3, 2};
      const int p = P[g], q = Q[g];
      const double apq = a[p][q], df = a[q][q] - a[p][p];
      const bool act = active(p, q);
      const double tn = jacobi_tangent(df, apq);
      const double t = act ? tn : 0.0, c = act ? rsqrt(fma(t, t, 1.0)) : 1.0, s = t * c;
      a[p][p] = fma(-t, apq, a[p][p]);
      a[q][q] = fma(t, apq, a[q][q]);
      a[p][q] = act ? 0.0 : apq;
#pragma unroll
      for (int r = 0; r < 4; r++) {
        if (r != p && r != q) {
          double& x = r < p ? a[r][p] : a[p][r];
          double& y = r < q ? a[r][q] : a[q][r];
          const double xv = x, yv = y;
          x = c * xv - s * yv;
          y = s * xv + c * yv;
        }
        const double xv = v[p][r], yv = v[q][r];
        v[p][r] = c * xv - s * yv;
        v[q][r] = s * xv + c * yv;
      }
    }
  }
  return false;
}

// The step of the secular iteration: a two-pole rational model through the neighbouring poles, at
// del1 and del2 from the current point, that matches f and f' (dpsi from the poles up to the first,
// dphi from the rest): its root between the poles, or for the last root the one right of both.
// One division, whichever branch.
NRG_DEV double secular_step(double f, double dpsi, double dphi, double del1, double del2, bool last) {
  const double cc = f - del1 * dpsi - del2 * dphi;
  const double s1 = del1 * del1 * dpsi, s2 = del2 * del2 * dphi;
  const double A1 = cc * (del1 + del2) + s1 + s2;
  const double A0 = cc * del1 * del2 + s1 * del2 + s2 * del1;
  const double disc = sqrt(fabs(A1 * A1 - 4.0 * cc * A0));
  const bool direct = last ? A1 >= 0.0 : A1 <= 0.0;  // no cancellation in A1 -+ disc over 2 cc
  const double r = last ? disc : -disc;
  double num = direct ? A1 + r : 2.0 * A0, den = direct ? 2.0 * cc : A1 - r;
  if (cc == 0.0) {
    num = A0;
    den = A1;
  }
  return num / den;
}

// Start of an inner root, measured from the nearer pole: at the midpoint of the two poles the function is f
// and, without their residues z1 and z2, c, which is taken as constant.
NRG_DEV double secular_start(double f, double c, double gap, double z1, double z2) {
  const double A1 = (f >= 0.0 ? c * gap : -c * gap) + z1 + z2, A0 = f >= 0.0 ? z1 * gap : -z2 * gap;
  const double disc = sqrt(fabs(A1 * A1 - 4.0 * c * A0));
  const bool pos = A1 > 0.0;
  return (pos ? 2.0 * A0 : A1 - disc) / (pos ? A1 + disc : 2.0 * c);
}

// Rows of a merged node: row j < K becomes sum_k U[j][k] Z[srow[k]], row j >= K the old row srow[j]
// (columns 0..n-1, n <= 8 CT), in place: all threads of the CTA take the barriers. A warp of the
// node's nw has up to NU tile rows of eight, all their columns at once (independent DMMA chains).
template <int CT, int NU>
NRG_DEV void dc_rows(const double* U, double* Z, int ld, const int* srow, int n, int K, int wn, int nw) {
  const int lane = threadIdx.x & 31, fr = lane >> 2, fc = lane & 3;
  double acc[NU][CT][2];
#pragma unroll
  for (int q = 0; q < NU; q++) {
    const int r0 = 8 * (wn + q * nw), row = r0 + fr;
#pragma unroll
    for (int c = 0; c < CT; c++) acc[q][c][0] = acc[q][c][1] = 0.0;
    if (r0 < K) {
      const double* u = U + min(row, K - 1) * ld;
      for (int k = 0; k < K; k += 4) {
        const int kk = min(k + fc, K - 1);
        const double x = k + fc < K && row < K ? u[kk] : 0.0;
        const double* z = Z + srow[kk] * ld;
        double y[CT];
#pragma unroll
        for (int c = 0; c < CT; c++) y[c] = z[min(8 * c + fr, n - 1)];
#pragma unroll
        for (int c = 0; c < CT; c++) dmma884(acc[q][c][0], acc[q][c][1], x, y[c]);
      }
    }
    if (row >= K && row < n) {
      const double* z = Z + srow[row] * ld + 2 * fc;
#pragma unroll
      for (int c = 0; c < CT; c++)
#pragma unroll
        for (int h = 0; h < 2; h++)
          if (8 * c + 2 * fc + h < n) acc[q][c][h] = z[8 * c + h];
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NU; q++) {
    const int row = 8 * (wn + q * nw) + fr;
    if (row < n) {
      double* z = Z + row * ld + 2 * fc;
#pragma unroll
      for (int c = 0; c < CT; c++)
#pragma unroll
        for (int h = 0; h < 2; h++)
          if (8 * c + 2 * fc + h < n) z[8 * c + h] = acc[q][c][h];
    }
  }
}

// x, or zero and ok = false if it is not finite: poles are compared with one another to index memory.
NRG_DEV double finite_or_zero(double x, bool& ok) {
  if (isfinite(x)) return x;
  ok = false;
  return 0.0;
}

// Bounds of node p of the 2^depth nodes that halving [0, N) `depth` times gives.
NRG_DEV void dc_bounds(int p, int depth, int N, int& lo, int& hi) {
  lo = 0;
  hi = N;
  for (int b = depth - 1; b >= 0; b--) {
    const int mid = lo + (hi - lo) / 2;
    if (p >> b & 1) lo = mid; else hi = mid;
  }
}

// Eigenvalues (into d, unsorted) and eigenvectors (rows of Z, row stride ld) of the symmetric
// tridiagonal matrix (d, e) of order N <= 32 R by divide and conquer in shared memory, T threads.
// U: N x ld doubles, scr: dc_scratch_bytes(N), ctl: 10 ints. Returns 0, or > 0 if a leaf did not
// converge or something came out that is not finite (d and Z then hold no solution, but d no NaN).
// d and e must be finite.
// Up to 32 leaves of order <= 4 are solved by one thread each; up to eight nodes of a level are
// merged at once, 256 / nodes threads each, with the method of the large merges (eig_large.cu:
// rank-one tearing, deflation, secular roots, Gu-Eisenstat vectors): an order-64 problem takes
// four levels of some ten thousand cycles where its QL chain is 3500 rotations of 350 cycles.
// The problem is scaled by a power of two to order one, and each merge again, so the tolerances are
// relative.
template <int R, int T = kCtaEigThreads>
NRG_DEV int smem_dc(double* d, double* e, int N, double* Z, double* U, int ld, void* scr, int* ctl) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* key = static_cast<double*>(scr);  // poles, sorted
  double* zs = key + N;                     // z, in that order
  double* pole = zs + N;                    // the non-deflated ones
  double* zz = pole + N;
  double* org = zz + N;                     // root j = org[j] + tau[j]
  double* tau = org + N;
  double* lamn = tau + N;                   // the node's new eigenvalues
  double* zh = lamn + N;
  double* rc = zh + N;                      // deflation rotations
  double* rs = rc + N;
  int* sidx = reinterpret_cast<int*>(rs + N);
  int* srow = sidx + N;                     // row of Z behind entry t (deflated ones from K on)
  int* flag = srow + N;                     // deflated
  int* rp = flag + N;
  int* rj = rp + N;
  int* nrot = ctl;       // per node, 8
  int* status = ctl + 8;

  // scale (by scalbn: 2^-ex itself is out of range for the smallest and the largest norms)
  if (warp == 0) {
    double m = 0.0;
    for (int i = lane; i < N; i += 32) m = fmax(m, fmax(fabs(d[i]), i < N - 1 ? fabs(e[i]) : 0.0));
    m = warp_max(m);
    if (lane == 0) {
      ctl[9] = m > 0.0 ? ilogb(m) : 0;
      *status = 0;
    }
  }
  for (int i = tid; i < N * ld; i += T) Z[i] = 0.0;
  __syncthreads();
  const int ex = ctl[9];
  if (tid < N) {
    d[tid] = scalbn(d[tid], -ex);
    if (tid < N - 1) e[tid] = scalbn(e[tid], -ex);
    Z[tid * ld + tid] = 1.0;
  }
  const int L = N > 64 ? 5 : N > 32 ? 4 : N > 16 ? 3 : N > 8 ? 2 : N > 4 ? 1 : 0;  // leaves of order 2..4
  __syncthreads();
  if (N == 2) {  // one rotation
    if (tid == 0 && e[0] != 0.0) {
      const double t = jacobi_tangent(d[1] - d[0], e[0]), c = rsqrt(fma(t, t, 1.0)), s = t * c;
      d[0] = fma(-t, e[0], d[0]);
      d[1] = fma(t, e[0], d[1]);
      Z[0] = Z[ld + 1] = c;
      Z[1] = -s;
      Z[ld] = s;
    }
  } else if (tid < 1 << L) {  // leaf `tid`: rank-one tearing at its cuts, then Jacobi
    int lo, hi;
    dc_bounds(tid, L, N, lo, hi);
    double a[4][4], v[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const bool in = lo + i < hi && lo + j < hi;
        a[i][j] = !in ? 0.0 : i == j ? d[lo + i] : j == i + 1 ? e[lo + i] : 0.0;
        if (i == j && i == 0 && lo > 0) a[i][i] -= fabs(e[lo - 1]);
        if (i == j && lo + i == hi - 1 && hi < N) a[i][i] -= fabs(e[hi - 1]);
      }
    bool ok = jacobi4(a, v);
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (lo + i < hi) {
        d[lo + i] = finite_or_zero(a[i][i], ok);
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (lo + j < hi) Z[(lo + i) * ld + lo + j] = v[i][j];
      }
    if (!ok) atomicMax(status, lo + 1);
  }
  __syncthreads();

  // (a level of 16 nodes takes two rounds of eight)
  for (int lev = L - 1, rnd = 0; lev >= 0; rnd == 0 && lev == 4 ? rnd++ : (rnd = 0, lev--)) {
    const int nodes = lev > 3 ? 8 : 1 << lev;
    const int G = T / nodes, node = tid / G, gt = tid % G, wn = gt >> 5, nw = G >> 5;
    int lo, hi;
    dc_bounds(node + 8 * rnd, lev, N, lo, hi);
    const int mid = lo + (hi - lo) / 2, n = hi - lo;
    const double beta = e[mid - 1], rho0 = 2.0 * fabs(beta), sg = beta >= 0.0 ? 1.0 : -1.0;
    // poles in order (each thread counts the smaller ones), z beside them
    if (gt < n) {
      const double di = d[lo + gt];
      int rank = 0;
      for (int j = 0; j < n; j++) {
        const double dj = d[lo + j];
        rank += dj < di || (dj == di && j < gt);
      }
      const double* row = Z + (lo + gt) * ld;
      key[lo + rank] = di;
      sidx[lo + rank] = gt;
      zs[lo + rank] = (lo + gt < mid ? row[mid - 1] : sg * row[mid]) * 0.70710678118654752440;
    }
    if (gt == 0) nrot[node] = 0;
    __syncthreads();
    // deflation: every warp of the node looks at all its entries (lane, lane + 32, lane + 64)
    double zv[R], zmx = 0.0;
#pragma unroll
    for (int q = 0; q < R; q++) {
      zv[q] = lane + 32 * q < n ? zs[lo + lane + 32 * q] : 0.0;
      zmx = fmax(zmx, fabs(zv[q]));
    }
    zmx = warp_max(zmx);
    const double tol = 8.0 * kEps * fmax(fmax(fabs(key[lo]), fabs(key[hi - 1])), rho0 * zmx);
    unsigned live[R];
#pragma unroll
    for (int q = 0; q < R; q++)
      live[q] = __ballot_sync(0xffffffffu, lane + 32 * q < n && !(rho0 * fabs(zv[q]) <= tol));
    bool close = false;
#pragma unroll
    for (int q = 0; q < R; q++) {
      if (live[q] >> lane & 1) {
        int nx = -1;  // next live entry
        unsigned m = live[q] & ~((2u << lane) - 1u);
#pragma unroll
        for (int u = q; u < R; u++) {
          if (u > q) m = live[u];
          if (nx < 0 && m) nx = 32 * u + __ffs(m) - 1;
        }
        if (nx >= 0) {
          const double zj = zs[lo + nx], t = hypot(zv[q], zj);
          close |= fabs((key[lo + nx] - key[lo + lane + 32 * q]) * (zj / t) * (zv[q] / t)) <= tol;
        }
      }
      if (wn == 0 && lane + 32 * q < n) flag[lo + lane + 32 * q] = live[q] >> lane & 1 ? 0 : 1;
    }
    close = __any_sync(0xffffffffu, close);
    if (close) {  // the same in every warp of the node
      __syncwarp();
      if (gt == 0) {
        // the recurrence over neighbours: rotate (p, s), z_p -> 0, z_s -> t; p deflates
        int p = -1, nr = 0;
        for (int s = 0; s < n; s++) {
          if (flag[lo + s]) continue;
          if (p >= 0) {
            const double zp = zs[lo + p], zj = zs[lo + s], t = hypot(zp, zj), c = zj / t, sn = zp / t;
            if (fabs((key[lo + s] - key[lo + p]) * c * sn) <= tol) {
              rc[lo + nr] = c;
              rs[lo + nr] = sn;
              rp[lo + nr] = sidx[lo + p];
              rj[lo + nr] = sidx[lo + s];
              nr++;
              const double dp = key[lo + p], ds = key[lo + s];
              key[lo + p] = c * c * dp + sn * sn * ds;
              key[lo + s] = sn * sn * dp + c * c * ds;
              zs[lo + s] = t;
              flag[lo + p] = 1;
            }
          }
          p = s;
        }
        nrot[node] = nr;
      }
    }
    __syncthreads();
    if (gt < n) {  // the rotations, one column per thread
      double* col = Z + lo * ld + lo + gt;
      const int nr = nrot[node];
      for (int q = 0; q < nr; q++) {
        const double c = rc[lo + q], sn = rs[lo + q];
        double* zp = col + rp[lo + q] * ld;
        double* zj = col + rj[lo + q] * ld;
        const double a = *zp, b = *zj;
        *zp = c * a - sn * b;
        *zj = sn * a + c * b;
      }
    }
    // The merge in units of 2^ex, in which poles and rho are at most of order one: a node far down a graded
    // problem (a matrix of low rank leaves remainders of 1e-16, 1e-32, ... of its norm) has poles whose
    // squares and reciprocal squares the problem's own units do not hold.
    const int ex = min(1000, max(-1000, ilogb(fmax(fmax(fabs(key[lo]), fabs(key[hi - 1])), rho0))));
    const double unit = scalbn(1.0, -ex), rho = rho0 * unit;
    int K = 0;
    {
      int before[R];
      bool al[R];
#pragma unroll
      for (int q = 0; q < R; q++) {
        al[q] = lane + 32 * q < n && !flag[lo + lane + 32 * q];
        const unsigned m = __ballot_sync(0xffffffffu, al[q]);
        before[q] = K + __popc(m & ((1u << lane) - 1u));
        K += __popc(m);
      }
      if (wn == 0) {
#pragma unroll
        for (int q = 0; q < R; q++) {
          const int s = lane + 32 * q;
          if (s >= n) continue;
          const int t = al[q] ? before[q] : K + (s - before[q]);
          srow[lo + t] = sidx[lo + s];
          if (al[q]) {
            pole[lo + t] = key[lo + s] * unit;
            zz[lo + t] = zs[lo + s];
          } else {
            lamn[lo + t] = key[lo + s];
          }
        }
      }
    }
    __syncthreads();
    // secular roots, W lanes each (eig_large.cu: dc_secular_kernel)
    const int W = 8 * n <= G ? 8 : 4 * n <= G ? 4 : 2;
    auto wsum = [&](double x) {
      for (int o = W >> 1; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      return x;
    };
    const double* P = pole + lo;
    const double* zp = zz + lo;
    const int j = gt / W, wl = gt % W;
    {
      double dorg = 0.0, low = 0.0, high = 0.0, t = 0.0;
      const bool act = j < K, last = j == K - 1;
      const int p1 = last ? K - 2 : j, p2 = p1 + 1;
      double s = 0.0;
      if (act && K > 1) {
        if (!last) {
          const double dj = P[j], m = 0.5 * (P[j + 1] - dj);
#pragma unroll 4
          for (int i = wl; i < K; i += W) s += zp[i] * zp[i] / ((P[i] - dj) - m);
        } else {
          for (int i = wl; i < K; i += W) s += zp[i] * zp[i];
        }
      }
      s = wsum(s);
      if (act && K == 1) {
        dorg = P[0];
        t = rho * zp[0] * zp[0];
      } else if (act && last) {
        dorg = P[K - 1];
        high = rho * s;
        t = 0.5 * high;
      } else if (act) {
        const double gap = P[j + 1] - P[j], m = 0.5 * gap, f = 1.0 + rho * s;
        const double z1 = rho * zp[j] * zp[j], z2 = rho * zp[j + 1] * zp[j + 1], c = f + (z1 - z2) / m;
        dorg = f >= 0.0 ? P[j] : P[j + 1];
        low = f >= 0.0 ? 0.0 : -m;
        high = f >= 0.0 ? m : 0.0;
        t = secular_start(f, c, gap, z1, z2);
        if (!(t > low && t < high)) t = 0.5 * (low + high);
      }
      bool done = !act || K == 1;
      const double d1 = done ? 0.0 : P[p1] - dorg, d2 = done ? 0.0 : P[p2] - dorg;
      for (int it = 0; it < 100 && !__all_sync(0xffffffffu, done); it++) {
        double psi = 0.0, dpsi = 0.0, phi = 0.0, dphi = 0.0;
        if (!done) {
#pragma unroll 4
          for (int i = wl; i < K; i += W) {
            const double z = zp[i], q = z / ((P[i] - dorg) - t);
            const double zl = i <= p1 ? z : 0.0, ql = i <= p1 ? q : 0.0, zr = i <= p1 ? 0.0 : z, qr = i <= p1 ? 0.0 : q;
            psi = fma(zl, q, psi);
            dpsi = fma(ql, q, dpsi);
            phi = fma(zr, q, phi);
            dphi = fma(qr, q, dphi);
          }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
          if (o < W) {
            psi += __shfl_xor_sync(0xffffffffu, psi, o);
            dpsi += __shfl_xor_sync(0xffffffffu, dpsi, o);
            phi += __shfl_xor_sync(0xffffffffu, phi, o);
            dphi += __shfl_xor_sync(0xffffffffu, dphi, o);
          }
        psi *= rho;
        dpsi *= rho;
        phi *= rho;
        dphi *= rho;
        const double f = 1.0 + psi + phi;
        const double err = 8.0 * (fabs(psi) + fabs(phi)) + 2.0 + 3.0 * fabs(t) * (dpsi + dphi);
        done = done || fabs(f) <= kEps * err;
        const double nlow = f < 0.0 ? t : low, nhigh = f < 0.0 ? high : t;
        const double tn = t + secular_step(f, dpsi, dphi, d1 - t, d2 - t, last);
        const double tm = tn > nlow && tn < nhigh ? tn : 0.5 * (nlow + nhigh);
        if (!done) {
          low = nlow;
          high = nhigh;
          done = tm == t;
          t = tm;
        }
      }
      if (act && wl == 0) {
        org[lo + j] = dorg;
        tau[lo + j] = t;
        lamn[lo + j] = scalbn(dorg + t, ex);
      }
    }
    __syncthreads();
    // z-hat of entry j
    const double* og = org + lo;
    const double* ta = tau + lo;
    {
      double p = 1.0;
      if (j < K) {
        const double di = P[j];
#pragma unroll 4
        for (int q = wl; q < K - 1; q += W) p *= -((di - og[q]) - ta[q]) / (P[q < j ? q : q + 1] - di);
        if (wl == 0) p *= -((di - og[K - 1]) - ta[K - 1]) / rho;
      }
      for (int o = W >> 1; o > 0; o >>= 1) p *= __shfl_xor_sync(0xffffffffu, p, o);
      if (j < K && wl == 0) zh[lo + j] = copysign(sqrt(fabs(p)), zp[j]);
    }
    __syncthreads();
    // vectors of the merged problem, rows of U
    {
      double* row = U + (lo + j) * ld + lo;
      double ss = 0.0;
      if (j < K)
#pragma unroll 4
        for (int i = wl; i < K; i += W) {
          const double u = zh[lo + i] / ((P[i] - og[j]) - ta[j]);
          row[i] = u;
          ss = fma(u, u, ss);
        }
      ss = wsum(ss);
      if (j < K) {
        if (wl == 0 && !(ss > 0.0 && isfinite(ss))) atomicMax(status, lo + j + 1);
        const double inv = 1.0 / sqrt(ss);
        for (int i = wl; i < K; i += W) row[i] *= inv;
      }
    }
    __syncthreads();
    // new rows = U times the old ones; deflated rows are moved
    {
      const double* Un = U + lo * ld + lo;
      double* Zn = Z + lo * ld + lo;
      constexpr int NU = R == 3 ? 2 : 1;  // n <= 12 / 2^level tile rows over 8 / 2^level warps
      // dc_rows has a barrier, so every node of the level takes the instance of its largest
      const int tn = ((N + (1 << lev) - 1 >> lev) + 7) / 8;
      constexpr int M = cta_eig_max(R, T) / 8;
      if (tn <= 1) dc_rows<1, NU>(Un, Zn, ld, srow + lo, n, K, wn, nw);
      else if (tn <= 2) dc_rows<2, NU>(Un, Zn, ld, srow + lo, n, K, wn, nw);
      else if (M > 2 && tn <= 4) dc_rows<M < 4 ? M : 4, NU>(Un, Zn, ld, srow + lo, n, K, wn, nw);
      else if (M > 4 && tn <= 8) dc_rows<M < 8 ? M : 8, NU>(Un, Zn, ld, srow + lo, n, K, wn, nw);
      else if (M > 8) dc_rows<M, NU>(Un, Zn, ld, srow + lo, n, K, wn, nw);
    }
    if (gt < n) {
      bool ok = true;
      d[lo + gt] = finite_or_zero(lamn[lo + gt], ok);
      if (!ok) atomicMax(status, lo + gt + 1);
    }
    __syncthreads();
  }
  if (tid < N) d[tid] = scalbn(d[tid], ex);
  __syncthreads();
  return *status;
}

// Sum over the lanes of x[c] for c = (lane >> 2) & 7, in every lane (9 shuffles).
NRG_DEV double colsum8(double (&x)[8], int lane) {
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

// Sum over the warp, in every lane, by two DMMAs with a matrix of ones: the first sums over the
// lanes of equal l/4, the second over the eight groups (87 cycles against 190 of five shuffles and
// adds).
NRG_DEV double warp_sum_mma(double x) {
  double d0 = 0.0, d1 = 0.0, e0 = 0.0, e1 = 0.0;
  dmma884(d0, d1, 1.0, x);
  dmma884(e0, e1, 1.0, d0 + d1);
  return e0;
}

// Householder reflectors of columns (alpha, x) whose squares leave the range of doubles. Where alpha^2 + |x|^2
// is below 1e-270 (0 for a column that is reduced already), |x|^2 is not known well enough for tau and x
// to give an orthogonal reflector, nor is A x for its update: the column is multiplied by kTinyUp, its squares
// are summed again, and the reflector is formed in these units. A column with |x| below 1e-290 counts
// as reduced. (Such columns come in blocks of norm one: each column of a matrix of low rank leaves a
// remainder of 1e-16 times the last.)
constexpr double kTinyUp = 0x1p700;
NRG_DEV bool tiny_column(double alpha, double sigma) { return fma(alpha, alpha, sigma) < 1e-270; }
NRG_DEV double tiny_squares(double sum) { return sum > 1e-160 ? sum : 0.0; }

// Householder reduction A = Q T Q^T of the symmetric matrix A of order n <= 32 R (2 <= n) in shared memory
// (row stride ld, both triangles), T threads. On exit d, e, taus and the reflectors v_k packed
// one after another in V (v_k's n-k-1 entries from row k+1 on, the first one 1).
// The matrix moves to registers: warp w of nw has the columns w + nw q, lane l the rows l + 32 s. As in
// tridiag_dsm_kernel (eig_large.cu) the previous rank-2 update and the product with the new
// reflector are one pass, and a column costs one barrier: the products and the next row go
// through shared memory, and every warp builds the reflector for itself.
// Scratch: yb, rb 2n doubles each, pr 16 n doubles (a (v, w) copy per warp).
template <int R, int T = kCtaEigThreads>
NRG_DEV void cta_tridiagonalise(const double* A, int ld, int n, double* d, double* e, double* taus, double* V,
                                double* yb, double* rb, double* pr) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nw = T / 32, Q = cta_eig_max(R, T) / nw;
  double x[R][Q];
#pragma unroll
  for (int s = 0; s < R; s++)
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const int i = lane + 32 * s, j = warp + nw * q;
      x[s][q] = i < n && j < n ? A[i * ld + j] : 0.0;
    }
  for (int i = tid; i < n; i += T) {
    yb[i] = 0.0;
    rb[i] = A[i];
  }
  double2* vw = reinterpret_cast<double2*>(pr) + warp * n;
  double u[R] = {}, tau = 0.0, scale = 1.0;
  __syncthreads();
  for (int k = 0; k < n - 1; k++) {
    const double* y = yb + (k & 1) * n;
    const double* row = rb + (k & 1) * n;
    const double f = tau * scale, yk = f * y[k];
    double v[R], w[R], pd = 0.0;
#pragma unroll
    for (int s = 0; s < R; s++) {
      const int i = lane + 32 * s;
      const bool in = k > 0 && i >= k && i < n;
      v[s] = !in ? 0.0 : i == k ? 1.0 : scale * u[s];
      w[s] = in ? f * y[i] : 0.0;
      pd = fma(w[s], v[s], pd);
    }
    const double Kc = 0.5 * tau * warp_sum_mma(pd);
    const double wk = k > 0 ? yk - Kc : 0.0;
    double ps = 0.0;
    const int vo = (k - 1) * n - (k - 1) * k / 2 - k;  // V[vo + i] = v_{k-1}(i), i >= k
#pragma unroll
    for (int s = 0; s < R; s++) {
      const int i = lane + 32 * s;
      w[s] -= Kc * v[s];
      u[s] = i >= k && i < n ? row[i] - v[s] * wk - w[s] : 0.0;
      if (i >= k + 2) ps = fma(u[s], u[s], ps);
      if (i < n) vw[i] = make_double2(v[s], w[s]);
      if (warp == 0 && k > 0 && i >= k && i < n) V[vo + i] = v[s];
      if (warp == 1 && i == k) d[k] = u[s];
    }
    double sigma = warp_sum_mma(ps), alpha = 0.0, unit = 1.0;
#pragma unroll
    for (int s = 0; s < R; s++) {
      const double a = __shfl_sync(0xffffffffu, u[s], (k + 1) & 31);
      if (s == (k + 1) >> 5) alpha = a;
    }
    __syncwarp();
    if (k == n - 2) {
#pragma unroll
      for (int s = 0; s < R; s++)
#pragma unroll
        for (int q = 0; q < Q; q++)
          if (lane + 32 * s == n - 1 && warp + nw * q == n - 1) d[n - 1] = x[s][q] - 2.0 * v[s] * w[s];
      if (tid == 0) {
        e[k] = alpha;
        e[n - 1] = 0.0;
        taus[k] = taus[n - 1] = 0.0;
      }
      break;
    }
    if (tiny_column(alpha, sigma)) {  // the same in every thread
      alpha *= kTinyUp;
      ps = 0.0;
#pragma unroll
      for (int s = 0; s < R; s++) {
        u[s] *= kTinyUp;
        if (lane + 32 * s >= k + 2) ps = fma(u[s], u[s], ps);
      }
      sigma = tiny_squares(warp_sum_mma(ps));
      unit = 1.0 / kTinyUp;
    }
    const double beta = sigma > 0.0 ? -copysign(sqrt(alpha * alpha + sigma), alpha) : alpha;
    const double u1 = alpha - beta;
#pragma unroll
    for (int s = 0; s < R; s++) {
      if (lane + 32 * s == k + 1) u[s] = u1;
      if (lane + 32 * s <= k) u[s] = 0.0;
    }
    double cs[(Q + 7) / 8 * 8];
#pragma unroll
    for (int q = 0; q < (Q + 7) / 8 * 8; q++) cs[q] = 0.0;
    // every column, dead or alive: those up to k have v_j = w_j = 0 or are not read again, and loads
    // behind a branch would wait for one another
    double2 c[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) c[q] = vw[min(warp + nw * q, n - 1)];
#pragma unroll
    for (int q = 0; q < Q; q++)
#pragma unroll
      for (int s = 0; s < R; s++) {
        x[s][q] = fma(-w[s], c[q].x, fma(-v[s], c[q].y, x[s][q]));
        cs[q] = fma(x[s][q], u[s], cs[q]);
      }
    // the reflector's divisions run beside the sums below
    tau = 0.0;
    scale = 1.0;
    if (sigma > 0.0) {
      tau = (beta - alpha) / beta;
      scale = 1.0 / u1;
    }
    if (tid == 0) {
      e[k] = beta * unit;
      taus[k] = tau;
    }
    double* ny = yb + ((k + 1) & 1) * n;
    double* nr = rb + ((k + 1) & 1) * n;
#pragma unroll
    for (int s = 0; s < R; s++)
      if (lane + 32 * s == k + 1) {
#pragma unroll
        for (int q = 0; q < Q; q++)
          if (warp + nw * q < n) nr[warp + nw * q] = x[s][q];
      }
#pragma unroll
    for (int g = 0; g < (Q + 7) / 8; g++) {
      double t[8];
#pragma unroll
      for (int c = 0; c < 8; c++) t[c] = cs[8 * g + c];
      const double sum = colsum8(t, lane);
      const int j = warp + nw * (8 * g + (lane >> 2));
      if ((lane & 3) == 0 && j < n) ny[j] = sum;
    }
    __syncthreads();
  }
  __syncthreads();
}

// Rows of Z <- rows of Z Q^T: every row z becomes H_0 H_1 ... H_{n-3} z. Four lanes hold a row in
// registers (columns 4 q + l), so the reflectors follow one another without a barrier.
template <int R, int T = kCtaEigThreads>
NRG_DEV void cta_apply_q(double* Z, int ld, int n, const double* taus, const double* V) {
  const int tid = threadIdx.x, l = tid & 3;
  constexpr int Q = cta_eig_max(R, T) / 4;
  for (int r0 = 0; r0 < n; r0 += T / 4) {  // uniform
    const int r = r0 + (tid >> 2);
    double z[Q];
#pragma unroll
    for (int q = 0; q < Q; q++) z[q] = r < n && 4 * q + l < n ? Z[r * ld + 4 * q + l] : 0.0;
    auto load = [&](double (&vc)[Q], int k) {
      const double* v = V + k * n - k * (k + 1) / 2 - (k + 1);  // v[c], c > k
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const int c = 4 * q + l;
        vc[q] = c > k && c < n ? v[c] : 0.0;
      }
    };
    double vc[Q];
    if (n > 2) load(vc, n - 3);
    for (int k = n - 3; k >= 0; k--) {
      const double tau = taus[k];
      double s[4] = {}, vn[Q];
      if (k > 0) load(vn, k - 1);  // beside this one's products
#pragma unroll
      for (int q = 0; q < Q; q++) s[q & 3] = fma(vc[q], z[q], s[q & 3]);
      double t = (s[0] + s[1]) + (s[2] + s[3]);
      t += __shfl_xor_sync(0xffffffffu, t, 1);
      t += __shfl_xor_sync(0xffffffffu, t, 2);
      t *= tau;
#pragma unroll
      for (int q = 0; q < Q; q++) z[q] = fma(-t, vc[q], z[q]);
#pragma unroll
      for (int q = 0; q < Q; q++) vc[q] = vn[q];
    }
#pragma unroll
    for (int q = 0; q < Q; q++)
      if (r < n && 4 * q + l < n) Z[r * ld + 4 * q + l] = z[q];
  }
}

}  // namespace nrg
