// cta_emulator.h -- runs one CTA of device code on the CPU: every thread is a fiber that yields at a
// barrier or a warp exchange until its partners have come there too. Stands in for
// <cuda_runtime.h> in a host build of csrc/eig_small.cuh (tests/test_small_solver_cpu.py).
#pragma once
#include <setjmp.h>
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <string>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __shared__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __restrict__
#define __align__(n)

using std::isfinite;
using std::max;
using std::min;

struct double2 { double x, y; };
inline double2 make_double2(double x, double y) { return {x, y}; }
inline double rsqrt(double x) { return 1.0 / std::sqrt(x); }

struct EmuThread {
  ucontext_t uc;
  jmp_buf jb;
  std::vector<char> stack = std::vector<char>(1 << 16);
  bool started = false, done = false;
  int wround = 0, bround = 0;  // exchanges and barriers it has come to
};
struct EmuWarp {
  uint64_t v[2][32];
  int here[2] = {0, 0}, round = 0;
};
struct EmuCta {
  std::vector<EmuThread> t;
  std::vector<EmuWarp> w;
  int here = 0, round = 0, any[2] = {0, 0};
  std::string at;      // where the first thread came to the barrier
  bool apart = false;  // threads met at different barriers
  jmp_buf sched;
  std::function<void()> body;
};
struct EmuDim { int x = 0, y = 0, z = 0; };
inline EmuDim threadIdx, blockIdx, blockDim;
inline EmuCta* emu = nullptr;
inline double* emu_smem = nullptr;

inline void emu_yield() {
  const int me = threadIdx.x;
  if (!_setjmp(emu->t[me].jb)) _longjmp(emu->sched, 1);
  threadIdx.x = me;
}
inline void emu_put(uint64_t v) {  // a value of this lane, for all lanes of its warp
  const int me = threadIdx.x, r = emu->t[me].wround++;
  EmuWarp& w = emu->w[me / 32];
  w.v[r & 1][me % 32] = v;
  if (++w.here[r & 1] == 32) {
    w.here[r & 1] = 0;
    w.round = r + 1;
  }
  while (w.round <= r) emu_yield();
}
inline uint64_t emu_get(int lane) {
  const int me = threadIdx.x;
  return emu->w[me / 32].v[(emu->t[me].wround - 1) & 1][lane];
}
inline uint64_t emu_bits(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
inline double emu_double(uint64_t u) { double d; memcpy(&d, &u, 8); return d; }

inline int emu_barrier(int p, const char* function, int line) {
  const int me = threadIdx.x, r = emu->t[me].bround++;
  const std::string at = std::string(function) + std::to_string(line);
  if (emu->here == 0) {
    emu->any[r & 1] = 0;
    emu->at = at;
  }
  emu->apart |= at != emu->at;
  emu->any[r & 1] |= p != 0;
  if (++emu->here == (int)emu->t.size()) {
    emu->here = 0;
    emu->round = r + 1;
  }
  while (emu->round <= r) emu_yield();
  return emu->any[r & 1];
}
#define __syncthreads_or(p) emu_barrier(p, __PRETTY_FUNCTION__, __LINE__)  // with its template arguments
#define __syncthreads() emu_barrier(0, __PRETTY_FUNCTION__, __LINE__)
inline void __syncwarp() { emu_put(0); }
inline double __shfl_sync(unsigned, double v, int src) {
  emu_put(emu_bits(v));
  return emu_double(emu_get(src & 31));
}
inline double __shfl_xor_sync(unsigned m, double v, int o) { return __shfl_sync(m, v, (threadIdx.x & 31) ^ o); }
inline unsigned __ballot_sync(unsigned, int p) {
  emu_put(p != 0);
  unsigned m = 0;
  for (int l = 0; l < 32; l++) m |= (unsigned)emu_get(l) << l;
  return m;
}
inline int __all_sync(unsigned m, int p) { return __ballot_sync(m, p) == 0xffffffffu; }
inline int __any_sync(unsigned m, int p) { return __ballot_sync(m, p) != 0; }
inline int __ffs(unsigned x) { return __builtin_ffs((int)x); }
inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline int atomicMax(int* p, int v) {
  const int old = *p;
  *p = max(old, v);
  return old;
}
// mma.sync m8n8k4 f64 (fragment layout as in common.cuh)
inline void emu_dmma884(double& d0, double& d1, double a, double b) {
  const int l = threadIdx.x & 31, r = l >> 2, c = 2 * (l & 3);
  double A[4], B0[4], B1[4];
  emu_put(emu_bits(a));
  for (int k = 0; k < 4; k++) A[k] = emu_double(emu_get(4 * r + k));
  emu_put(emu_bits(b));
  for (int k = 0; k < 4; k++) {
    B0[k] = emu_double(emu_get(4 * c + k));
    B1[k] = emu_double(emu_get(4 * (c + 1) + k));
  }
  for (int k = 0; k < 4; k++) {
    d0 = std::fma(A[k], B0[k], d0);
    d1 = std::fma(A[k], B1[k], d1);
  }
}

inline void emu_entry() {
  const int me = threadIdx.x;
  emu->body();
  emu->t[me].done = true;
  _longjmp(emu->sched, 1);
}
// Runs `body` as a CTA of `threads` with `smem` doubles of shared memory, each set to `fill`: 0, or 1000 if it
// wrote outside them, or 1001 if threads met at different barriers.
inline int emu_run(int threads, size_t smem, double fill, const std::function<void()>& body) {
  constexpr size_t kGuard = 4096;
  std::vector<double> mem(smem + 2 * kGuard, 0.5);
  std::fill(mem.begin() + kGuard, mem.end() - kGuard, fill);
  EmuCta cta;
  cta.t.resize(threads);
  cta.w.resize(threads / 32);
  cta.body = body;
  emu = &cta;
  emu_smem = mem.data() + kGuard;
  blockDim.x = threads;
  for (EmuThread& t : cta.t) {
    getcontext(&t.uc);
    t.uc.uc_stack.ss_sp = t.stack.data();
    t.uc.uc_stack.ss_size = t.stack.size();
    t.uc.uc_link = nullptr;
    makecontext(&t.uc, emu_entry, 0);
  }
  for (bool left = true; left;) {
    left = false;
    for (volatile int i = 0; i < threads; i = i + 1) {
      EmuThread& t = cta.t[i];
      if (t.done) continue;
      left = true;
      threadIdx.x = i;
      if (!_setjmp(cta.sched)) {
        if (!t.started) {
          t.started = true;
          setcontext(&t.uc);
        }
        _longjmp(t.jb, 1);
      }
    }
  }
  for (size_t i = 0; i < kGuard; i++)
    if (mem[i] != 0.5 || mem[mem.size() - 1 - i] != 0.5) return 1000;
  return cta.apart ? 1001 : 0;
}
