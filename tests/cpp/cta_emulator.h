// cta_emulator.h -- runs a CTA or a cluster of device code on the CPU: every thread is a fiber that
// yields at a barrier, a warp exchange or an mbarrier until what it waits for has come. Stands in for
// <cuda_runtime.h> in host builds of csrc (tests/test_small_solver_cpu.py,
// tests/test_cluster_exchange_cpu.py).
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
  int wround = 0, bround = 0, cround = 0;  // exchanges and barriers it has come to
};
struct EmuWarp {
  uint64_t v[2][32];
  int here[2] = {0, 0}, round = 0;
};
struct EmuCta {
  std::vector<EmuWarp> w;
  std::vector<double> mem;
  int here = 0, round = 0, any[2] = {0, 0};
  std::string at;      // where the first thread came to the barrier
  bool apart = false;  // threads met at different barriers
};
struct Emu {
  int threads;  // per CTA
  std::vector<EmuThread> t;
  std::vector<EmuCta> cta;
  int here = 0, round = 0;  // the cluster's barrier
  long long events = 0;     // anything that may let a thread go on
  int me = 0;               // the running thread
  jmp_buf sched;
  std::function<void()> body;
};
struct EmuDim { int x = 0, y = 0, z = 0; };
inline EmuDim threadIdx, blockIdx, blockDim;
inline Emu* emu = nullptr;
constexpr size_t kEmuGuard = 4096;

inline EmuThread& emu_thread() { return emu->t[emu->me]; }
inline EmuCta& emu_cta() { return emu->cta[blockIdx.x]; }
inline double* emu_smem() { return emu_cta().mem.data() + kEmuGuard; }
inline void emu_switch(int me) {
  emu->me = me;
  threadIdx.x = me % emu->threads;
  blockIdx.x = me / emu->threads;
}
inline void emu_yield() {
  const int me = emu->me;
  if (!_setjmp(emu->t[me].jb)) _longjmp(emu->sched, 1);
  emu_switch(me);
}
inline void emu_put(uint64_t v) {  // a value of this lane, for all lanes of its warp
  const int r = emu_thread().wround++;
  EmuWarp& w = emu_cta().w[threadIdx.x / 32];
  w.v[r & 1][threadIdx.x % 32] = v;
  if (++w.here[r & 1] == 32) {
    w.here[r & 1] = 0;
    w.round = r + 1;
    emu->events++;
  }
  while (w.round <= r) emu_yield();
}
inline uint64_t emu_get(int lane) { return emu_cta().w[threadIdx.x / 32].v[(emu_thread().wround - 1) & 1][lane]; }
inline uint64_t emu_bits(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
inline double emu_double(uint64_t u) { double d; memcpy(&d, &u, 8); return d; }

inline int emu_barrier(int p, const char* function, int line) {
  EmuCta& c = emu_cta();
  const int r = emu_thread().bround++;
  const std::string at = std::string(function) + std::to_string(line);
  if (c.here == 0) {
    c.any[r & 1] = 0;
    c.at = at;
  }
  c.apart |= at != c.at;
  c.any[r & 1] |= p != 0;
  if (++c.here == emu->threads) {
    c.here = 0;
    c.round = r + 1;
    emu->events++;
  }
  while (c.round <= r) emu_yield();
  return c.any[r & 1];
}
#define __syncthreads_or(p) emu_barrier(p, __PRETTY_FUNCTION__, __LINE__)  // with its template arguments
#define __syncthreads() emu_barrier(0, __PRETTY_FUNCTION__, __LINE__)
inline void emu_cluster_sync() {
  const int r = emu_thread().cround++;
  if (++emu->here == (int)emu->t.size()) {
    emu->here = 0;
    emu->round = r + 1;
    emu->events++;
  }
  while (emu->round <= r) emu_yield();
}
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
inline int atomicMin(int* p, int v) {
  const int old = *p;
  *p = min(old, v);
  return old;
}
inline int atomicExch(int* p, int v) {
  const int old = *p;
  *p = v;
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

// An mbarrier in shared memory (8 bytes, one arrival per phase) with the bytes expected less those that have
// come. Shared memory addresses are the CTA's rank and a byte offset.
inline unsigned emu_address(const void* p) {
  return (unsigned)blockIdx.x << 24 | (unsigned)(static_cast<const char*>(p) - reinterpret_cast<char*>(emu_smem()));
}
inline void* emu_pointer(unsigned a) {
  return reinterpret_cast<char*>(emu->cta[a >> 24].mem.data() + kEmuGuard) + (a & 0xffffff);
}
struct EmuMbar { int bytes; unsigned missing : 31, phase : 1; };
inline void emu_mbar_settle(EmuMbar* b) {
  if (b->missing == 0 && b->bytes == 0) {
    b->phase ^= 1;
    b->missing = 1;
    emu->events++;
  }
}
inline void emu_mbar_init(void* bar) { *static_cast<EmuMbar*>(bar) = EmuMbar{0, 1, 0}; }
inline void emu_mbar_expect(void* bar, unsigned bytes) {
  EmuMbar* b = static_cast<EmuMbar*>(bar);
  b->bytes += (int)bytes;
  b->missing--;
  emu_mbar_settle(b);
}
inline void emu_mbar_complete(unsigned bar, unsigned bytes) {
  EmuMbar* b = static_cast<EmuMbar*>(emu_pointer(bar));
  b->bytes -= (int)bytes;
  emu_mbar_settle(b);
}
inline bool emu_mbar_wait(void* bar, unsigned parity) {
  while (static_cast<EmuMbar*>(bar)->phase == parity) emu_yield();
  return true;
}

inline void emu_entry() {
  emu->body();
  emu_thread().done = true;
  emu->events++;
  _longjmp(emu->sched, 1);
}
// Runs `body` as `ctas` CTAs of `threads` with `smem` doubles of shared memory each, set to `fill`. The threads
// of CTA `slow` run only when nothing else can. Returns 0, or 1000 if a CTA wrote outside its shared
// memory, 1001 if threads met at different barriers, 1002 if nothing could go on.
inline int emu_run(int ctas, int threads, size_t smem, double fill, const std::function<void()>& body, int slow = -1) {
  Emu e;
  e.threads = threads;
  e.t.resize(ctas * threads);
  e.cta.resize(ctas);
  e.body = body;
  emu = &e;
  blockDim.x = threads;
  for (EmuCta& c : e.cta) {
    c.w.resize(threads / 32);
    c.mem.assign(smem + 2 * kEmuGuard, 0.5);
    std::fill(c.mem.begin() + kEmuGuard, c.mem.end() - kEmuGuard, fill);
  }
  for (EmuThread& t : e.t) {
    getcontext(&t.uc);
    t.uc.uc_stack.ss_sp = t.stack.data();
    t.uc.uc_stack.ss_size = t.stack.size();
    t.uc.uc_link = nullptr;
    makecontext(&t.uc, emu_entry, 0);
  }
  volatile bool left = true, waited = false;
  while (left) {
    left = false;
    const long long before = e.events;
    for (volatile int i = 0; i < ctas * threads; i = i + 1) {
      EmuThread& t = e.t[i];
      if (t.done) continue;
      left = true;
      if (i / threads == slow && !waited) continue;
      emu_switch(i);
      if (!_setjmp(e.sched)) {
        if (!t.started) {
          t.started = true;
          setcontext(&t.uc);
        }
        _longjmp(t.jb, 1);
      }
    }
    if (left && e.events == before && (waited || slow < 0)) return 1002;
    waited = e.events == before;
  }
  for (const EmuCta& c : e.cta) {
    for (size_t i = 0; i < kEmuGuard; i++)
      if (c.mem[i] != 0.5 || c.mem[c.mem.size() - 1 - i] != 0.5) return 1000;
    if (c.apart) return 1001;
  }
  return 0;
}
