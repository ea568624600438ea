// SideStreams (csrc/ctx.h) with fakes of the CUDA calls it makes: the main stream waits for every side stream
// that was added, at join() and when a function is left before it.
#include <cstdio>
#include <string>

#include "ctx.h"

static std::string calls;
static int failing = 0;  // the n-th call fails

static cudaError_t fake(const char* what, void* a, void* b) {
  calls += std::string(what) + " " + std::to_string((long)a) + " " + std::to_string((long)b) + "; ";
  return failing && --failing == 0 ? cudaErrorUnknown : cudaSuccess;
}
extern "C" {
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return fake("record", e, s); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { return fake("wait", s, e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

static int work(bool leave_early) {
  nrg::SideStreams sides((cudaStream_t)1);
  sides.add((cudaStream_t)2, (cudaEvent_t)12);
  sides.add((cudaStream_t)3, (cudaEvent_t)13);
  if (leave_early) return 1;
  return sides.join() == cudaSuccess ? 0 : 2;
}

static bool check(const char* what, bool early, int fail_at, int rc) {
  calls.clear();
  failing = fail_at;
  const bool ok = work(early) == rc && calls.find("record 12 2; ") != std::string::npos &&
                  calls.find("record 13 3; wait 1 13; ") != std::string::npos && calls.rfind("record 12") == 0;
  if (!ok) std::printf("%s: %s\n", what, calls.c_str());
  return ok;
}

int main() {
  bool ok = check("joined", false, 0, 0) && calls == "record 12 2; wait 1 12; record 13 3; wait 1 13; ";
  ok &= check("left early", true, 0, 1) && calls == "record 12 2; wait 1 12; record 13 3; wait 1 13; ";
  ok &= check("a failed record", false, 1, 2);
  ok &= check("a failed wait", false, 2, 2);
  std::puts(ok ? "SIDE STREAMS OK" : "FAILED");
  return ok ? 0 : 1;
}
