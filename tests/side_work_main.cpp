// SideWork against a recording stand-in for the CUDA calls it makes.
#include "side_stream.h"

#include <cstdio>
#include <cstdlib>
#include <string>

namespace {
std::string g_log;
cudaStream_t stream(long v) { return reinterpret_cast<cudaStream_t>(v); }
const char* name(cudaStream_t s) { return s == stream(1) ? "main" : s == stream(2) ? "side" : "?"; }
int g_events = 0;
}  // namespace

extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(16L + g_events++);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) {
  --g_events;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  g_log += std::string("record ") + name(s) + (e == reinterpret_cast<cudaEvent_t>(16L) ? " r;" : " d;");
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  g_log += std::string("wait ") + name(s) + (e == reinterpret_cast<cudaEvent_t>(16L) ? " r;" : " d;");
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "error"; }
}

namespace aosb {
int side_stream(cudaStream_t, SideKind, cudaStream_t* out, char*, size_t) {
  *out = stream(2);
  return 0;
}
}  // namespace aosb

// A factorization in outline: `fail_at` is the step that ends with an error
// between its fork and its join.
static int run(int steps, int fail_at) {
  aosb::SideWork work;
  if (int rc = work.open(stream(1), aosb::kSideFactor, nullptr, 0)) return rc;
  for (int k = 0; k < steps; ++k) {
    if (int rc = work.fork(nullptr, 0)) return rc;
    g_log += "launch side;";
    if (k == fail_at) return 7;
    if (int rc = work.join(nullptr, 0)) return rc;
  }
  return 0;
}

int main(int argc, char** argv) {
  if (argc != 3) return 2;
  const int rc = run(std::atoi(argv[1]), std::atoi(argv[2]));
  std::printf("%d %d %s\n", rc, g_events, g_log.c_str());
  return 0;
}
