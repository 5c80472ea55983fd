#include "side_stream.h"

#include <mutex>
#include <vector>

namespace aosb {
namespace {

struct Side {
  cudaStream_t main, side;
  SideKind kind;
};
std::mutex g_mutex;
std::vector<Side> g_sides;

}  // namespace

int side_stream(cudaStream_t main, SideKind kind, cudaStream_t* out, char* err, size_t cap) {
  int device = 0;
  cudaGetDevice(&device);
  std::lock_guard<std::mutex> lock(g_mutex);
  for (const Side& s : g_sides) {
    int other = -1;
    if (s.main == main && s.kind == kind &&
        cudaStreamGetDevice(s.side, &other) == cudaSuccess && other == device) {
      *out = s.side;
      return 0;
    }
  }
  int least = 0, greatest = 0;
  AOSB_CUDA_TRY(cudaDeviceGetStreamPriorityRange(&least, &greatest), err, cap);
  cudaStream_t side = nullptr;
  AOSB_CUDA_TRY(cudaStreamCreateWithPriority(&side, cudaStreamNonBlocking,
                                             kind == kSideFactor ? greatest : 0),
                err, cap);
  g_sides.push_back({main, side, kind});
  *out = side;
  return 0;
}

int side_stream_forget(cudaStream_t main) {
  std::lock_guard<std::mutex> lock(g_mutex);
  int n = 0;
  for (size_t i = g_sides.size(); i-- > 0;) {
    if (g_sides[i].main != main) continue;
    cudaStreamDestroy(g_sides[i].side);
    g_sides.erase(g_sides.begin() + (std::ptrdiff_t)i);
    ++n;
  }
  return n;
}

}  // namespace aosb

extern "C" int32_t aosb_stream_release(void* stream) {
  return aosb::side_stream_forget((cudaStream_t)stream);
}
