// Side streams: work that runs beside the caller's stream.
#pragma once

#include "common.cuh"

namespace aosb {

// The factorization's is of the highest priority (its chain of small kernels
// must not queue behind the updates beside it), the solve's of the default one.
enum SideKind : int { kSideFactor = 0, kSideSolve = 1 };

// Side stream of a caller stream on the current device: created once,
// non-blocking, kept until side_stream_forget(main).
int side_stream(cudaStream_t main, SideKind kind, cudaStream_t* out, char* err, size_t cap);
// Gives back every side stream of `main` (work on it still completes); returns
// how many there were.  Whoever makes streams calls it before it destroys one.
int side_stream_forget(cudaStream_t main);

// A side stream in use: fork() lets it start after the work enqueued on the
// caller's stream so far, join() makes the caller's stream wait for it.  A call
// that returns between the two, with an error, joins on its way out, so that the
// caller's stream never ends before work on the caller's buffers.
class SideWork {
 public:
  SideWork() = default;
  SideWork(const SideWork&) = delete;
  SideWork& operator=(const SideWork&) = delete;
  ~SideWork() {
    if (forked_) {
      cudaEventRecord(done_, stream);
      cudaStreamWaitEvent(main_, done_, 0);
    }
    if (ready_) cudaEventDestroy(ready_);
    if (done_) cudaEventDestroy(done_);
  }
  int open(cudaStream_t main, SideKind kind, char* err, size_t cap) {
    if (int rc = side_stream(main, kind, &stream, err, cap)) return rc;
    main_ = main;
    AOSB_CUDA_TRY(cudaEventCreateWithFlags(&ready_, cudaEventDisableTiming), err, cap);
    AOSB_CUDA_TRY(cudaEventCreateWithFlags(&done_, cudaEventDisableTiming), err, cap);
    return 0;
  }
  int fork(char* err, size_t cap) {
    AOSB_CUDA_TRY(cudaEventRecord(ready_, main_), err, cap);
    AOSB_CUDA_TRY(cudaStreamWaitEvent(stream, ready_, 0), err, cap);
    forked_ = true;
    return 0;
  }
  int join(char* err, size_t cap) {
    AOSB_CUDA_TRY(cudaEventRecord(done_, stream), err, cap);
    AOSB_CUDA_TRY(cudaStreamWaitEvent(main_, done_, 0), err, cap);
    forked_ = false;
    return 0;
  }

  cudaStream_t stream = nullptr;

 private:
  cudaStream_t main_ = nullptr;
  cudaEvent_t ready_ = nullptr, done_ = nullptr;
  bool forked_ = false;
};

}  // namespace aosb
