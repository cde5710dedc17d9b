// A helper stream beside the caller's.
#pragma once

#include "common.cuh"

namespace {

// A second stream of higher priority and the two events that fork it from and join it back to the caller's stream.  The
// destructor joins as well, so that every return path leaves the caller's stream ordered after all work on it.
struct SideStream {
  cudaStream_t main = nullptr, side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  int create(cudaStream_t s) {
    main = s;
    int least = 0, greatest = 0;
    UPDES_CUDA_TRY(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    UPDES_CUDA_TRY(cudaStreamCreateWithPriority(&side, cudaStreamNonBlocking, greatest));
    UPDES_CUDA_TRY(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    UPDES_CUDA_TRY(cudaEventCreateWithFlags(&join, cudaEventDisableTiming));
    return UPDES_OK;
  }
  int start() {  // the side stream waits for all work issued on the caller's stream so far
    UPDES_CUDA_TRY(cudaEventRecord(fork, main));
    UPDES_CUDA_TRY(cudaStreamWaitEvent(side, fork, 0));
    return UPDES_OK;
  }
  int finish() {  // the caller's stream waits for all work issued on the side stream so far
    UPDES_CUDA_TRY(cudaEventRecord(join, side));
    UPDES_CUDA_TRY(cudaStreamWaitEvent(main, join, 0));
    return UPDES_OK;
  }
  ~SideStream() {
    bool bad = false;
    if (side && join) {
      bad |= cudaEventRecord(join, side) != cudaSuccess;
      bad |= cudaStreamWaitEvent(main, join, 0) != cudaSuccess;
    }
    if (fork) bad |= cudaEventDestroy(fork) != cudaSuccess;
    if (join) bad |= cudaEventDestroy(join) != cudaSuccess;
    if (side) bad |= cudaStreamDestroy(side) != cudaSuccess;
    if (bad) (void)cudaGetLastError();
  }
};

}  // namespace
