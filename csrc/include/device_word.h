// A zeroed 32-bit word of device memory that lives as long as the process. Made so that it is legal, and done at once, also while the calling thread
// captures a stream: a captured fill would not run until the graph is replayed, and then again at every replay.
#pragma once
#include <cuda_runtime.h>

namespace fb {

inline cudaError_t zeroed_device_word(int** out) {
  *out = nullptr;
  cudaStream_t own = nullptr;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(out), sizeof(int));
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&own, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMemsetAsync(*out, 0, sizeof(int), own);
  if (e == cudaSuccess) e = cudaStreamSynchronize(own);
  if (own) cudaStreamDestroy(own);
  cudaThreadExchangeStreamCaptureMode(&mode);
  return e;
}

}  // namespace fb
