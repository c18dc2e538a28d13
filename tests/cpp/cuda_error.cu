// A CUDA call that fails and is thrown leaves no error behind for the next one's check.
#include <cstdio>

#include "common.cuh"

int main() {
  int status = SBDGB_OK;
  try {
    SBDGB_CUDA(cudaSetDevice(1 << 20));  // no such device
  } catch (const sbdgb::Error &e) {
    status = e.status;
  }
  const cudaError_t left = cudaGetLastError();
  std::printf("status %d, left behind: %s\n", status, cudaGetErrorName(left));
  return status == SBDGB_E_CUDA && left == cudaSuccess ? 0 : 1;
}
