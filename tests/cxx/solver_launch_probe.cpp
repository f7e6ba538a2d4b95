// csrc/solve.cu on a CUDA runtime that runs nothing and refuses one launch:
//   solver_launch_probe bicgstab|gcrm K    the K-th kernel launch fails
// The workspace holds what a converged solve left there (or, for GCR, sums of one).
// Prints the status, the steps and the residual that the caller gets, and the launches.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "hmvm_b200.h"

static int g_launches = 0, g_fail = 0;
static cudaError_t refuse() { return ++g_launches == g_fail ? cudaErrorInvalidConfiguration : cudaSuccess; }

extern "C" {
void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return refuse() != cudaSuccess; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return refuse(); }
const char* cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t) {
  if (kind == cudaMemcpyDeviceToHost) std::memcpy(dst, src, n);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }

int hmvm_b200_apply(hmvm_plan*, const void*, void*, void*) { return HMVM_OK; }
int hmvm_b200_plan_status(hmvm_plan*) { return HMVM_OK; }
int hmvm_b200_plan_get_info(const hmvm_plan*, hmvm_plan_info* i) {
  std::memset(i, 0, sizeof *i);
  i->nd = 100;
  i->precision = HMVM_FP64;
  return HMVM_OK;
}
}

namespace hmvm {
int set_error(int status, const std::string&) { return status; }
int solve_workspace(hmvm_plan*, size_t bytes, void** dev, bool* kept) {
  static std::vector<double> ws;
  ws.assign(bytes / sizeof(double) + 1, 1.0);  // every scalar that a solve reads back: 1
  *dev = ws.data();
  *kept = true;
  return HMVM_OK;
}
}  // namespace hmvm

int main(int, char** argv) {
  g_fail = std::atoi(argv[2]);
  double b[100] = {}, u[100] = {}, relres = -1;
  int32_t steps = -1;
  const int rc = std::string(argv[1]) == "bicgstab"
                     ? hmvm_b200_bicgstab(nullptr, b, u, 3, 0.5, &steps, &relres, nullptr)
                     : hmvm_b200_gcrm(nullptr, b, u, 3, 2, 0.5, &steps, &relres, nullptr);
  std::printf("%d %d %g %d\n", rc, steps, relres, g_launches);
  return 0;
}
