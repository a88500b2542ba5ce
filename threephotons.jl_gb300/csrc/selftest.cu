// Failure-detection self test: a kernel whose bounded mbarrier wait cannot complete
// (no thread ever arrives on the barrier, no copy is in flight), so the wait runs out,
// the kernel records TP3_ERR_TIMEOUT in the context's error flag and returns.  The host
// sees the status at its next synchronising call and the context stays usable.  This
// exercises the same bounded-wait path the tensor-core kernels use around their TMA and
// MMA barriers, without faulting or hanging the device.
//
// Scalar self test: the conversions and the logarithm of the scoring kernels on values of the
// caller's choice.
#include <cuda_runtime.h>

#include <string>

#include "ctx_internal.h"
#include "scalar.cuh"
#include "tc_prims.cuh"

namespace {

__global__ void k_wait_selftest(int* err, long long limit) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    tp3::mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) tp3::mbar_wait_limit(&bar, 0u, limit, err);
}

__global__ void k_scalar_selftest(int op, int n, const void* in, void* out, const tp3::SlabLog* logtab) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (op == 0) ((double*)out)[i] = tp3::slab_log(((const double*)in)[i], logtab);
    if (op == 1) ((double*)out)[i] = tp3::widen(((const float*)in)[i]);
    if (op == 2) ((float*)out)[i] = tp3::narrow(((const double*)in)[i]);
  }
}

}  // namespace

extern "C" {

int tp3_selftest_timeout(tp3_ctx* c, long long cycles) {
  if (int r = tp3::ctx_check(c)) return r;
  if (cycles < 1000 || cycles > 4000000000LL) return tp3::ctx_fail(c, TP3_ERR_ARG, "cycles out of range");
  k_wait_selftest<<<1, 32, 0, c->stream>>>(c->d_err, cycles);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return tp3::ctx_cuda_fail(c, e, "self test");
  return TP3_OK;
}

int tp3_selftest_scalar(tp3_ctx* c, int op, int n, const void* in, void* out) {
  if (int r = tp3::ctx_check(c)) return r;
  if (op < 0 || op > 2 || n < 1 || !in || !out) return tp3::ctx_fail(c, TP3_ERR_ARG, "bad self test arguments");
  if (!c->tc_ok) return tp3::ctx_fail(c, TP3_ERR_UNSUPPORTED, "tensor-core path unavailable: " + c->tc_why);
  const size_t bi = (size_t)n * (op == 1 ? 4 : 8), bo = (size_t)n * (op == 2 ? 4 : 8);
  void *d_in = nullptr, *d_out = nullptr;
  cudaError_t e = cudaMalloc(&d_in, bi);
  if (e == cudaSuccess) e = cudaMalloc(&d_out, bo);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_in, in, bi, cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) {
    k_scalar_selftest<<<64, 256, 0, c->stream>>>(op, n, d_in, d_out, c->tc.logtab);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, d_out, bo, cudaMemcpyDeviceToHost, c->stream);
  const cudaError_t es = cudaStreamSynchronize(c->stream);
  cudaFree(d_in);
  cudaFree(d_out);
  if (e == cudaSuccess) e = es;
  if (e != cudaSuccess) return tp3::ctx_cuda_fail(c, e, "scalar self test");
  return TP3_OK;
}

}  // extern "C"
