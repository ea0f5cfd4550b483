// What a step does with the values of its loss layers: their sum over the mini-batch, the objective's
// scale, the gradient that goes back to them, and the running statistics of the mode.  A handful of
// numbers: the launches are all that it costs, so there are three instead of the eleven of one operator
// each (1.2 to 2 us apiece in a replayed step).
#include "common.cuh"

namespace lb {

// out[0] = sum(y) / mini-batch (given as its reciprocal), out[1] = out[0] * scale
template <typename T>
__global__ void __launch_bounds__(1024)
objective_fwd_kernel(const T* __restrict__ y, long long n, float inv, float scale, float* __restrict__ out) {
  __shared__ float scratch[32];
  float s = 0.f;
  for (long long i = threadIdx.x; i < n; i += 1024) s += to_f32<T>(y[i]);
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  s = warp_sum(scratch[threadIdx.x]);
  if (threadIdx.x == 0) {
    const float mean = s * inv;
    out[0] = mean;
    out[1] = mean * scale;
  }
}
template <typename T>
__global__ void __launch_bounds__(256)
objective_bwd_kernel(const float* __restrict__ g, float scale, float inv, T* __restrict__ dy, long long n) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i < n) dy[i] = from_f32<T>(*g * scale * inv);
}

constexpr int kStatsMost = 8;
struct StatsArgs {
  double* sum[kStatsMost];
  const float* value[kStatsMost];
  int count;
};
__global__ void add_statistics_kernel(const StatsArgs a, double weight) {
  if ((int)threadIdx.x < a.count) *a.sum[threadIdx.x] += weight * (double)*a.value[threadIdx.x];
}

}  // namespace lb

extern "C" {

// y: dense, dtype 0 fp16, 1 bf16, 2 fp32; out: fp32[2].
int lb_objective_fwd(const void* y, long long n, float inv, float scale, float* out, int dtype, void* stream_) {
  using namespace lb;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  if (n < 0) return -1;
  if (dtype == kF32) objective_fwd_kernel<float><<<1, 1024, 0, s>>>((const float*)y, n, inv, scale, out);
  else if (dtype == kBF16) objective_fwd_kernel<__nv_bfloat16><<<1, 1024, 0, s>>>((const __nv_bfloat16*)y, n, inv, scale, out);
  else if (dtype == kF16) objective_fwd_kernel<__half><<<1, 1024, 0, s>>>((const __half*)y, n, inv, scale, out);
  else return -1;
  return (int)cudaGetLastError();
}
int lb_objective_bwd(const float* g, float scale, float inv, void* dy, long long n, int dtype, void* stream_) {
  using namespace lb;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  if (n <= 0) return 0;
  const int blocks = (int)((n + 255) / 256);
  if (dtype == kF32) objective_bwd_kernel<float><<<blocks, 256, 0, s>>>(g, scale, inv, (float*)dy, n);
  else if (dtype == kBF16) objective_bwd_kernel<__nv_bfloat16><<<blocks, 256, 0, s>>>(g, scale, inv, (__nv_bfloat16*)dy, n);
  else if (dtype == kF16) objective_bwd_kernel<__half><<<blocks, 256, 0, s>>>(g, scale, inv, (__half*)dy, n);
  else return -1;
  return (int)cudaGetLastError();
}
// *sums[i] += weight * *values[i], at most eight; the sums are different ones.
int lb_add_statistics(void* const* sums, const void* const* values, int count, double weight, void* stream_) {
  using namespace lb;
  if (count < 1 || count > kStatsMost) return -1;
  StatsArgs a;
  a.count = count;
  for (int i = 0; i < count; ++i) {
    a.sum[i] = (double*)sums[i];
    a.value[i] = (const float*)values[i];
  }
  add_statistics_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(a, weight);
  return (int)cudaGetLastError();
}

}  // extern "C"
