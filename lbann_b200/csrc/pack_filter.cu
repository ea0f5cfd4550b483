// Convolution filters for the implicit-GEMM kernels, repacked from the fp32 master copy in
// ONE launch per layer and optimizer step:
//   fwd  [tap][Kp][Cp]            = w[k][c][tap]                 (forward operand)
//   dgrad[tap][Cp][Kp]            = w[k][c][taps - 1 - tap]      (data-gradient operand: taps
//                                                                 reversed, channel roles swapped)
// Kp / Cp are the channel counts padded to the kernels' granularity; padding is zero.  The
// reference keeps filters in the vendor library's layout and has no such step.
#include "common.cuh"

namespace lb {

template <typename T>
__global__ void __launch_bounds__(256)
pack_filter_kernel(const float* __restrict__ w, T* __restrict__ fwd, T* __restrict__ dgrad, int K,
                   int C, int taps, int Kp, int Cp) {
  const long long total = (long long)taps * Kp * Cp;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % Cp);
    const int k = (int)((i / Cp) % Kp);
    const int t = (int)(i / ((long long)Cp * Kp));
    const float v = (k < K && c < C) ? w[((long long)k * C + c) * taps + t] : 0.f;
    const T o = from_f32<T>(v);
    if (fwd) fwd[i] = o;
    if (dgrad) dgrad[((long long)(taps - 1 - t) * Cp + c) * Kp + k] = o;
  }
}

// The same for 16-bit layouts through shared memory, 8 filters x CH channels x all taps a block.  The
// master copy is read in runs of CH * taps floats, eight rows in flight; then threads take (filter, channel)
// pairs and taps: forward rows leave in runs of CH * 2 bytes, data-gradient rows in runs of 16.  (Element by
// element, lanes were taps * 4 bytes apart on the way in and Kp * 2 on the way out.)  A block is one
// round trip to memory, so the launch takes 32, 16 or 8 channels, whichever gives four blocks an SM:
// 27 taps, 32 -> 64 channels 7.5 us with 8 blocks of 32, 3.6 with 32 of 8.
constexpr int kPackK = 8;

template <typename T, int CH>
__global__ void __launch_bounds__(256)
pack_filter_tiled_kernel(const float* __restrict__ w, T* __restrict__ fwd, T* __restrict__ dgrad, int K, int C, int taps,
                         int Kp, int Cp) {
  extern __shared__ __align__(16) uint8_t pack_smem[];
  T* tile = reinterpret_cast<T*>(pack_smem);                 // [k][c * taps + t], rows two elements further apart
  const int k0 = blockIdx.y * kPackK, c0 = blockIdx.x * CH;
  const int run = CH * taps, pitch = run + 2;
  const int live = max(0, min(C - c0, CH)) * taps;           // elements of a run that exist
  const float* src = w + ((long long)k0 * C + c0) * taps;
  const long long row = (long long)C * taps;
  for (int i = threadIdx.x; i < run; i += 256) {
    float v[kPackK];
#pragma unroll
    for (int k = 0; k < kPackK; ++k) v[k] = i < live && k0 + k < K ? __ldg(src + k * row + i) : 0.f;
#pragma unroll
    for (int k = 0; k < kPackK; ++k) tile[k * pitch + i] = from_f32<T>(v[k]);
  }
  __syncthreads();
  constexpr int kPairs = CH * kPackK, kSplit = 256 / kPairs;   // threads of a pair take every kSplit-th tap
  const int pair = threadIdx.x % kPairs, t0 = threadIdx.x / kPairs;
  const long long step = (long long)Kp * Cp;
  if (fwd) {
    const int c = pair % CH, k = pair / CH;
    if (c0 + c < Cp && k0 + k < Kp) {
      T* dst = fwd + (long long)(k0 + k) * Cp + c0 + c;
      const T* from = tile + k * pitch + c * taps;
#pragma unroll 4
      for (int t = t0; t < taps; t += kSplit) dst[t * step] = from[t];
    }
  }
  if (dgrad) {
    const int k = pair % kPackK, c = pair / kPackK;
    if (c0 + c < Cp && k0 + k < Kp) {
      T* dst = dgrad + (long long)(c0 + c) * Kp + k0 + k;
      const T* from = tile + k * pitch + c * taps;
#pragma unroll 4
      for (int t = t0; t < taps; t += kSplit) dst[(taps - 1 - t) * step] = from[t];
    }
  }
}

template <typename T>
static int launch_pack_tiled(const float* w, T* fwd, T* dgrad, int K, int C, int taps, int Kp, int Cp, cudaStream_t s) {
  const int rows = (Kp + kPackK - 1) / kPackK;
  int CH = 32;
  while (CH > 8 && (long long)((Cp + CH - 1) / CH) * rows < 4 * lbhost::sm_count()) CH /= 2;
  const dim3 grid((Cp + CH - 1) / CH, rows);
  const int smem = kPackK * (CH * taps + 2) * 2;
  if (CH == 32) pack_filter_tiled_kernel<T, 32><<<grid, 256, smem, s>>>(w, fwd, dgrad, K, C, taps, Kp, Cp);
  else if (CH == 16) pack_filter_tiled_kernel<T, 16><<<grid, 256, smem, s>>>(w, fwd, dgrad, K, C, taps, Kp, Cp);
  else pack_filter_tiled_kernel<T, 8><<<grid, 256, smem, s>>>(w, fwd, dgrad, K, C, taps, Kp, Cp);
  return (int)cudaGetLastError();
}

// The first layer's operand (conv_c8_tc.cu), K index = tap * cr + channel: out [kpad / 8][32 rows][8].  One launch
// instead of the five operators that pad, permute and cast it (7.5 -> 2 us).
template <typename T>
__global__ void __launch_bounds__(256)
pack_first_kernel(const float* __restrict__ w, T* __restrict__ out, int K, int C, int taps, int cr, int kpad) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= kpad * 32) return;
  const int k = (i >> 8) * 8 + (i & 7), row = (i >> 3) & 31, tap = k / cr, c = k - tap * cr;
  out[i] = from_f32<T>(row < K && tap < taps && c < C ? w[((long long)row * C + c) * taps + tap] : 0.f);
}

}  // namespace lb

extern "C" int lb_pack_filter(const float* w, void* fwd, void* dgrad, int K, int C, int taps, int Kp,
                              int Cp, int dtype, void* stream_) {
  using namespace lb;
  if (K < 1 || C < 1 || taps < 1 || Kp < K || Cp < C) return -1;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  // filters of up to 95 taps fit the default 48 KB of shared memory
  const long long smem = (long long)kPackK * (32 * (long long)taps + 2) * 2;
  if (dtype != kF32 && smem <= 48 * 1024 && (Kp + kPackK - 1) / kPackK <= 65535) {
    if (dtype == kF16) return launch_pack_tiled(w, (__half*)fwd, (__half*)dgrad, K, C, taps, Kp, Cp, s);
    if (dtype == kBF16) return launch_pack_tiled(w, (__nv_bfloat16*)fwd, (__nv_bfloat16*)dgrad, K, C, taps, Kp, Cp, s);
    return -1;
  }
  const long long total = (long long)taps * Kp * Cp;
  long long blocks = (total + 255) / 256;
  const long long cap = (long long)lbhost::sm_count() * 8;
  if (blocks > cap) blocks = cap;
  if (dtype == kF16)
    pack_filter_kernel<__half><<<(int)blocks, 256, 0, s>>>(w, (__half*)fwd, (__half*)dgrad, K, C, taps, Kp, Cp);
  else if (dtype == kBF16)
    pack_filter_kernel<__nv_bfloat16><<<(int)blocks, 256, 0, s>>>(w, (__nv_bfloat16*)fwd, (__nv_bfloat16*)dgrad, K, C, taps, Kp, Cp);
  else if (dtype == kF32)
    pack_filter_kernel<float><<<(int)blocks, 256, 0, s>>>(w, (float*)fwd, (float*)dgrad, K, C, taps, Kp, Cp);
  else
    return -1;
  return (int)cudaGetLastError();
}

// w: fp32 [K <= 32][C <= cr][taps], out: 16-bit, kpad a multiple of 16 and not below taps * cr.
extern "C" int lb_pack_first(const float* w, void* out, int K, int C, int taps, int cr, int kpad, int dtype, void* stream_) {
  using namespace lb;
  if (K > 32 || C > cr || kpad % 16 || kpad < taps * cr) return -1;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  if (dtype == kF16) pack_first_kernel<__half><<<kpad / 8, 256, 0, s>>>(w, (__half*)out, K, C, taps, cr, kpad);
  else if (dtype == kBF16) pack_first_kernel<__nv_bfloat16><<<kpad / 8, 256, 0, s>>>(w, (__nv_bfloat16*)out, K, C, taps, cr, kpad);
  else return -1;
  return (int)cudaGetLastError();
}
