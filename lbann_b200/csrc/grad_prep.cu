// What a linear or convolution layer does to a gradient before its products, in one pass over it:
//   g = dy * act'(y)  (activations whose derivative is a function of the output's sign),
//   bias gradient += column sums of g (of the 16-bit values that the products see),
//   g with a row pitch of a multiple of eight elements, which TMA asks of a matrix operand.
// And the last of these alone, for the other operands.
//
// Bound by launches for small layers (three to five kernels before, 2-4 us each) and by memory for
// large ones: a thread owns eight columns and keeps eight 16-byte loads in flight; blocks are
// as wide as the rows allow (up to 4 KB of a row: 512-byte pieces of 16 KB rows ran at half the
// rate), the partial sums of a block's rows meet in shared memory, and one 16-byte atomic per four
// columns and block follows.
#include "common.cuh"

namespace lb {

template <typename T, bool kVec>
__device__ __forceinline__ uint4 gp_load8(const T* p, int n) {      // n columns exist (8 where kVec)
  if (kVec) return *reinterpret_cast<const uint4*>(p);
  const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
  uint32_t v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = j < n ? h[j] : 0;
  return make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
}

// Block (bx, 256 / bx): bx groups of eight columns, the rest of the threads along the rows of a band.
template <typename T, bool kVec, bool kAct>
__global__ void __launch_bounds__(256)
grad_prep_kernel(const T* __restrict__ dy, const T* __restrict__ y, T* __restrict__ g, float* __restrict__ bias_grad,
                 long long rows, int C, long long pitch, long long rows_per_block, int act, float act_param) {
  __shared__ float sm[256 * 8];
  const int bx = blockDim.x, by = blockDim.y;
  const int c0 = (blockIdx.x * bx + threadIdx.x) * 8, n = min(8, C - c0);
  const long long r0 = (long long)blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  float s[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s[j] = 0.f;
  constexpr int U = kAct ? 4 : 8;
  auto finish = [&](uint4 q, const uint4& w, long long r) {
    T* e = reinterpret_cast<T*>(&q);
    if (kAct) {
      const T* o = reinterpret_cast<const T*>(&w);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (!(to_f32<T>(o[j]) > 0.f)) e[j] = from_f32<T>(act == 1 ? 0.f : act_param * to_f32<T>(e[j]));
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] += to_f32<T>(e[j]);
    if (g) *reinterpret_cast<uint4*>(g + r * pitch + c0) = q;        // columns C .. pitch are zero
  };
  if (n > 0) {
    long long r = r0 + threadIdx.y;
    for (; r + (U - 1LL) * by < r1; r += (long long)U * by) {
      uint4 q[U], w[kAct ? U : 1];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        q[u] = gp_load8<T, kVec>(dy + (r + (long long)u * by) * C + c0, n);
        if (kAct) w[kAct ? u : 0] = gp_load8<T, kVec>(y + (r + (long long)u * by) * C + c0, n);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) finish(q[u], w[kAct ? u : 0], r + (long long)u * by);
    }
    for (; r < r1; r += by) {
      const uint4 q = gp_load8<T, kVec>(dy + r * C + c0, n);
      const uint4 w = kAct ? gp_load8<T, kVec>(y + r * C + c0, n) : make_uint4(0, 0, 0, 0);
      finish(q, w, r);
    }
  }
  if (!bias_grad) return;
#pragma unroll
  for (int j = 0; j < 8; ++j) sm[(threadIdx.y * 8 + j) * bx + threadIdx.x] = s[j];
  __syncthreads();
  // the block's 8 bx columns, four to a thread (bias_grad is 16-byte aligned where kVec)
  for (int i = (threadIdx.y * bx + threadIdx.x) * 4; i < 8 * bx; i += 1024) {
    const int c = blockIdx.x * bx * 8 + i;
    float t[4] = {0.f, 0.f, 0.f, 0.f};
    for (int r = 0; r < by; ++r) {
#pragma unroll
      for (int j = 0; j < 4; ++j) t[j] += sm[(r * 8 + ((i + j) & 7)) * bx + (i >> 3)];
    }
    if (kVec) {
      if (c < C) atomicAdd(reinterpret_cast<float4*>(bias_grad + c), make_float4(t[0], t[1], t[2], t[3]));
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c + j < C) atomicAdd(bias_grad + c + j, t[j]);
    }
  }
}

// dst[r][0 .. pitch) = src[r][0 .. cols) and zeros; 16-bit elements, any source alignment.
__global__ void __launch_bounds__(256)
pad_rows_kernel(const uint16_t* __restrict__ src, uint16_t* __restrict__ dst, long long rows, int cols, long long src_pitch,
                int pitch) {
  const int v = pitch / 8;
  const long long total = rows * v;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
    const long long r = i / v;
    const int c0 = (int)(i - r * v) * 8;
    reinterpret_cast<uint4*>(dst)[i] =
        gp_load8<uint16_t, false>(src + r * src_pitch + c0, cols - c0);
  }
}

}  // namespace lb

extern "C" {

// dy, y: dense [rows][C], 16 bits; y and act (1 ReLU, 2 leaky ReLU of slope act_param) or null and
// 0.  g (may be null): [rows][pitch], pitch a multiple of 8 and >= C, 16-byte aligned; may be dy
// itself when pitch == C.  bias_grad (may be null): fp32 [C], added to.
int lb_grad_prep(const void* dy, const void* y, void* g, float* bias_grad, long long rows, int C, long long pitch,
                 int act, float act_param, int dtype, void* stream_) {
  using namespace lb;
  if (rows < 1 || C < 1 || (dtype != kF16 && dtype != kBF16)) return -1;
  if (act && !y) return -1;
  if (g && (pitch % 8 || pitch < C || pitch >= C + 8 || (reinterpret_cast<uintptr_t>(g) & 15))) return -1;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  const bool vec = C % 8 == 0 && ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(y) |
                                   reinterpret_cast<uintptr_t>(bias_grad)) & 15) == 0;
  const int cv = (C + 7) / 8;
  int bx = 256;
  while (bx > 1 && bx / 2 >= cv) bx /= 2;
  const dim3 block(bx, 256 / bx);
  const int gx = (cv + bx - 1) / bx;
  // Four blocks an SM at most.  Blocks that share columns add into the same cache lines, which the
  // L2 takes one after another (about 2 ns each): at most one block per SM and column group.
  long long bands = 4LL * lbhost::sm_count() / gx;
  if (bias_grad && bands > lbhost::sm_count()) bands = lbhost::sm_count();
  const long long per = 4LL * block.y;                       // one unrolled round
  if (bands > (rows + per - 1) / per) bands = (rows + per - 1) / per;
  if (bands < 1) bands = 1;
  const long long rpb = (rows + bands - 1) / bands;
  const dim3 grid(gx, (unsigned)((rows + rpb - 1) / rpb));
#define LB_PREP(T, V)                                                                                             \
  (act ? grad_prep_kernel<T, V, true> : grad_prep_kernel<T, V, false>)<<<grid, block, 0, s>>>(                    \
      (const T*)dy, (const T*)y, (T*)g, bias_grad, rows, C, pitch, rpb, act, act_param)
  if (dtype == kBF16) {
    if (vec) LB_PREP(__nv_bfloat16, true);
    else LB_PREP(__nv_bfloat16, false);
  } else {
    if (vec) LB_PREP(__half, true);
    else LB_PREP(__half, false);
  }
#undef LB_PREP
  return (int)cudaGetLastError();
}

// src: 16-bit rows of `cols` elements, src_pitch elements apart; dst: dense [rows][pitch], 16-byte
// aligned, pitch a multiple of 8.
int lb_pad_rows(const void* src, void* dst, long long rows, int cols, long long src_pitch, int pitch, void* stream_) {
  using namespace lb;
  if (rows < 1 || cols < 1 || pitch % 8 || pitch < cols || (reinterpret_cast<uintptr_t>(dst) & 15)) return -1;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  long long blocks = (rows * (pitch / 8) + 255) / 256;
  const long long cap = 8LL * lbhost::sm_count();
  if (blocks > cap) blocks = cap;
  pad_rows_kernel<<<(int)blocks, 256, 0, s>>>((const uint16_t*)src, (uint16_t*)dst, rows, cols, src_pitch, pitch);
  return (int)cudaGetLastError();
}

}  // extern "C"
