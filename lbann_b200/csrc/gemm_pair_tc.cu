// tcgen05 GEMM by pairs of SMs: C[b] (+)= act(alpha * A[b] . B[b]^T + bias), 16-bit inputs, fp32
// accumulation in TMEM.  Two CTAs of a cluster compute one 256 x 256 tile with
// tcgen05.mma.cta_group::2: each holds 128 rows of A and 128 rows of B in its shared memory and
// 128 rows of the accumulator in its TMEM, so an SM fetches 32 KB per 64 steps of the reduction
// for the same MMAs for which the one-SM kernel (gemm_tc.cu) fetches 48 KB.  That is what bounds
// the large products: an SM brings in about 55 B/clk from L2, and a 128 x 256 tile wants 96.
//
// Roles in each CTA (320 threads): warp 4 loads (TMA, one elected thread; the boxes of both CTAs
// count towards the stage barrier of the leader), warp 5 of the leader issues the MMAs, warps 0-3
// and 6-9 drain half the columns of an accumulator each (two accumulators: the next tile's MMAs
// run meanwhile) through shared memory and TMA: 128-byte rows leave as whole lines, and beta = 1
// on an fp32 output is an add at the L2 (cp.reduce) instead of a read of C.
// Every wait is bounded and reports through the status word; both CTAs of a pair run to the
// cluster barrier at the end whatever happened.
#include <atomic>

#include "tc_pipeline.cuh"

namespace lb {

constexpr int kPairStages = 6;
constexpr int kPairOperand = 128 * kBK * 2;               // 16 KB: this CTA's rows of A or of B
constexpr int kPairStage = 2 * kPairOperand;
constexpr int kPairStaging = 4096;                        // one warp's 32 rows of 128 bytes
constexpr int kPairSmem = kPairStages * kPairStage + 8 * kPairStaging + 1024;
constexpr int kPairThreads = 320;
constexpr int kPairTile = 256;
constexpr int kPairGroupM = 8;      // tiles are walked in bands of eight rows of tiles: L2 keeps both panels

struct PairParams {
  int M, N, K, batch;
  int tiles_m, tiles_n, num_tiles, k_iters;
  int a_mn, b_mn, in_dtype, out_dtype;
  int add;                          // fp32 output: add to C
  float alpha, act_param;
  int act, bias_mode;
  const float* bias;
};

struct PairShared {
  uint64_t full[kPairStages];       // leader: both CTAs' operands have landed
  uint64_t empty[kPairStages];      // each CTA: the MMAs that read the stage have retired
  uint64_t tmem_full[2];            // each CTA
  uint64_t tmem_empty[2];           // leader: 16 epilogue warps (8 of each CTA)
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ bool mbar_wait_bounded_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  uint64_t t0 = 0;
  uint32_t spins = 0;
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (t0 == 0) t0 = globaltimer_ns();
    if ((++spins & 0x3ff) == 0) {
      if (*abort_flag) return false;
      if (globaltimer_ns() - t0 > LB_WAIT_BUDGET_NS) return false;
    }
  }
}
// This CTA's shared memory, bytes counted on a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1,
                                                 int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, uint32_t src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(src), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void tma_add_3d(const CUtensorMap* m, uint32_t src, int c0, int c1, int c2) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(src), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(tmem_d),
      "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate));
}
// Arrives on the barrier at this offset in both CTAs when the MMAs issued so far have retired.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"((uint16_t)3)
      : "memory");
}

struct PairTile {
  int m0, n0, b;
};
__device__ __forceinline__ PairTile pair_tile(const PairParams& p, int t) {
  const int per_batch = p.tiles_m * p.tiles_n;
  PairTile tl;
  tl.b = t / per_batch;
  const int r = t - tl.b * per_batch;
  const int band = r / (kPairGroupM * p.tiles_n), in_band = r - band * (kPairGroupM * p.tiles_n);
  const int height = min(kPairGroupM, p.tiles_m - band * kPairGroupM);
  const int nt = in_band / height;
  tl.m0 = (band * kPairGroupM + (in_band - nt * height)) * kPairTile;
  tl.n0 = nt * kPairTile;
  return tl;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const __grid_constant__ PairParams p, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ PairShared sh;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  volatile int* abort_flag = &sh.abort_flag;
  const int first = (int)blockIdx.x >> 1, step = (int)gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairStages; ++s) {
      mbar_init(smem_u32(&sh.full[s]), 1);
      mbar_init(smem_u32(&sh.empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&sh.tmem_full[a]), 1);
      mbar_init(smem_u32(&sh.tmem_empty[a]), 16);
    }
    sh.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 4 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmC);
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // both CTAs' barriers are initialised before either signals the other's
  tc_fence_after();
  const uint32_t tmem = sh.tmem_base;

  if (warp == 4) {
    if (elect_one()) {
      const uint32_t full0 = map_to_rank(smem_u32(&sh.full[0]), 0);
      RingPos rp;
      uint32_t issued = 0;
      bool ok = true;
      for (int t = first; t < p.num_tiles && ok; t += step) {
        const PairTile tl = pair_tile(p, t);
        const int m0 = tl.m0 + (int)rank * 128, n0 = tl.n0 + (int)rank * 128;
        for (int k = 0; k < p.k_iters; ++k, ++issued) {
          if (!mbar_wait_bounded(smem_u32(&sh.empty[rp.s]), rp.ph ^ 1, abort_flag)) {
            raise_status(status, abort_flag, kTimeoutStageEmpty);
            ok = false;
            break;
          }
          if (rank == 0) mbar_expect_tx(smem_u32(&sh.full[rp.s]), 2 * kPairStage);
          const uint32_t bar = full0 + rp.s * 8u;
          const uint32_t sA = base + rp.s * kPairStage, sB = sA + kPairOperand;
          const int k0 = k * kBK;
          if (!p.a_mn) {
            tma_load_3d_pair(sA, &tmA, bar, k0, m0, tl.b);
          } else {
            tma_load_3d_pair(sA, &tmA, bar, m0, k0, tl.b);
            tma_load_3d_pair(sA + 8192, &tmA, bar, m0 + 64, k0, tl.b);
          }
          if (!p.b_mn) {
            tma_load_3d_pair(sB, &tmB, bar, k0, n0, tl.b);
          } else {
            tma_load_3d_pair(sB, &tmB, bar, n0, k0, tl.b);
            tma_load_3d_pair(sB + 8192, &tmB, bar, n0 + 64, k0, tl.b);
          }
          rp.advance(kPairStages);
        }
      }
      // Every load must have landed before the shared memory goes away.  The MMAs that read a
      // stage wait for it, so this matters only when a role gave up: then the copies of this CTA
      // are let land by time (their barrier may be the other CTA's).
      if (!ok || *abort_flag) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < LB_WAIT_BUDGET_NS / 8) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 5) {
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = make_idesc_f16(p.in_dtype == kBF16 ? 1u : 0u, p.a_mn, p.b_mn, 256, 256);
      const uint64_t da = p.a_mn ? make_smem_desc(0, 8192, 1024, kLayoutSw128) : make_smem_desc(0, 16, 1024, kLayoutSw128);
      const uint64_t db = p.b_mn ? make_smem_desc(0, 8192, 1024, kLayoutSw128) : make_smem_desc(0, 16, 1024, kLayoutSw128);
      const uint32_t a_hi = (uint32_t)(da >> 32), b_hi = (uint32_t)(db >> 32);
      const uint32_t a0 = (uint32_t)da + (base >> 4), b0 = (uint32_t)db + ((base + kPairOperand) >> 4);
      const uint32_t a_step = p.a_mn ? (2048u >> 4) : (32u >> 4), b_step = p.b_mn ? (2048u >> 4) : (32u >> 4);
      RingPos rp, acc;
      bool ok = true;
      for (int t = first; t < p.num_tiles && ok; t += step) {
        if (!mbar_wait_bounded_cluster(smem_u32(&sh.tmem_empty[acc.s]), acc.ph ^ 1, abort_flag)) {
          raise_status(status, abort_flag, kTimeoutTmemEmpty);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem + acc.s * 256;
        for (int k = 0; k < p.k_iters; ++k) {
          if (!mbar_wait_bounded_cluster(smem_u32(&sh.full[rp.s]), rp.ph, abort_flag)) {
            raise_status(status, abort_flag, kTimeoutTmaFull);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a = a0 + rp.s * (kPairStage >> 4), b = b0 + rp.s * (kPairStage >> 4);
#pragma unroll
          for (int kk = 0; kk < kBK / 16; ++kk)
            umma_pair(d, a + kk * a_step, a_hi, b + kk * b_step, b_hi, idesc, (k | kk) ? 1u : 0u);
          umma_commit_pair(smem_u32(&sh.empty[rp.s]));
          rp.advance(kPairStages);
        }
        if (ok) umma_commit_pair(smem_u32(&sh.tmem_full[acc.s]));
        acc.advance(2);
      }
    }
    __syncwarp();
  } else {
    const int eg = warp >= 6 ? 1 : 0, quarter = warp & 3;
    const uint32_t staging = base + kPairStages * kPairStage + (eg * 4 + quarter) * kPairStaging;
    const uint32_t my_row = staging + lane * 128;
    const uint32_t swz = lane & 7;
    const uint32_t empty0 = map_to_rank(smem_u32(&sh.tmem_empty[0]), 0);
    RingPos acc;
    bool ok = true;
    for (int t = first; t < p.num_tiles && ok; t += step, acc.advance(2)) {
      const PairTile tl = pair_tile(p, t);
      LaneBias<128> bias;
      bias.load(p.bias_mode == 1 ? p.bias : nullptr, tl.n0 + eg * 128, p.N, lane);
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&sh.tmem_full[acc.s]), acc.ph, abort_flag));
      if (!ok) {
        if (lane == 0) raise_status(status, abort_flag, kTimeoutTmemFull);
        break;
      }
      tc_fence_after();
      const int row0 = tl.m0 + (int)rank * 128 + quarter * 32;
      const bool rows_ok = row0 < p.M;
      const uint32_t taddr = tmem + acc.s * 256 + (static_cast<uint32_t>(quarter * 32) << 16);
      const float row_bias = (p.bias_mode == 2 && row0 + lane < p.M) ? p.bias[row0 + lane] : 0.f;
      const int width = p.out_dtype == kF32 ? 32 : 64;           // columns of a 128-byte row
      for (int c = eg * 128; c < eg * 128 + 128 && rows_ok; c += width) {
        const int n = tl.n0 + c;
        if (n >= p.N) break;
        uint32_t q[2][32];
        tmem_ld_32x32(taddr + c, q[0]);
        if (width == 64) tmem_ld_32x32(taddr + c + 32, q[1]);
        if (lane == 0) bulk_wait_read<0>();                      // the staging rows have been read
        __syncwarp();
        tmem_ld_wait();
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int h = hh * 32;
          if (h >= width) break;
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(q[hh][j]) * p.alpha + row_bias;
          if (p.bias_mode == 1) bias.add(v, (c - eg * 128 + h) / 32);
          tc_apply_act32(v, p.act, p.act_param);
          if (p.out_dtype == kF32) {
#pragma unroll
            for (int u = 0; u < 8; ++u)
              sts128(my_row + ((u ^ swz) << 4),
                     make_uint4(__float_as_uint(v[4 * u]), __float_as_uint(v[4 * u + 1]), __float_as_uint(v[4 * u + 2]),
                                __float_as_uint(v[4 * u + 3])));
          } else {
            const int u0 = h >> 3;
            const int dt = p.out_dtype;
#pragma unroll
            for (int u = 0; u < 4; ++u)
              sts128(my_row + (((u0 + u) ^ swz) << 4),
                     make_uint4(pack2(v[8 * u], v[8 * u + 1], dt), pack2(v[8 * u + 2], v[8 * u + 3], dt),
                                pack2(v[8 * u + 4], v[8 * u + 5], dt), pack2(v[8 * u + 6], v[8 * u + 7], dt)));
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          if (p.add) tma_add_3d(&tmC, staging, n, row0, tl.b);
          else tma_store_3d(&tmC, staging, n, row0, tl.b);
          bulk_commit();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(empty0 + acc.s * 8u);
    }
    if (lane == 0) bulk_wait_read<0>();      // the rows are written when the grid is through
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // no CTA leaves while the other's MMAs or arrivals may touch its memory
  if (warp == 5) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// Pairs that the device holds at once (0: none).
static int pair_slots() {
  static std::atomic<int> slots[16];
  int dev = 0;
  cudaGetDevice(&dev);
  int n = slots[dev & 15].load();
  if (n == 0) {
    cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = kPairSmem;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    if (n < 1) n = -1;
    slots[dev & 15].store(n);
  }
  return n > 0 ? n : 0;
}

int gemm_pair_slots() { return pair_slots(); }

// The product of lb_gemm_tc for the forms the caller has checked: 16-byte aligned C rows, beta 0
// or (fp32 output) 1.  Returns -2 when the device holds no pair.
int gemm_pair_launch(const void* A, const void* B, void* C, const float* bias, int M, int N, int K, int batch,
                     long long lda, long long ldb, long long ldc, long long strideA, long long strideB,
                     long long strideC, int a_mn, int b_mn, int in_dtype, int out_dtype, float alpha, int add,
                     int bias_mode, int act, float act_param, cudaStream_t stream) {
  const int slots = pair_slots();
  if (slots < 1) return -2;
  PairParams p;
  p.M = M; p.N = N; p.K = K; p.batch = batch;
  p.tiles_m = (M + kPairTile - 1) / kPairTile;
  p.tiles_n = (N + kPairTile - 1) / kPairTile;
  p.num_tiles = p.tiles_m * p.tiles_n * batch;
  p.k_iters = (K + kBK - 1) / kBK;
  p.a_mn = a_mn; p.b_mn = b_mn; p.in_dtype = in_dtype; p.out_dtype = out_dtype;
  p.add = add; p.alpha = alpha; p.act = act; p.act_param = act_param;
  p.bias = bias; p.bias_mode = bias ? bias_mode : 0;
  CUtensorMap tmA, tmB, tmC;
  const uint64_t sa = strideA > 0 ? (uint64_t)strideA : (uint64_t)lda * (a_mn ? K : M);
  const uint64_t sb = strideB > 0 ? (uint64_t)strideB : (uint64_t)ldb * (b_mn ? K : N);
  const uint64_t es = out_dtype == kF32 ? 4 : 2;
  const uint64_t sc = strideC > 0 ? (uint64_t)strideC : (uint64_t)ldc * M;
  {
    uint64_t dims[3] = {(uint64_t)(a_mn ? M : K), (uint64_t)(a_mn ? K : M), (uint64_t)batch};
    uint64_t strides[2] = {(uint64_t)lda * 2, sa * 2};
    uint32_t box[3] = {64, a_mn ? 64u : 128u, 1};
    if (!lbhost::encode_tmap(&tmA, in_dtype, 3, A, dims, strides, box, nullptr, 128)) return -1;
  }
  {
    uint64_t dims[3] = {(uint64_t)(b_mn ? N : K), (uint64_t)(b_mn ? K : N), (uint64_t)batch};
    uint64_t strides[2] = {(uint64_t)ldb * 2, sb * 2};
    uint32_t box[3] = {64, b_mn ? 64u : 128u, 1};
    if (!lbhost::encode_tmap(&tmB, in_dtype, 3, B, dims, strides, box, nullptr, 128)) return -1;
  }
  {
    uint64_t dims[3] = {(uint64_t)N, (uint64_t)M, (uint64_t)batch};
    uint64_t strides[2] = {(uint64_t)ldc * es, sc * es};
    uint32_t box[3] = {(uint32_t)(128 / es), 32, 1};
    if (!lbhost::encode_tmap(&tmC, out_dtype, 3, C, dims, strides, box, nullptr, 128)) return -1;
  }
  const int pairs = p.num_tiles < slots ? p.num_tiles : slots;
  gemm_pair_kernel<<<2 * pairs, kPairThreads, kPairSmem, stream>>>(tmA, tmB, tmC, p, lbhost::status_word());
  return (int)cudaGetLastError();
}

}  // namespace lb
