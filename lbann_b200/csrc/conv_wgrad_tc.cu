// tcgen05 filter-gradient kernel for channels-last convolutions:
//
//   dW[tap][k][c] += alpha * sum_pixels dy[pixel][k] * x[pixel*stride - pad + tap*dil][c]
//
// GEMM view: the reduction runs over output pixels, 64 at a time (one TMA brick per
// pipeline stage); both operands are "MN-major" (pixel rows, channels contiguous), so
// x and dy are consumed exactly as they sit in memory.  The accumulator rows stack
// several (tap, channel-block) slices: with Cb = 16/32/64 channels per slice an M = 128
// accumulator holds 8/4/2 slices.  Where the sizes allow it, all taps of a brick are read
// from one halo slab of x (conv_wgrad_slab_kernel).  The pixel range is split over CTAs, whose
// partial results go to a workspace; wgrad_reduce_kernel adds them up and into the (pre-scaled)
// gradient buffer, matching the reference's dst_scale / grad_scale accumulation contract
// (src/layers/learning/base_convolution.cpp:1397-1445).
#include <algorithm>

#include "common.cuh"

namespace lb {

struct WgradGeom {
  int N, D, H, W, C;
  int Do, Ho, Wo, Kout;
  int kd, kh, kw;
  int pd, ph, pw;
  int sd, sh, sw;
  int dd, dh, dw;
};

constexpr int kWgSlabGroups = 8, kWgSlabSteps = 8, kWgSlabMost = 64;

struct WgradParams {
  WgradGeom g;
  int TW, TH, TD, TN, rows_used;        // pixel brick (<= 64 rows)
  int bricks_w, bricks_h, bricks_d, bricks_n, bricks_total;
  int Cb, cblocks, slices_total, spg;   // spg = slices per accumulator = 128 / Cb
  int groups_total, G, group_sets;      // G accumulators per CTA
  int parts, room;                      // a CTA's bricks are summed in parts, room of them at a time in TMEM
  int BN, n_tiles, splits;
  int a_layout, b_layout;
  int stage_bytes, stages, a_bytes;     // a_bytes = G * 16384
  int tmem_cols, in_dtype;
  float alpha;
  float* dW;
  long long s_tap, s_k, s_c;            // output strides in elements
  float* ws;                            // partial sums: [CTA][G * BN / 4][128 rows][4]
  FastDiv fd_bw, fd_bh, fd_bd;          // brick decode without run-time divisions
  // Taps from one halo slab a brick (conv_wgrad_slab_kernel); 0: a box for every tap
  int slab, runs, group_sets_c;         // full accumulators a tap column, sets of accumulators a channel block
  // low words of the operands' descriptors, computed on the host (constants are uniform operands): an
  // accumulator's taps, a step's pixels in the slab and in dy
  uint32_t ga[kWgSlabMost], ka[kWgSlabSteps], kb[kWgSlabSteps];
};

// Accumulator of a channel block and slice in it that hold tap (a, b, c) of the slab kernel: slices of an
// accumulator are equally far apart in the slab.  Along j = b * kd + a full ones, then what is left of
// the kd * kh along c.
__device__ __forceinline__ void wgrad_slab_slot(int kd, int kw, int runs, int log_spg, int a, int b, int c, int& grp, int& slot) {
  const int j = b * kd + a, full = runs << log_spg, last = (1 << log_spg) - 1;
  if (j < full) {
    grp = c * runs + (j >> log_spg);
    slot = j & last;
  } else {
    grp = kw * runs + (j - full) * ((kw + last) >> log_spg) + (c >> log_spg);
    slot = c & last;
  }
}

struct WgradShared {
  uint64_t full[4];
  uint64_t empty[4];
  uint64_t done;                        // the accumulators of a round are complete
  uint64_t drained;                     // ... and have been read by the four epilogue warps
  uint32_t tmem_base;
  int abort_flag;
};

// Epilogue of both kernels (warps 0 to 3): per round, add the parts up and store the sums, or add them at
// the L2 to those of the rounds before.
// Four consecutive columns of a row are one 16-byte unit and the units of a column group
// lie row by row, so a warp stores 512 contiguous bytes.  (fp32 atomics straight into dW,
// whose rows are taps * 4 bytes apart, touched one sector per lane: with 296 CTAs adding
// 64 x 64 x 9 weights each that tail took three quarters of the kernel.)
__device__ __forceinline__ void wgrad_epilogue(const WgradParams& p, WgradShared& sh, uint32_t tmem_base, int my_bricks,
                                               int per_part, int g_count, int n0, int* status) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &sh.abort_flag;
  const int used = (my_bricks + per_part - 1) / per_part;          // a CTA of few bricks has fewer parts
  const int row = warp * 32 + lane;
  float4* out = reinterpret_cast<float4*>(p.ws) + (size_t)blockIdx.x * (p.G * p.BN * 32) + row;
  for (int round = 0; round * p.room < used; ++round) {
    const int here = min(p.room, used - round * p.room);
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&sh.done), round & 1, abort_flag))) {
      if (lane == 0) raise_status(status, abort_flag, kTimeoutTmemFull);
      break;
    }
    tc_fence_after();
    for (int gi = 0; gi < g_count; ++gi) {
      for (int c = 0; c < p.BN; c += 32) {
        if (n0 + c >= p.g.Kout) break;
        const uint32_t from = tmem_base + gi * p.BN + c + ((uint32_t)(warp * 32) << 16);
        uint32_t r[32];
        tmem_ld_32x32(from, r);
        tmem_ld_wait();
        for (int part = 1; part < here; ++part) {
          uint32_t q[32];
          tmem_ld_32x32(from + part * (p.G * p.BN), q);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(q[j]));
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float4* at = out + ((gi * p.BN + c) / 4 + j) * 128;
          const float4 f = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                       __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
          if (round == 0) __stcg(at, f);
          else atomicAdd(at, f);             // by the thread that stored it: one order
        }
      }
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&sh.drained));
  }
}

__global__ void __launch_bounds__(192, 1)
conv_wgrad_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmDy,
                  const WgradParams p, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ WgradShared sh;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &sh.abort_flag;
  const int S = p.stages;

  // Rows of a stage that no TMA box covers must read as zero: they are part of the
  // reduction.  TMA only ever writes the first rows_used rows, so one clear suffices.
  if (p.rows_used < 64) {
    uint8_t* base = smem_raw + (smem_base - smem_u32(smem_raw));
    uint4* q = reinterpret_cast<uint4*>(base);
    const int n16 = S * p.stage_bytes / 16;
    for (int i = threadIdx.x; i < n16; i += blockDim.x) q[i] = make_uint4(0, 0, 0, 0);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(smem_u32(&sh.full[s]), 1);
      mbar_init(smem_u32(&sh.empty[s]), 1);
    }
    mbar_init(smem_u32(&sh.done), 1);
    mbar_init(smem_u32(&sh.drained), 4);
    sh.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 5) {
    tmem_alloc(smem_u32(&sh.tmem_base), p.tmem_cols);
    tmem_relinquish();
  }
  // make the generic-proxy zero fill visible to the async proxy (TMA / MMA reads)
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh.tmem_base;

  // work decomposition
  int wi = blockIdx.x;
  const int split = wi % p.splits; wi /= p.splits;
  const int nt = wi % p.n_tiles;   wi /= p.n_tiles;
  const int gs = wi;
  const int n0 = nt * p.BN;
  const int g_first = gs * p.G;
  const int g_count = min(p.G, p.groups_total - g_first);
  const WgradGeom& g = p.g;
  const int my_bricks = (p.bricks_total - split + p.splits - 1) / p.splits;
  const int per_part = (my_bricks + p.parts - 1) / p.parts;

  if (warp == 4) {
    // The whole warp walks the bricks: lane 0 owns the barrier protocol, and the
    // boxes of one stage go out from different lanes so that they enter the
    // copy engine side by side instead of one after another.  What a lane loads is
    // the same for every brick (which box, which tap, which channel block), so it is
    // worked out once; per brick only the brick origin changes.
    uint32_t it = 0;
    bool ok = true;
    // slices this CTA loads per brick (the same for every brick)
    int nsl = 0;
    for (int gi = 0; gi < g_count; ++gi)
      nsl += min(p.spg, p.slices_total - (g_first + gi) * p.spg);
    const int ndy = p.BN == 32 ? 1 : p.BN / 64;
    const int njobs = ndy + g_count * p.spg;
    // this lane's jobs q = lane, lane + 32 (at most two: njobs <= 4 + 4 * 8)
    struct Job { int kind; uint32_t dst; int c0, ow, oh, od; };   // kind 0 none, 1 dy box, 2 x slice
    Job jobs[2];
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      const int q = lane + 32 * jj;
      Job jb = {0, 0u, 0, 0, 0, 0};
      if (q < ndy) {
        jb.kind = 1; jb.dst = (uint32_t)p.a_bytes + q * 8192u; jb.c0 = n0 + q * 64;
      } else if (q < njobs) {
        const int gi = (q - ndy) / p.spg, j = (q - ndy) - gi * p.spg;
        const int sl = (g_first + gi) * p.spg + j;
        if (sl < p.slices_total) {
          const int tap = sl / p.cblocks;
          const int ta = tap / (g.kh * g.kw), tb = (tap / g.kw) % g.kh, tc = tap % g.kw;
          jb.kind = 2; jb.dst = gi * 16384u + j * (64u * p.Cb * 2u);
          jb.c0 = (sl - tap * p.cblocks) * p.Cb;
          jb.ow = tc * g.dw - g.pw; jb.oh = tb * g.dh - g.ph; jb.od = ta * g.dd - g.pd;
        }
      }
      jobs[jj] = jb;
    }
    const uint32_t tx_bytes = (uint32_t)(p.rows_used * 2 * (nsl * p.Cb + p.BN));
    RingPos rp;
    for (int b = split; b < p.bricks_total && ok; b += p.splits, ++it) {
      uint32_t r, bw, bh, bd, nb;
      p.fd_bw.divmod((uint32_t)b, r, bw);
      p.fd_bh.divmod(r, r, bh);
      p.fd_bd.divmod(r, nb, bd);
      const int w0 = bw * p.TW, h0 = bh * p.TH, d0 = bd * p.TD, nn0 = nb * p.TN;
      const uint32_t sA = smem_base + rp.s * p.stage_bytes;
      const uint32_t bar = smem_u32(&sh.full[rp.s]);
      int go = 1;
      if (lane == 0) {
        if (!mbar_wait_bounded(smem_u32(&sh.empty[rp.s]), rp.ph ^ 1, abort_flag)) {
          raise_status(status, abort_flag, kTimeoutStageEmpty);
          go = 0;
        } else {
          // every slice brings rows_used * Cb * 2 bytes, dy brings rows_used * BN * 2
          mbar_expect_tx(bar, tx_bytes);
        }
      }
      go = __shfl_sync(0xffffffffu, go, 0);
      if (!go) {
        ok = false;
        break;
      }
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const Job& jb = jobs[jj];
        if (jb.kind == 1) {
          tma_load_5d(sA + jb.dst, &tmDy, bar, jb.c0, w0, h0, d0, nn0);
        } else if (jb.kind == 2) {
          tma_load_5d(sA + jb.dst, &tmX, bar, jb.c0, w0 * g.sw + jb.ow, h0 * g.sh + jb.oh,
                      d0 * g.sd + jb.od, nn0);
        }
      }
      __syncwarp();
      rp.advance((uint32_t)S);
    }
    if (lane == 0) {
      if (!ok || *abort_flag) {
        const uint32_t pending = it < (uint32_t)S ? it : (uint32_t)S;
        for (uint32_t j = 0; j < pending; ++j) {
          const uint32_t q = it - 1 - j;
          mbar_wait_budget_only(smem_u32(&sh.full[q % S]), (q / S) & 1);
        }
      }
    }
  } else if (warp == 5) {
    if (elect_one()) {
      // descriptors differ in the start-address field of the low word only; four MMAs per
      // accumulator and stage, issued straight-line (see slab_issue_plane for why)
      const uint32_t idesc =
          make_idesc_f16(p.in_dtype == kBF16 ? 1u : 0u, 1, 1, 128, (uint32_t)p.BN);
      const uint32_t a_lbo = 64u * p.Cb * 2u, a_sbo = 8u * p.Cb * 2u, a_adv = (16u * p.Cb * 2u) >> 4;
      const uint32_t b_row = (p.BN == 32) ? 64u : 128u;
      const uint32_t b_lbo = 8192u, b_sbo = 8u * b_row, b_adv = (16u * b_row) >> 4;
      const uint64_t a_desc = make_smem_desc(0, a_lbo, a_sbo, p.a_layout);
      const uint64_t b_desc = make_smem_desc(0, b_lbo, b_sbo, p.b_layout);
      const uint32_t a_lo0 = (uint32_t)a_desc, a_hi = (uint32_t)(a_desc >> 32);
      const uint32_t b_lo0 = (uint32_t)b_desc, b_hi = (uint32_t)(b_desc >> 32);
      const uint32_t stage_step = (uint32_t)p.stage_bytes >> 4;
      const uint32_t a_base = a_lo0 + (smem_base >> 4);
      const uint32_t b_base = b_lo0 + ((smem_base + (uint32_t)p.a_bytes) >> 4);
      const uint32_t BNu = (uint32_t)p.BN;
      uint32_t accum = 0, acc = tmem_base;
      int left = per_part, set = 0;                   // bricks until the next part, its place in TMEM
      uint32_t round = 0;
      bool ok = true;
      RingPos rp;
      for (int b = split; b < p.bricks_total && ok; b += p.splits) {
        if (left == 0) {
          if (++set == p.room) {
            umma_commit(smem_u32(&sh.done));
            if (!mbar_wait_bounded(smem_u32(&sh.drained), round++ & 1u, abort_flag)) {
              raise_status(status, abort_flag, kTimeoutTmemEmpty);
              ok = false;
              break;
            }
            set = 0;
          }
          acc = tmem_base + (uint32_t)(set * p.G * p.BN);
          accum = 0;
          left = per_part;
        }
        --left;
        if (!mbar_wait_bounded(smem_u32(&sh.full[rp.s]), rp.ph, abort_flag)) {
          raise_status(status, abort_flag, kTimeoutTmaFull);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = a_base + rp.s * stage_step, sb = b_base + rp.s * stage_step;
#pragma unroll
        for (int gi = 0; gi < 4; ++gi) {
          if (gi < g_count) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_f16_lo(acc + gi * BNu, sa + gi * 1024u + kk * a_adv, a_hi, sb + kk * b_adv,
                          b_hi, idesc, kk == 0 ? accum : 1u);   // the first MMA of an accumulator overwrites
          }
        }
        accum = 1u;
        umma_commit(smem_u32(&sh.empty[rp.s]));
        rp.advance((uint32_t)S);
      }
      if (ok) umma_commit(smem_u32(&sh.done));
    }
  } else {
    wgrad_epilogue(p, sh, tmem_base, my_bricks, per_part, g_count, n0, status);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
}

// ------------------------------------------------------------------ taps from one halo slab a brick
// The same sums for filters of several taps, stride and dilation 1.  The kernel above brings the pixels of a
// brick once for every tap, so 32 -> 64 channels and 27 taps cost 118 KB of copies per 64 pixels where an SM takes in
// about 58 bytes a cycle: 2480 cycles for MMAs worth 1344.  Here ONE box brings the brick with its
// halo, lines of [kd planes][TW + kw - 1 pixels], and a tap is an offset of whole pixel rows into it: 29 to 46 KB.
// The slices of an accumulator (128 / Cb of them) are one operand, so they have to be equally far apart:
// taps of one column c follow one another at the distance of a plane, across lines as well (planes lie inside lines).
// A brick has TW x TH output pixels of one plane, whole groups of eight along W; a step of the
// reduction takes two groups side by side, or from two lines where TW / 8 is odd.
// 8 x 64^3, 32 -> 64 channels, fp16: 387 -> 219 us; the MMAs (58 cycles at N = 64) take 188 of them.
template <int KS>
__device__ __forceinline__ void wgrad_slab_issue(uint32_t acc, uint32_t BN, int g_first, int g_count, const WgradParams& p,
                                                 uint32_t a_stage, uint32_t b_stage, uint32_t a_hi, uint32_t b_hi,
                                                 uint32_t idesc, uint32_t accum) {
#pragma unroll
  for (int gi = 0; gi < kWgSlabGroups; ++gi) {
    if (gi < g_count) {
      const uint32_t a = p.ga[g_first + gi] + a_stage;
#pragma unroll
      for (int kk = 0; kk < KS; ++kk)
        umma_f16_lo(acc + gi * BN, a + p.ka[kk], a_hi, p.kb[kk] + b_stage, b_hi, idesc, kk == 0 ? accum : 1u);
    }
  }
}

__global__ void __launch_bounds__(192, 1)
conv_wgrad_slab_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmDy,
                       const WgradParams p, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ WgradShared sh;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5;
  volatile int* abort_flag = &sh.abort_flag;
  const int S = p.stages;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(smem_u32(&sh.full[s]), 1);
      mbar_init(smem_u32(&sh.empty[s]), 1);
    }
    mbar_init(smem_u32(&sh.done), 1);
    mbar_init(smem_u32(&sh.drained), 4);
    sh.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 5) {
    tmem_alloc(smem_u32(&sh.tmem_base), p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh.tmem_base;

  int wi = blockIdx.x;
  const int split = wi % p.splits; wi /= p.splits;
  const int nt = wi % p.n_tiles;   wi /= p.n_tiles;
  const int gs = wi % p.group_sets_c, cb = wi / p.group_sets_c;
  const int n0 = nt * p.BN;
  const int g_first = gs * p.G, g_count = min(p.G, p.groups_total - g_first);
  const WgradGeom& g = p.g;
  const int my_bricks = (p.bricks_total - split + p.splits - 1) / p.splits;
  const int per_part = (my_bricks + p.parts - 1) / p.parts;

  if (warp == 4) {
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      const int ndy = p.BN == 32 ? 1 : p.BN / 64;
      const uint32_t pixels = (uint32_t)(p.TW * p.TH);
      const uint32_t tx_bytes = (uint32_t)((p.TH + g.kh - 1) * g.kd * (p.TW + g.kw - 1) * p.Cb * 2) + pixels * p.BN * 2u;
      RingPos rp;
      for (int b = split; b < p.bricks_total; b += p.splits, ++it) {
        uint32_t r, bw, bh, d, n;
        p.fd_bw.divmod((uint32_t)b, r, bw);
        p.fd_bh.divmod(r, r, bh);
        p.fd_bd.divmod(r, n, d);
        const int w0 = (int)bw * p.TW, h0 = (int)bh * p.TH;
        if (!mbar_wait_bounded(smem_u32(&sh.empty[rp.s]), rp.ph ^ 1, abort_flag)) {
          raise_status(status, abort_flag, kTimeoutStageEmpty);
          ok = false;
          break;
        }
        const uint32_t sA = smem_base + rp.s * p.stage_bytes, bar = smem_u32(&sh.full[rp.s]);
        mbar_expect_tx(bar, tx_bytes);
        tma_load_5d(sA, &tmX, bar, cb * p.Cb, w0 - g.pw, (int)d - g.pd, h0 - g.ph, (int)n);
        for (int q = 0; q < ndy; ++q)
          tma_load_5d(sA + p.a_bytes + q * (pixels * 128u), &tmDy, bar, n0 + q * 64, w0, h0, (int)d, (int)n);
        rp.advance((uint32_t)S);
      }
      if (!ok || *abort_flag) {
        const uint32_t pending = it < (uint32_t)S ? it : (uint32_t)S;
        for (uint32_t j = 0; j < pending; ++j) {
          const uint32_t q = it - 1 - j;
          mbar_wait_budget_only(smem_u32(&sh.full[q % S]), (q / S) & 1);
        }
      }
    }
  } else if (warp == 5) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_f16(p.in_dtype == kBF16 ? 1u : 0u, 1, 1, 128, (uint32_t)p.BN);
      const uint32_t rb = p.Cb * 2u, brow = p.BN == 32 ? 64u : 128u;
      const uint32_t line = (uint32_t)(p.TW + g.kw - 1) * g.kd;       // pixel rows
      const bool pair = p.TW % 16 != 0;             // a step's two groups of eight come from two lines
      const uint64_t a_desc = make_smem_desc(smem_base, 0, pair ? line * rb : 8 * rb, p.a_layout);
      const uint64_t b_desc = make_smem_desc(smem_base + p.a_bytes, p.TW * p.TH * brow, pair ? p.TW * brow : 8 * brow, p.b_layout);
      const uint32_t a_hi = (uint32_t)(a_desc >> 32), b_hi = (uint32_t)(b_desc >> 32);
      const uint32_t a_lo = (uint32_t)a_desc, b_lo = (uint32_t)b_desc;
      const int steps = p.TW * p.TH / 16;
      const uint32_t stage_step = (uint32_t)p.stage_bytes >> 4, BNu = (uint32_t)p.BN;
      uint32_t accum = 0, acc = tmem_base;
      int left = per_part, set = 0;                 // bricks until the next part, its place in TMEM
      uint32_t round = 0;
      bool ok = true;
      RingPos rp;
      for (int b = split; b < p.bricks_total; b += p.splits) {
        if (left == 0) {
          if (++set == p.room) {
            umma_commit(smem_u32(&sh.done));
            if (!mbar_wait_bounded(smem_u32(&sh.drained), round++ & 1u, abort_flag)) {
              raise_status(status, abort_flag, kTimeoutTmemEmpty);
              ok = false;
              break;
            }
            tc_fence_after();
            set = 0;
          }
          acc = tmem_base + (uint32_t)(set * p.G * p.BN);
          accum = 0;
          left = per_part;
        }
        --left;
        if (!mbar_wait_bounded(smem_u32(&sh.full[rp.s]), rp.ph, abort_flag)) {
          raise_status(status, abort_flag, kTimeoutTmaFull);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t stage = rp.s * stage_step;
#define LB_STEPS(KS) case KS: wgrad_slab_issue<KS>(acc, BNu, g_first, g_count, p, a_lo + stage, b_lo + stage, a_hi, b_hi, idesc, accum); break;
        switch (steps) {
          LB_STEPS(1) LB_STEPS(2) LB_STEPS(3) LB_STEPS(4) LB_STEPS(5) LB_STEPS(6) LB_STEPS(7) LB_STEPS(8)
        }
#undef LB_STEPS
        accum = 1u;
        umma_commit(smem_u32(&sh.empty[rp.s]));
        rp.advance((uint32_t)S);
      }
      if (ok) umma_commit(smem_u32(&sh.done));
    }
  } else {
    wgrad_epilogue(p, sh, tmem_base, my_bricks, per_part, g_count, n0, status);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
}

// dW += alpha * sum over the splits of the partial sums.  A block owns four filters (one 16-byte
// unit of the partials), CH channels and NT taps; its threads are these items times `groups` groups of
// splits, so that CH lanes load contiguous bytes and the stores (filter layout: taps innermost) are runs
// of taps, through shared memory.  Large filters are bound by the bytes (a division by a run-time number
// for every index took as long: 512 x 512 x 9 21 -> 16 us), small ones by the latency of a thread's loads:
// eight are in flight, and the launch cuts the splits into as many groups as fill the GPU with threads
// (64 x 32 x 27, 148 splits: 20 -> 8 us).
constexpr int kRedThreads = 256;
struct WgradReduce {
  int log_ch, NT, groups, items;                                   // items = NT << log_ch
  int log_cb, log_spg;
  FastDiv fd_items, fd_nt, fd_kw, fd_khkw, fd_G;
};

__global__ void __launch_bounds__(kRedThreads)
wgrad_reduce_kernel(const WgradParams p, const WgradReduce q) {
  __shared__ float4 part[kRedThreads];
  const WgradGeom& g = p.g;
  const int taps = g.kd * g.kh * g.kw;
  const int k0 = blockIdx.x * 4, c0 = blockIdx.y << q.log_ch, t0 = blockIdx.z * q.NT;
  const int n_tile = k0 / p.BN, col = k0 - n_tile * p.BN;
  const size_t cta_stride = (size_t)p.G * p.BN * 32;               // in float4
  const int sg = (int)q.fd_items.div(threadIdx.x), i = threadIdx.x - sg * q.items;
  const int tap = t0 + (i >> q.log_ch), ch = c0 + (i & ((1 << q.log_ch) - 1)), cb = ch >> q.log_cb;
  if (sg < q.groups && tap < taps && ch < g.C) {
    int grp, slot, set;
    if (p.slab) {
      uint32_t a, r, b, c;
      q.fd_khkw.divmod((uint32_t)tap, a, r);
      q.fd_kw.divmod(r, b, c);
      wgrad_slab_slot(p.g.kd, p.g.kw, p.runs, q.log_spg, (int)a, (int)b, (int)c, grp, slot);
      set = cb * p.group_sets_c;
    } else {
      const int sl = tap * p.cblocks + cb;
      grp = sl >> q.log_spg;
      slot = sl & ((1 << q.log_spg) - 1);
      set = 0;
    }
    uint32_t gs, gi;
    q.fd_G.divmod((uint32_t)grp, gs, gi);
    const int row = (slot << q.log_cb) + ch - (cb << q.log_cb);
    const int s0 = sg * p.splits / q.groups, s1 = (sg + 1) * p.splits / q.groups;
    const float4* src = reinterpret_cast<const float4*>(p.ws) + ((size_t)((set + gs) * p.n_tiles + n_tile) * p.splits + s0) * cta_stride +
                        ((gi * p.BN + col) / 4) * 128 + row;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = s0; s < s1; s += 8, src += 8 * cta_stride) {
      float4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = s + j < s1 ? __ldcg(src + j * cta_stride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 8; ++j) { a.x += v[j].x; a.y += v[j].y; a.z += v[j].z; a.w += v[j].w; }
    }
    part[threadIdx.x] = a;
  }
  __syncthreads();
  // element e of the output order: filter, channel, tap (adjacent in a packed filter)
  for (int e = threadIdx.x; e < 4 * q.items; e += kRedThreads) {
    uint32_t kk, r, chl, tl;
    q.fd_items.divmod((uint32_t)e, kk, r);
    q.fd_nt.divmod(r, chl, tl);
    const int k = k0 + (int)kk, c = c0 + (int)chl, t = t0 + (int)tl;
    if (k >= g.Kout || c >= g.C || t >= taps) continue;
    const float* from = reinterpret_cast<const float*>(&part[(tl << q.log_ch) + chl]) + kk;
    float v = 0.f;
    for (int j = 0; j < q.groups; ++j) v += from[4 * j * q.items];
    atomicAdd(p.dW + t * p.s_tap + k * p.s_k + c * p.s_c, p.alpha * v);
  }
}

static int wg_largest_tile(int extent, int limit) {
  if (extent <= limit) return extent;
  int best = 1;
  for (int t = limit; t >= 1; --t)
    if (extent % t == 0) { best = t; break; }
  return best * 2 > limit ? best : limit;
}

// What a plan costs besides its bricks: the first stage's copies, the sums' way to the workspace (about
// 40 B/clk an SM) and back through the reduction (30).
static double wgrad_ends(int stage_bytes, int G, int BN, long long ctas, long long waves) {
  return waves * (stage_bytes / 58.0 + G * BN * 512 / 40.0) + (double)ctas * G * BN * 512 / (30.0 * lbhost::sm_count());
}

// The slab kernel's tiling, taken where its estimate is the shorter one.  `terms`: what an accumulator may
// sum; `best`: the estimate for the plan in p.  345 cycles a stage beside its MMAs are a fit to the times below
// (8 x 64^3, 32 -> 64: the tensor pipe is active for 55 % of the cycles, shared memory for 83).
// With their reductions, bf16 / fp16, a box for every tap / slabs: 8 x 64^3, 32 -> 64 channels 402 / 227 us;
// 45 x 52 x 60, 32 -> 64 47 / 36; 32 x 56^2, 64 -> 64 26 / 21; 8 x 32^3, 64 -> 128 120 / 113; the other way
// 16^3, 64 -> 128 14 / 17 (two bricks of 110 KB a CTA), 12^3, 256 -> 64 15 / 20.
static void wgrad_slab_plan(WgradParams& p, int mma, long long terms, double best) {
  const WgradGeom& g = p.g;
  if (g.sd != 1 || g.sh != 1 || g.sw != 1 || g.dd != 1 || g.dh != 1 || g.dw != 1) return;
  const int J = g.kd * g.kh, taps = J * g.kw, sms = lbhost::sm_count();
  if (taps == 1 || g.kd > 255 || g.kh > 128 || g.kw > 128) return;
  WgradParams q = p;
  q.runs = J / p.spg;
  q.groups_total = g.kw * q.runs + (J - q.runs * p.spg) * ((g.kw + p.spg - 1) / p.spg);
  if (q.groups_total > kWgSlabMost) return;
  const int g_most = std::min(512 / p.BN, kWgSlabGroups);
  q.group_sets_c = (q.groups_total + g_most - 1) / g_most;
  q.G = (q.groups_total + q.group_sets_c - 1) / q.group_sets_c;
  q.group_sets = q.group_sets_c * p.cblocks;
  const int base = q.group_sets * p.n_tiles;
  for (int TW = 8; TW <= 64; TW += 8) {
    if (TW - 8 >= g.Wo) break;
    for (int TH = 1; TW * TH <= 16 * kWgSlabSteps && TH - 1 < g.Ho; ++TH) {
      if (TW * TH % 16 || (TW % 16 && TH % 2)) continue;
      const long long rows = (long long)(TH + g.kh - 1) * g.kd * (TW + g.kw - 1);
      const long long slab = (rows * p.Cb * 2 + 1023) & ~1023ll, dy = (long long)TW * TH * p.BN * 2;
      const long long stage = (slab + dy + 1023) & ~1023ll;
      // a slice that no tap fills reads up to 8 pixels behind the slab: dy or the next stage
      const long long stages = std::min(4ll, (232448 - 2048) / stage);
      if (stages < 2) continue;
      const long long bricks = (long long)((g.Wo + TW - 1) / TW) * ((g.Ho + TH - 1) / TH) * g.Do * g.N;
      const long long most = std::max({(long long)(g.Wo + TW - 1) / TW, (long long)(g.Ho + TH - 1) / TH, (long long)g.Do});
      if (bricks * most >= (1ll << 32) || bricks >= (1ll << 31)) continue;
      long long splits = base < sms ? sms / base : 1;
      splits = std::max(1ll, std::min(splits, (bricks + 1) / 2));
      const long long per_cta = (bricks + splits - 1) / splits;
      const long long pixels = ((long long)g.Wo * g.Ho * g.Do * g.N * per_cta + bricks - 1) / bricks;     // a CTA's, on average
      const long long parts = std::min(per_cta, (pixels + terms - 1) / terms);
      const long long room = std::min<long long>(parts, 512 / (q.G * p.BN));
      const long long rounds = (parts + room - 1) / room, waves = (base * splits + sms - 1) / sms;
      const double brick = std::max(stage / 58.0, (double)q.G * (TW * TH / 16) * mma) * (stages >= 3 ? 1.0 : 1.05) + 345.0;
      const double store = (double)base * splits * (rounds - 1) * q.G * p.BN * 512 / (21.0 * sms);
      const double cost = waves * (per_cta * brick + 3000.0 * rounds) + store + wgrad_ends((int)stage, q.G, p.BN, base * splits, waves);
      if (cost < best) {
        best = cost;
        p = q;
        p.slab = 1;
        p.TW = TW; p.TH = TH; p.TD = p.TN = 1; p.rows_used = TW * TH;
        p.bricks_w = (g.Wo + TW - 1) / TW; p.bricks_h = (g.Ho + TH - 1) / TH; p.bricks_d = g.Do; p.bricks_n = g.N;
        p.bricks_total = (int)bricks;
        p.fd_bw = FastDiv((uint32_t)p.bricks_w); p.fd_bh = FastDiv((uint32_t)p.bricks_h); p.fd_bd = FastDiv((uint32_t)g.Do);
        p.splits = (int)splits; p.parts = (int)parts; p.room = (int)room;
        p.stages = (int)stages; p.stage_bytes = (int)stage; p.a_bytes = (int)slab;
      }
    }
  }
}

// Offsets of the slab kernel's operands, in 16-byte units; the distance of an accumulator's slices above them.
static void wgrad_slab_offsets(WgradParams& p) {
  const WgradGeom& g = p.g;
  const int rb = p.Cb * 2, brow = p.BN == 32 ? 64 : 128, plane = p.TW + g.kw - 1, line = plane * g.kd;
  const int rest = (g.kw + p.spg - 1) / p.spg;      // accumulators of a line that is left over
  for (int grp = 0; grp < p.groups_total; ++grp) {
    const int main = g.kw * p.runs;
    const bool along = grp < main;
    const int c = along ? grp / p.runs : (grp - main) % rest * p.spg;
    const int j = along ? grp % p.runs * p.spg : p.runs * p.spg + (grp - main) / rest;
    p.ga[grp] = (uint32_t)((j * plane + c) * rb / 16) + ((uint32_t)((along ? plane : 1) * rb / 16) << 16);
  }
  const bool pair = p.TW % 16 != 0;
  const int per_line = pair ? p.TW / 8 : p.TW / 16;
  for (int kk = 0; kk < kWgSlabSteps; ++kk) {
    const int y = kk / per_line * (pair ? 2 : 1), x = kk % per_line * (pair ? 8 : 16);
    p.ka[kk] = (uint32_t)((y * line + x) * rb / 16);
    p.kb[kk] = (uint32_t)((y * p.TW + x) * brow / 16);
  }
}

// Tiling of a filter gradient; a function of the sizes only.  False: not covered.
static bool wgrad_plan(WgradParams& p) {
  const WgradGeom& g = p.g;
  p.slab = p.runs = p.group_sets_c = 0;
  if (g.C % 8 || g.Kout % 8) return false;
  p.Cb = g.C >= 64 ? 64 : (g.C >= 32 ? 32 : 16);
  p.cblocks = (g.C + p.Cb - 1) / p.Cb;
  p.slices_total = g.kd * g.kh * g.kw * p.cblocks;
  p.spg = 128 / p.Cb;
  p.groups_total = (p.slices_total + p.spg - 1) / p.spg;
  p.BN = g.Kout > 128 ? 256 : (g.Kout > 64 ? 128 : (g.Kout > 32 ? 64 : 32));
  p.n_tiles = (g.Kout + p.BN - 1) / p.BN;
  p.a_layout = p.Cb == 64 ? kLayoutSw128 : (p.Cb == 32 ? kLayoutSw64 : kLayoutSw32);
  p.b_layout = p.BN == 32 ? kLayoutSw64 : kLayoutSw128;

  p.TW = wg_largest_tile(g.Wo, 64);
  p.TH = wg_largest_tile(g.Ho, 64 / p.TW);
  p.TD = wg_largest_tile(g.Do, 64 / (p.TW * p.TH));
  p.TN = wg_largest_tile(g.N, 64 / (p.TW * p.TH * p.TD));
  p.rows_used = p.TW * p.TH * p.TD * p.TN;
  p.bricks_w = (g.Wo + p.TW - 1) / p.TW;
  p.bricks_h = (g.Ho + p.TH - 1) / p.TH;
  p.bricks_d = (g.Do + p.TD - 1) / p.TD;
  p.bricks_n = (g.N + p.TN - 1) / p.TN;
  p.bricks_total = p.bricks_w * p.bricks_h * p.bricks_d * p.bricks_n;
  if ((long long)p.bricks_total * 256 >= (1ll << 32)) return false;
  p.fd_bw = FastDiv((uint32_t)p.bricks_w);
  p.fd_bh = FastDiv((uint32_t)p.bricks_h);
  p.fd_bd = FastDiv((uint32_t)p.bricks_d);

  // Accumulators per CTA (G) and splits of the pixels: the choice with the shortest longest CTA.
  // A brick costs its bytes at the ~58 B/clk that an SM's copies bring in (or ~75 cycles per
  // box), or its MMAs (44 / 48 / 64 / 128 cycles at N = 32 / 64 / 128 / 256), whichever is
  // longer; with two stages in flight part of the copies' latency shows, with one all of it.
  // The workspace (CTAs x G x BN rows) is bounded by the CTAs that the device holds, except where the
  // filter alone needs more of them.
  const int sms = lbhost::sm_count();
  const int mma = p.BN == 32 ? 44 : (p.BN == 64 ? 48 : (p.BN == 128 ? 64 : 128));
  const int g_max = min(min(512 / p.BN, 4), p.groups_total);
  // Sums on the tensor core drift by about 1.1e-9 of the result per term, so no accumulator takes more
  // bricks than it would in two waves of the widest CTAs (8 x 64^3 pixels, 32 -> 64 channels: error 2.9e-5
  // with one accumulator per CTA of one wave, 1.3e-5 so).  A CTA sums its bricks in parts: in as many
  // accumulators as TMEM holds, which costs nothing, in rounds where they do not suffice.
  const int widest = (p.groups_total + g_max - 1) / g_max * p.n_tiles;
  const int least = std::max(1, std::min((2 * sms + widest - 1) / widest, (p.bricks_total + 7) / 8));
  const int most = (p.bricks_total + least - 1) / least;
  double best = 0.0, ends = 0.0;
  for (int G = g_max; G >= 1; --G) {
    const int stage_bytes = G * 16384 + 64 * p.BN * 2;
    int stages = (232448 - 2048) / stage_bytes;
    if (stages > 4) stages = 4;
    if (stages < 1) continue;
    const int sets = (p.groups_total + G - 1) / G, base = sets * p.n_tiles;
    // Filters of one or a few taps load so little a brick (4 to 16 KB) that four stages do not cover the
    // copies' latency: two CTAs share an SM where both fit.  Forward and backward of 1 x 1 filters, bf16,
    // one CTA / two: 4 x 96^3, 32 -> 32 channels 560 / 483 us, 64 x 112^2, 16 -> 64 209 / 199.
    const int slices = min(G * p.spg, p.slices_total);
    const bool pair = 64 * 2 * (slices * p.Cb + p.BN) <= 16384 && 2 * (stages * stage_bytes + 3072) <= 232448;
    const int slots = pair ? 2 * sms : sms;
    int splits = base < slots ? slots / base : 1;
    if (splits > (p.bricks_total + 3) / 4) splits = (p.bricks_total + 3) / 4;   // amortise the pipeline fill
    const int per_cta = (p.bricks_total + splits - 1) / splits, parts = (per_cta + most - 1) / most;
    const int room = std::min(parts, std::max(1, (pair ? 256 : 512) / (G * p.BN)));
    const int rounds = (parts + room - 1) / room;
    const int waves = (base * splits + slots - 1) / slots;
    const double copy = max(stage_bytes / 58.0, 75.0 * (G * p.spg + p.BN / 64));
    const double brick = max(copy, 4.0 * G * mma) * (stages >= 3 ? 1.0 : (stages == 2 ? 1.25 : 2.0));
    // a further round adds its sums to the workspace at the L2: 21 B/clk an SM (8 x 16^3, 128 -> 256
    // channels in three rounds 67 us, in one 55; with a slot of its own for every round 74)
    const double store = (double)base * splits * (rounds - 1) * G * p.BN * 512 / (21.0 * sms);
    const double cost = waves * (per_cta * brick + 3000.0 * rounds) + store;
    if (best == 0.0 || cost < best) {
      best = cost;
      ends = wgrad_ends(stage_bytes, G, p.BN, (long long)base * splits, waves);
      p.G = G; p.group_sets = sets; p.splits = splits;
      p.parts = parts; p.room = room; p.stages = stages; p.stage_bytes = stage_bytes;
    }
  }
  if (best == 0.0) return false;
  p.a_bytes = p.G * 16384;
  wgrad_slab_plan(p, mma, (long long)most * p.rows_used, best + ends);
  const int cols = p.room * p.G * p.BN;
  p.tmem_cols = 32;
  while (p.tmem_cols < cols) p.tmem_cols *= 2;
  return true;
}

static long long wgrad_ws_floats(const WgradParams& p) {
  return (long long)p.group_sets * p.n_tiles * p.splits * p.G * p.BN * 128;
}

// The same, with this thread's last plan kept: a pass asks twice, for the workspace and for the launch, and the
// tilings that the slab kernel tries take 1 us each time (3x3, 64 -> 64 channels, 32 x 56^2: backward 2.5 us of host).
static bool wgrad_plan_twice(WgradParams& p) {
  struct Last {
    int sms = 0;
    bool covered = false;
    WgradParams p;
  };
  static thread_local Last last;
  const int sms = lbhost::sm_count();
  if (last.sms != sms || memcmp(&last.p.g, &p.g, sizeof(WgradGeom))) {
    last.covered = wgrad_plan(p);
    last.p = p;
    last.sms = sms;
  }
  p = last.p;
  return last.covered;
}

}  // namespace lb

extern "C" {

// fp32 words of workspace that lb_conv_wgrad_tc needs for these sizes; -1: not covered.
long long lb_conv_wgrad_ws(const int* geom) {
  lb::WgradParams p;
  memcpy(&p.g, geom, sizeof(lb::WgradGeom));
  return lb::wgrad_plan_twice(p) ? lb::wgrad_ws_floats(p) : -1;
}

// 1: these sizes take their taps from halo slabs, 0: a box for every tap, -1: not covered.
int lb_conv_wgrad_slab(const int* geom) {
  lb::WgradParams p;
  memcpy(&p.g, geom, sizeof(lb::WgradGeom));
  return lb::wgrad_plan(p) ? p.slab : -1;
}

// x:  [N][D][H][W][C] (strides xs, C contiguous), dy: [N][Do][Ho][Wo][Kout] (strides ys).
// dW: fp32, element (tap, k, c) at tap*s_tap + k*s_k + c*s_c; the kernel ADDS alpha * grad.
// geom as in lb_conv_fwd_tc; ws: lb_conv_wgrad_ws(geom) words, 16-byte aligned, whose contents
// do not matter.  Requires C % 8 == 0 and Kout % 8 == 0.
int lb_conv_wgrad_tc(const void* x, const void* dy, float* dW, float* ws, const int* geom,
                     const long long* xs, const long long* ys, long long s_tap, long long s_k,
                     long long s_c, int in_dtype, float alpha, void* stream_) {
  using namespace lb;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  WgradParams p;
  static_assert(sizeof(WgradGeom) == 21 * sizeof(int), "geom layout");
  memcpy(&p.g, geom, sizeof(WgradGeom));
  const WgradGeom& g = p.g;
  if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(dy) & 15)) return -1;
  for (int i = 0; i < 4; ++i)
    if (xs[i] % 8 || ys[i] % 8) return -1;
  if (!wgrad_plan_twice(p) || !ws || (reinterpret_cast<uintptr_t>(ws) & 15)) return -1;
  if (p.slab) wgrad_slab_offsets(p);
  p.in_dtype = in_dtype;
  p.alpha = alpha;
  p.dW = dW;
  p.ws = ws;
  p.s_tap = s_tap; p.s_k = s_k; p.s_c = s_c;

  const uint32_t bw = (p.TW - 1) * g.sw + (p.slab ? g.kw : 1), bh = (p.TH - 1) * g.sh + (p.slab ? g.kh : 1),
                 bd = (p.TD - 1) * g.sd + (p.slab ? g.kd : 1);
  if (bw > 256 || bh > 256 || bd > 256) return -1;
  CUtensorMap tmX, tmDy;
  {
    uint64_t dims[5] = {(uint64_t)g.C, (uint64_t)g.W, (uint64_t)g.H, (uint64_t)g.D, (uint64_t)g.N};
    uint64_t strides[4] = {(uint64_t)xs[3] * 2, (uint64_t)xs[2] * 2, (uint64_t)xs[1] * 2,
                           (uint64_t)xs[0] * 2};
    uint32_t box[5] = {(uint32_t)p.Cb, bw, bh, bd, (uint32_t)p.TN};
    uint32_t es[5] = {1, (uint32_t)g.sw, (uint32_t)g.sh, (uint32_t)g.sd, 1};
    if (p.slab) {                                   // planes lie inside lines
      std::swap(dims[2], dims[3]); std::swap(strides[1], strides[2]); std::swap(box[2], box[3]);
    }
    if (!lbhost::encode_tmap(&tmX, in_dtype, 5, x, dims, strides, box, es, p.Cb * 2)) return -1;
  }
  {
    uint64_t dims[5] = {(uint64_t)g.Kout, (uint64_t)g.Wo, (uint64_t)g.Ho, (uint64_t)g.Do,
                        (uint64_t)g.N};
    uint64_t strides[4] = {(uint64_t)ys[3] * 2, (uint64_t)ys[2] * 2, (uint64_t)ys[1] * 2,
                           (uint64_t)ys[0] * 2};
    const uint32_t inner = p.BN == 32 ? 32 : 64;
    uint32_t box[5] = {inner, (uint32_t)p.TW, (uint32_t)p.TH, (uint32_t)p.TD, (uint32_t)p.TN};
    if (!lbhost::encode_tmap(&tmDy, in_dtype, 5, dy, dims, strides, box, nullptr, inner * 2))
      return -1;
  }
  const int smem = p.stages * p.stage_bytes + 1024;
  static int configured_smem = 0;
  if (smem > configured_smem) {
    cudaFuncSetAttribute(conv_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaFuncSetAttribute(conv_wgrad_slab_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    configured_smem = smem;
  }
  const int grid = p.group_sets * p.n_tiles * p.splits;
  if (p.slab) conv_wgrad_slab_kernel<<<grid, 192, smem, stream>>>(tmX, tmDy, p, lbhost::status_word());
  else conv_wgrad_kernel<<<grid, 192, smem, stream>>>(tmX, tmDy, p, lbhost::status_word());
  const int rc = (int)cudaGetLastError();
  if (rc) return rc;
  // as many groups of splits as give every SM 1024 threads, at least four splits each
  const int taps = g.kd * g.kh * g.kw, kq = (g.Kout + 3) / 4;
  const long long sums = (long long)kq * g.C * taps, want = 1024ll * lbhost::sm_count();
  WgradReduce q;
  q.groups = 1;
  while (q.groups < 16 && q.groups * 8 <= p.splits && sums * q.groups < want) q.groups *= 2;
  q.NT = std::min(taps, kRedThreads / 8 / q.groups);
  q.log_ch = 3;
  while (q.log_ch < 5 && (1 << q.log_ch) < g.C && (2 << q.log_ch) * q.NT * q.groups <= kRedThreads) ++q.log_ch;
  q.items = q.NT << q.log_ch;
  q.log_cb = p.Cb == 64 ? 6 : (p.Cb == 32 ? 5 : 4);
  q.log_spg = 7 - q.log_cb;
  q.fd_items = FastDiv((uint32_t)q.items); q.fd_nt = FastDiv((uint32_t)q.NT);
  q.fd_kw = FastDiv((uint32_t)g.kw); q.fd_khkw = FastDiv((uint32_t)(g.kh * g.kw)); q.fd_G = FastDiv((uint32_t)p.G);
  const int CH = 1 << q.log_ch;
  wgrad_reduce_kernel<<<dim3(kq, (g.C + CH - 1) / CH, (taps + q.NT - 1) / q.NT), kRedThreads, 0, stream>>>(p, q);
  return (int)cudaGetLastError();
}

}  // extern "C"
