// Fused scaled-dot-product attention for head dimension 128 on tcgen05 / TMEM.
//
//   O = softmax(scale * Q K^T  [+ causal mask]) V        per (batch, head)
//
// The reference composes attention from eight layers (python/lbann/modules/transformer/
// attention.py:215-299: two batched MatMuls, a scale, a mask addition, ChannelwiseSoftmax,
// dropout and two permutes) and materialises the [heads, S, S] score tensor twice.  Here
// the scores never leave the SM: S = Q K^T is accumulated in TMEM, four warps turn it into
// probabilities (online softmax, fp32), write them as a 16-bit A operand into shared
// memory and the tensor core adds P V to the output accumulator, also in TMEM.
//
// Tensors are token-major: q, k, v, o are [B][S][H][128] views with arbitrary batch / token /
// head strides (so the three slices of a packed [B][S][3 H 128] projection are used in
// place, and the output needs no permute).  Sequence lengths are multiples of 128.
//
// Warp roles (320 threads): warp 4 loads (TMA), warp 5 allocates TMEM and issues the MMAs (one
// elected thread each), warps 0-3 and 6-9 own the accumulator rows.
//
// Backward is one launch of two kinds of CTA, both recomputing P from Q, K and the saved
// log-sum-exp: one per 128 keys (loop over queries: dV += P^T dO, dK += dS^T Q) and one per 128
// queries (loop over keys: dQ += dS K), with dS = P * (dP - rowsum(dO * O)) * scale.
//
// Every wait is bounded; a wait that runs out records a status code and all roles leave.
#include <type_traits>

#include <algorithm>

#include "common.cuh"

namespace lb {

constexpr int kAttD = 128;                 // head dimension
constexpr int kAttTile = 128 * kAttD * 2;  // one [128][128] 16-bit tile: 32 KiB
constexpr int kAttHalf = kAttTile / 2;     // its two [128][64] halves (128-byte swizzled rows)

struct AttnParams {
  int B, H, Sq, Sk;
  int causal;
  int in_dtype;
  float scale;           // multiplies Q K^T
  float scale_log2;      // scale * log2(e)
  // outputs / side inputs (element strides: batch, token, head; head dim contiguous)
  void* o; long long o_sb, o_ss, o_sh;
  float* lse;            // [B][H][Sq], log2 domain: max + log2(sum)
  const float* delta;    // [B][H][Sq] scale * rowsum(dO * O) (backward)
  void* dq; long long dq_sb, dq_ss, dq_sh;
  void* dk; long long dk_sb, dk_ss, dk_sh;
  void* dv; long long dv_sb, dv_ss, dv_sh;
};

constexpr int kFwdSlots = 3;               // ring of K and V tiles: K0 V0 K1 V1 ...
constexpr int kFwdSmem = (2 + 2 + kFwdSlots) * kAttTile + 1024;

struct AttnShared {
  uint64_t q_full;
  uint64_t kv_full[kFwdSlots], kv_empty[kFwdSlots];
  uint64_t s_full[2], s_empty[2];      // scores of a query tile: complete / read by its four warps
  uint64_t p_full[2], pv_done[2];      // probabilities written by four warps / their product retired
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
      "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
      "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem desc]: A has one row per lane, two 16-bit K elements per column.
__device__ __forceinline__ void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// acc (+)= A . B^T over K = 128 with both operands K-major tiles [2][128 rows][64 k].
__device__ __forceinline__ void att_mma_kk(uint32_t acc, uint32_t a, uint32_t b, uint32_t idesc,
                                           bool accumulate) {
  // the eight descriptors differ in the start-address field of the low word only
  const uint64_t d0 = make_smem_desc(0, 16, 1024, kLayoutSw128);
  const uint32_t hi = (uint32_t)(d0 >> 32);
  const uint32_t alo = (uint32_t)d0 + (a >> 4), blo = (uint32_t)d0 + (b >> 4);
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
    const uint32_t off = ((kk >> 2) * kAttHalf + (kk & 3) * 32) >> 4;
    umma_f16_lo(acc, alo + off, hi, blo + off, hi, idesc, (accumulate || kk) ? 1u : 0u);
  }
}
// acc (+)= A . B with A a K-major tile [2][128 rows][64 k] and B given as rows of K:
// [2 halves of N][128 k rows][64 n] ("MN-major"; the layout of a token-major tile as loaded).
__device__ __forceinline__ void att_mma_kn(uint32_t acc, uint32_t a, uint32_t b, uint32_t idesc,
                                           bool accumulate) {
  const uint64_t da = make_smem_desc(0, 16, 1024, kLayoutSw128);
  const uint64_t db = make_smem_desc(0, kAttHalf, 1024, kLayoutSw128);
  const uint32_t ahi = (uint32_t)(da >> 32), bhi = (uint32_t)(db >> 32);
  const uint32_t alo = (uint32_t)da + (a >> 4), blo = (uint32_t)db + (b >> 4);
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
    const uint32_t aoff = ((kk >> 2) * kAttHalf + (kk & 3) * 32) >> 4;
    umma_f16_lo(acc, alo + aoff, ahi, blo + ((kk * 2048) >> 4), bhi, idesc,
                (accumulate || kk) ? 1u : 0u);
  }
}

// Byte offset of element (row, col) in a K-major tile [2][128 rows][64 cols], 128-byte swizzle.
__device__ __forceinline__ uint32_t att_tile_off(int row, int col) {
  const int half = col >> 6, c = col & 63;
  return half * kAttHalf + row * 128 + (((c >> 3) ^ (row & 7)) << 4) + ((c & 7) << 1);
}

// Loads one [128 tokens][128] tile of head h: two boxes {64, 1, 128, 1}.
__device__ __forceinline__ void att_load_tile(uint32_t dst, const CUtensorMap* tm, uint32_t bar,
                                              int h, int s0, int b) {
  tma_load_4d(dst, tm, bar, 0, h, s0, b);
  tma_load_4d(dst + kAttHalf, tm, bar, 64, h, s0, b);
}

constexpr int kAttThreads = 320;

// Role of a warp among the 8 that work on accumulator rows: `group` 0 or 1 (four warps each),
// `quarter` the 32 TMEM lanes (= rows) that the warp may access (warp index modulo 4).
__device__ __forceinline__ bool att_row_role(int warp, int& group, int& quarter) {
  if (warp == 4 || warp == 5) return false;
  group = warp < 4 ? 0 : 1;
  quarter = warp & 3;
  return true;
}

// 64 accumulator columns of one row, scaled, -> 16-bit global row (16-byte stores).
__device__ __forceinline__ void att_store_out64(uint16_t* dst, const uint32_t (&a)[32], const uint32_t (&b)[32],
                                                float mul, int dtype) {
#pragma unroll
  for (int k = 0; k < 32; k += 8) {
    uint4 w;
    w.x = pack2(__uint_as_float(a[k]) * mul, __uint_as_float(a[k + 1]) * mul, dtype);
    w.y = pack2(__uint_as_float(a[k + 2]) * mul, __uint_as_float(a[k + 3]) * mul, dtype);
    w.z = pack2(__uint_as_float(a[k + 4]) * mul, __uint_as_float(a[k + 5]) * mul, dtype);
    w.w = pack2(__uint_as_float(a[k + 6]) * mul, __uint_as_float(a[k + 7]) * mul, dtype);
    *reinterpret_cast<uint4*>(dst + k) = w;
  }
#pragma unroll
  for (int k = 0; k < 32; k += 8) {
    uint4 w;
    w.x = pack2(__uint_as_float(b[k]) * mul, __uint_as_float(b[k + 1]) * mul, dtype);
    w.y = pack2(__uint_as_float(b[k + 2]) * mul, __uint_as_float(b[k + 3]) * mul, dtype);
    w.z = pack2(__uint_as_float(b[k + 4]) * mul, __uint_as_float(b[k + 5]) * mul, dtype);
    w.w = pack2(__uint_as_float(b[k + 6]) * mul, __uint_as_float(b[k + 7]) * mul, dtype);
    *reinterpret_cast<uint4*>(dst + 32 + k) = w;
  }
}

// ------------------------------------------------------------------------------------
// Forward.  A CTA holds two tiles of 128 queries (one, where that gives every SM a CTA) and walks
// the keys 128 at a time.  Each tile has four warps, one thread per query, and its own scores,
// probabilities and output accumulator; scores of the next keys are computed as soon as a
// tile's warps have read the present ones, so a tile's warps never wait for the tensor core and
// the tensor core works for one tile while the other's exponentials run.  (One tile per CTA
// with two threads per query left every latency of the chain exposed and cost 5700 cycles a
// block of 128 x 128, whose MMAs and exponentials take 1024 each.)  B = 2, H = 16, S = 2048,
// causal, bf16: 89 -> 50 us.
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kAttThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ AttnParams p, int tiles, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ AttnShared sh;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sQ = base, sP = base + 2 * kAttTile, sKV = base + 4 * kAttTile;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &sh.abort_flag;

  // the longest (late) query blocks first; tile t of this CTA is query block qb0 + t
  const int nqb = p.Sq / 128;
  const int h = blockIdx.x, b = blockIdx.y;
  const int qb0 = ((nqb + tiles - 1) / tiles - 1 - (int)blockIdx.z) * tiles;
  const int have = min(tiles, nqb - qb0);                // 1 or 2 tiles
  int n[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) n[t] = t < have ? (p.causal ? qb0 + t + 1 : p.Sk / 128) : 0;
  const int nmax = max(n[0], n[1]);

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&sh.q_full), 1);
    for (int s = 0; s < kFwdSlots; ++s) {
      mbar_init(smem_u32(&sh.kv_full[s]), 1);
      mbar_init(smem_u32(&sh.kv_empty[s]), 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(smem_u32(&sh.s_full[t]), 1);
      mbar_init(smem_u32(&sh.s_empty[t]), 4);
      mbar_init(smem_u32(&sh.p_full[t]), 4);
      mbar_init(smem_u32(&sh.pv_done[t]), 1);
    }
    sh.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 4 && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 5) {
    tmem_alloc(smem_u32(&sh.tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem_base;                    // scores of tile t at 128 t, outputs at 256 + 128 t

  if (warp == 4) {
    if (elect_one()) {
      mbar_expect_tx(smem_u32(&sh.q_full), (uint32_t)have * kAttTile);
      for (int t = 0; t < have; ++t)
        att_load_tile(sQ + t * kAttTile, &tmQ, smem_u32(&sh.q_full), h, (qb0 + t) * 128, b);
      RingPos rp;
      int seq = 0;
      bool ok = true;
      for (; seq < 2 * nmax; ++seq) {                    // K of block seq / 2, then its V
        if (!mbar_wait_bounded(smem_u32(&sh.kv_empty[rp.s]), rp.ph ^ 1, abort_flag)) {
          raise_status(status, abort_flag, kTimeoutStageEmpty);
          ok = false;
          break;
        }
        const uint32_t bar = smem_u32(&sh.kv_full[rp.s]);
        mbar_expect_tx(bar, kAttTile);
        att_load_tile(sKV + rp.s * kAttTile, (seq & 1) ? &tmV : &tmK, bar, h, (seq >> 1) * 128, b);
        rp.advance(kFwdSlots);
      }
      if (!ok || *abort_flag) {
        // let the copies in flight land before shared memory is released
        mbar_wait_budget_only(smem_u32(&sh.q_full), 0);
        for (int j = seq > kFwdSlots ? seq - kFwdSlots : 0; j < seq; ++j)
          mbar_wait_budget_only(smem_u32(&sh.kv_full[j % kFwdSlots]), (j / kFwdSlots) & 1);
      }
    }
  } else if (warp == 5) {
    if (elect_one()) {
      const uint32_t fmt = p.in_dtype == kBF16 ? 1u : 0u;
      const uint32_t idesc_qk = make_idesc_f16(fmt, 0, 0, 128, 128);
      const uint32_t idesc_pv = make_idesc_f16(fmt, 0, 1, 128, 128);
      bool ok = mbar_wait_bounded(smem_u32(&sh.q_full), 0, abort_flag);
      if (!ok) raise_status(status, abort_flag, kTimeoutTmaFull);
      RingPos kp, vp;                                    // slots of K(j) and V(j - 1): sequence 2 j and 2 j - 1
      vp.advance(kFwdSlots);
      for (int j = 0; j <= nmax && ok; ++j) {
        if (j < nmax) {
          if (!mbar_wait_bounded(smem_u32(&sh.kv_full[kp.s]), kp.ph, abort_flag)) {
            raise_status(status, abort_flag, kTimeoutTmaFull);
            ok = false;
            break;
          }
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (j >= n[t]) continue;
            if (j >= 1 && !mbar_wait_bounded(smem_u32(&sh.s_empty[t]), (j - 1) & 1, abort_flag)) {
              raise_status(status, abort_flag, kTimeoutTmemEmpty);
              ok = false;
              break;
            }
            tc_fence_after();
            att_mma_kk(tmem + t * 128, sQ + t * kAttTile, sKV + kp.s * kAttTile, idesc_qk, false);
            umma_commit(smem_u32(&sh.s_full[t]));
          }
          if (!ok) break;
          umma_commit(smem_u32(&sh.kv_empty[kp.s]));
          kp.advance(kFwdSlots);
          kp.advance(kFwdSlots);
        }
        if (j >= 1) {
          const int jj = j - 1;
          if (!mbar_wait_bounded(smem_u32(&sh.kv_full[vp.s]), vp.ph, abort_flag)) {
            raise_status(status, abort_flag, kTimeoutTmaFull);
            ok = false;
            break;
          }
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (jj >= n[t]) continue;
            if (!mbar_wait_bounded(smem_u32(&sh.p_full[t]), jj & 1, abort_flag)) {
              raise_status(status, abort_flag, kTimeoutTmemEmpty);
              ok = false;
              break;
            }
            tc_fence_after();
            att_mma_kn(tmem + 256 + t * 128, sP + t * kAttTile, sKV + vp.s * kAttTile, idesc_pv, jj > 0);
            umma_commit(smem_u32(&sh.pv_done[t]));
          }
          if (!ok) break;
          umma_commit(smem_u32(&sh.kv_empty[vp.s]));
          vp.advance(kFwdSlots);
          vp.advance(kFwdSlots);
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax / epilogue
    int t = 0, quarter = 0;
    att_row_role(warp, t, quarter);
    const int row = quarter * 32 + lane;                 // query row of this thread in tile t
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tS = tmem + t * 128 + lane_off, tO = tmem + 256 + t * 128 + lane_off;
    const uint32_t tile = sP + t * kAttTile;
    const int nt = t == 0 ? n[0] : n[1];
    float m = -1e30f, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nt && ok; ++j) {
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&sh.s_full[t]), j & 1, abort_flag));
      if (!ok) {
        if (lane == 0) raise_status(status, abort_flag, kTimeoutTmemFull);
        break;
      }
      tc_fence_after();
      uint32_t r[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(tS + 32 * c, r[c]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh.s_empty[t]));
      const bool diag = p.causal && j == nt - 1;         // columns up to `row` are visible
      auto row_max = [&](auto masked) {
        float mx[4] = {-1e30f, -1e30f, -1e30f, -1e30f};
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (!decltype(masked)::value || 32 * c + i <= row) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(r[c][i]));
        return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      };
      const float top = (diag ? row_max(std::true_type{}) : row_max(std::false_type{})) * p.scale_log2;
      // the running maximum is only moved when it would grow by more than 2^8: until then
      // the probabilities stay below 256 and O needs no rescaling
      float alpha = 1.f;
      if (top > m + 8.f) {
        alpha = fast_exp2(m - top);
        m = top;
      }
      l *= alpha;
      if (j >= 1) {
        // the previous P V has retired: the P buffer is free and O is consistent
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&sh.pv_done[t]), (j - 1) & 1, abort_flag));
        if (!ok) {
          if (lane == 0) raise_status(status, abort_flag, kTimeoutTmemFull);
          break;
        }
        if (__any_sync(0xffffffffu, alpha != 1.f)) {
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t o[32];
            tmem_ld_32x32(tO + 32 * c, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x32(tO + 32 * c, o);
          }
          tmem_st_wait();
        }
      }
      auto probabilities = [&](auto masked) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            float e[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              e[k] = fast_exp2(fmaf(__uint_as_float(r[c][i + k]), p.scale_log2, -m));
              if (decltype(masked)::value && 32 * c + i + k > row) e[k] = 0.f;
              sum[k & 3] += e[k];
            }
            sts128(tile + att_tile_off(row, 32 * c + i),
                   make_uint4(pack2(e[0], e[1], p.in_dtype), pack2(e[2], e[3], p.in_dtype),
                              pack2(e[4], e[5], p.in_dtype), pack2(e[6], e[7], p.in_dtype)));
          }
          l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        }
      };
      if (diag) probabilities(std::true_type{});
      else probabilities(std::false_type{});
      tc_fence_before();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh.p_full[t]));
    }
    if (ok && nt > 0) {
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&sh.pv_done[t]), (nt - 1) & 1, abort_flag));
      if (!ok && lane == 0) raise_status(status, abort_flag, kTimeoutTmemFull);
    }
    if (ok && nt > 0) {
      tc_fence_after();
      const float inv = 1.f / l;
      const long long q = (long long)(qb0 + t) * 128 + row;
      uint16_t* orow = reinterpret_cast<uint16_t*>(p.o) + b * p.o_sb + q * p.o_ss + h * p.o_sh;
#pragma unroll
      for (int c = 0; c < 128; c += 64) {
        uint32_t oa[32], ob[32];
        tmem_ld_32x32(tO + c, oa);
        tmem_ld_32x32(tO + c + 32, ob);
        tmem_ld_wait();
        att_store_out64(orow + c, oa, ob, inv, p.in_dtype);
      }
      if (p.lse) p.lse[((long long)b * p.H + h) * p.Sq + q] = m + log2f(l);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------
// delta[b][h][q] = scale * sum_d dO[b][q][h][d] * O[b][q][h][d]: 16 lanes of 16 bytes a row, two
// rows of a warp at a time, four rounds in flight
// ------------------------------------------------------------------------------------
// 64 rows of a batch entry a block.  B = 2, H = 16, S = 2048, bf16: 6.4 us for 67 MB.  (64-bit divisions by
// run-time values for every row, 11.5 us.)
template <typename T>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const T* __restrict__ o, const T* __restrict__ dout, float* __restrict__ delta, FastDiv heads, int exact,
                  int H, int S, float scale, long long o_sb, long long o_ss, long long o_sh, long long d_sb, long long d_ss,
                  long long d_sh) {
  const uint32_t rows = (uint32_t)H * (uint32_t)S;
  const int half = (threadIdx.x >> 4) & 1, lane = threadIdx.x & 15, b = blockIdx.y;
  const uint32_t row0 = (blockIdx.x * 256 + threadIdx.x) / 32 * 8 + half;
  o += b * o_sb + lane * 8;
  dout += b * d_sb + lane * 8;
  delta += (long long)b * rows;
  uint4 a[4], g[4];
  uint32_t at[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const uint32_t r = min(row0 + 2 * u, rows - 1);
    // consecutive rows are the heads of a token: they are adjacent in memory
    const uint32_t q = exact ? heads.div(r) : r / (uint32_t)H, h = r - q * (uint32_t)H;
    at[u] = h * (uint32_t)S + q;
    a[u] = *reinterpret_cast<const uint4*>(o + q * o_ss + h * o_sh);
    g[u] = *reinterpret_cast<const uint4*>(dout + q * d_ss + h * d_sh);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const T* ea = reinterpret_cast<const T*>(&a[u]);
    const T* eg = reinterpret_cast<const T*>(&g[u]);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += to_f32<T>(ea[i]) * to_f32<T>(eg[i]);
#pragma unroll
    for (int m = 8; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    if (lane == 0 && row0 + 2 * u < rows) delta[at[u]] = s * scale;
  }
}

// ------------------------------------------------------------------------------------
// Backward.  One launch holds two kinds of CTA:
//   keys    (KV): 128 keys stay, the loop runs over 64 queries at a time; rows = keys
//       S^T = K Q_i^T, dP^T = V dO_i^T;  dV += P^T dO_i,  dK += dS^T Q_i
//   queries (Q):  128 queries stay, the loop runs over 64 keys at a time; rows = queries
//       S = Q K_n^T, dP = dO V_n^T;      dQ += dS K_n
// with P = exp2(S c - lse) and dS = P * (dP - delta) * scale.  In both, with R0, R1 the operands
// that stay and T0, T1 the streamed ones: S = R0 T0^T, dP = R1 T1^T, acc1 += dS T0 and for keys
// acc0 += P T1.
//
// The chain S -> exp -> P, dS -> accumulate is 2-3 thousand cycles long and the MMAs of a step 1.0
// to 1.3 thousand, so steps overlap: 64 columns a step leave room in TMEM for two S / dP pairs
// beside the accumulators.  P and dS overwrite the scores they came from, as 16-bit operands in
// TMEM: through shared memory they cost as much of its bandwidth as half the MMAs.  The issuer
// starts step i + 1's scores before it waits for step i's probabilities.  One arrival per warp (256
// single arrivals on a barrier took longer than the exponentials).
// The CTAs stay and take items in turn: the next item's operands arrive and its first scores run while
// the rows of the last one are written.
// B = 2, H = 16, S = 2048, bf16: causal 308 us as two kernels with one step in flight -> 161 with P and dS in
// shared memory -> 153 with a CTA an item -> 142; not causal 242 -> 226.  What is left is a step's 16 MMAs of
// N = 64, which read 128 rows of A for half the arithmetic (48 cycles where 32 would do), and the wait from the
// end of an accumulation to the scores that overwrite its operands: rows that do nothing leave 124 us.  The tensor
// pipe is active for 47 % of the cycles.
// (Waiting for P and dS separately: 143; scores read into registers first, P and dS elsewhere: 157; 16 row
// warps: no change.)
// ------------------------------------------------------------------------------------
constexpr int kBwdCols = 64;                          // streamed rows (= score columns) per step
constexpr int kBwdTile = kBwdCols * kAttD * 2;        // 16 KB: one streamed operand
constexpr int kBwdHalf = kBwdTile / 2;                // its two [64 rows][64] halves
constexpr int kBwdStages = 4;
constexpr int kBwdSmem = 2 * kAttTile + kBwdStages * 2 * kBwdTile + 1024;

struct __align__(128) AttnBwdShared {
  float lse[kBwdStages][kBwdCols];     // keys: of the streamed queries
  float delta[kBwdStages][kBwdCols];
  uint64_t resident;                   // the operands that stay have landed
  uint64_t res_empty;                  // their last scores have retired
  uint64_t acc_empty;                  // the accumulators have been read (8 warps)
  uint64_t st_full[kBwdStages];        // a stage has landed
  uint64_t st_empty[kBwdStages];       // the MMAs of a step have retired: stage, P and dS are free
  uint64_t s_full[2];                  // scores and dP of a step are complete
  uint64_t p_full[2];                  // P and dS of a step are in TMEM (8 warps)
  uint32_t tmem_base;
  int abort_flag;
};

// acc = A . B^T over K = 128: A a K-major tile [2][128 rows][64], B [2][64 rows][64]
__device__ __forceinline__ void bwd_mma_scores(uint32_t acc, uint32_t a, uint32_t b, uint32_t idesc) {
  const uint64_t d0 = make_smem_desc(0, 16, 1024, kLayoutSw128);
  const uint32_t hi = (uint32_t)(d0 >> 32);
  const uint32_t alo = (uint32_t)d0 + (a >> 4), blo = (uint32_t)d0 + (b >> 4);
#pragma unroll
  for (int kk = 0; kk < 8; ++kk)
    umma_f16_lo(acc, alo + (((kk >> 2) * kAttHalf + (kk & 3) * 32) >> 4), hi,
                blo + (((kk >> 2) * kBwdHalf + (kk & 3) * 32) >> 4), hi, idesc, kk ? 1u : 0u);
}
// acc (+)= A . B over K = 64: A in TMEM (two pieces of 16 columns, 32 apart: each group of row
// warps packs into its own half), B rows of K ([2 halves of N][64][64])
__device__ __forceinline__ void bwd_mma_accumulate(uint32_t acc, uint32_t a, uint32_t b, uint32_t idesc, bool accumulate) {
  const uint64_t db = make_smem_desc(0, kBwdHalf, 1024, kLayoutSw128);
  const uint32_t bhi = (uint32_t)(db >> 32), blo = (uint32_t)db + (b >> 4);
#pragma unroll
  for (int kk = 0; kk < 4; ++kk)
    umma_f16_ta(acc, a + (kk >> 1) * 32 + (kk & 1) * 8, blo + ((kk * 2048) >> 4), bhi, idesc, (accumulate || kk) ? 1u : 0u);
}

// 32 columns of P and dS of one row, packed: cols[k] of this thread's columns are visible from
// `first` on (keys) or up to `last` (queries).
template <bool KV>
__device__ __forceinline__ void bwd_probabilities(const uint32_t (&rs)[32], const uint32_t (&rd)[32], const float* lse,
                                                  const float* delta, float my_lse, float my_delta, int first, int last,
                                                  const AttnParams& p, uint32_t (&pk)[16], uint32_t (&dk)[16]) {
  const bool masked = first > 0 || last < 31;
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    float4 l4, d4;
    if (KV) {
      l4 = *reinterpret_cast<const float4*>(lse + k);
      d4 = *reinterpret_cast<const float4*>(delta + k);
    } else {
      l4 = make_float4(my_lse, my_lse, my_lse, my_lse);
      d4 = make_float4(my_delta, my_delta, my_delta, my_delta);
    }
    const float l[4] = {l4.x, l4.y, l4.z, l4.w}, dl[4] = {d4.x, d4.y, d4.z, d4.w};
    float e[4], d[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      e[j] = fast_exp2(fmaf(__uint_as_float(rs[k + j]), p.scale_log2, -l[j]));
      if (masked) e[j] = (k + j >= first && k + j <= last) ? e[j] : 0.f;
      d[j] = e[j] * fmaf(__uint_as_float(rd[k + j]), p.scale, -dl[j]);
    }
    if (KV) {
      pk[k / 2] = pack2(e[0], e[1], p.in_dtype);
      pk[k / 2 + 1] = pack2(e[2], e[3], p.in_dtype);
    }
    dk[k / 2] = pack2(d[0], d[1], p.in_dtype);
    dk[k / 2 + 1] = pack2(d[2], d[3], p.in_dtype);
  }
}

// One work item: 128 keys (KV) or queries of a head.
struct BwdItem {
  bool kv;
  int blk, h, b, i0, iters;            // first step that sees these rows, steps
};
// Items in the order of their lengths, the longest first, and dealt to the CTAs forwards and backwards in turn, so
// that the sums of the lengths are nearly the same.  False: this CTA's rounds are over.
__device__ __forceinline__ bool bwd_item(const AttnParams& p, int round, BwdItem& w) {
  const int nkb = p.Sk / 128, nqb = p.Sq / 128, heads = p.H * p.B, total = (nkb + nqb) * heads;
  const int base = round * (int)gridDim.x;
  const int idx = base + ((round & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
  if (base >= total) return false;
  w.iters = 0;
  if (idx >= total) return true;       // an incomplete last round
  const int z = idx / heads, hb = idx - z * heads;
  w.b = hb / p.H;
  w.h = hb - w.b * p.H;
  if (p.causal) {                      // keys see the queries behind them, queries the keys before them
    w.kv = (z & 1) == 0;
    w.blk = w.kv ? z >> 1 : nqb - 1 - (z >> 1);
  } else if (p.Sq >= p.Sk) {           // keys walk the queries
    w.kv = z < nkb;
    w.blk = w.kv ? z : z - nkb;
  } else {
    w.kv = z >= nqb;
    w.blk = w.kv ? z - nqb : z;
  }
  const int all = (w.kv ? p.Sq : p.Sk) / kBwdCols;
  w.i0 = w.kv && p.causal ? 2 * w.blk : 0;
  w.iters = w.kv ? all - w.i0 : (p.causal ? 2 * w.blk + 2 : all);
  return true;
}

struct BwdMaps {
  const CUtensorMap *r0, *r1, *t0, *t1;
};

// The producer's part of an item; `step` counts the CTA's steps, `item` its items.
template <bool KV>
__device__ __forceinline__ bool bwd_produce(const BwdMaps& m, const AttnParams& p, const BwdItem& w, int item, uint32_t base,
                                            AttnBwdShared& sh, RingPos& rp, int& step, volatile int* abort_flag, int* status) {
  const uint32_t sT = base + 2 * kAttTile;
  const long long stat0 = ((long long)w.b * p.H + w.h) * p.Sq;     // this head's lse / delta
  if (!mbar_wait_bounded(smem_u32(&sh.res_empty), (item & 1) ^ 1, abort_flag)) {
    raise_status(status, abort_flag, kTimeoutStageEmpty);
    return false;
  }
  mbar_expect_tx(smem_u32(&sh.resident), 2 * kAttTile);
  att_load_tile(base, m.r0, smem_u32(&sh.resident), w.h, w.blk * 128, w.b);
  att_load_tile(base + kAttTile, m.r1, smem_u32(&sh.resident), w.h, w.blk * 128, w.b);
  for (int it = 0; it < w.iters; ++it, ++step) {
    if (!mbar_wait_bounded(smem_u32(&sh.st_empty[rp.s]), rp.ph ^ 1, abort_flag)) {
      raise_status(status, abort_flag, kTimeoutStageEmpty);
      return false;
    }
    const uint32_t bar = smem_u32(&sh.st_full[rp.s]), dst = sT + rp.s * 2 * kBwdTile;
    const int r0 = (w.i0 + it) * kBwdCols;
    mbar_expect_tx(bar, 2 * kBwdTile + (KV ? 2 * kBwdCols * 4 : 0));
    tma_load_4d(dst, m.t0, bar, 0, w.h, r0, w.b);
    tma_load_4d(dst + kBwdHalf, m.t0, bar, 64, w.h, r0, w.b);
    tma_load_4d(dst + kBwdTile, m.t1, bar, 0, w.h, r0, w.b);
    tma_load_4d(dst + kBwdTile + kBwdHalf, m.t1, bar, 64, w.h, r0, w.b);
    if (KV) {
      bulk_load_1d(smem_u32(sh.lse[rp.s]), p.lse + stat0 + r0, kBwdCols * 4, bar);
      bulk_load_1d(smem_u32(sh.delta[rp.s]), p.delta + stat0 + r0, kBwdCols * 4, bar);
    }
    rp.advance(kBwdStages);
  }
  return true;
}

// The issuer's part: scores of step it + 1 before the accumulation of step it.
template <bool KV>
__device__ __forceinline__ bool bwd_issue(const AttnParams& p, const BwdItem& w, int item, uint32_t base, uint32_t tmem,
                                          AttnBwdShared& sh, RingPos& next, RingPos& cur, int& step,
                                          volatile int* abort_flag, int* status) {
  const uint32_t sR0 = base, sR1 = base + kAttTile, sT = base + 2 * kAttTile, tAcc0 = tmem + 256, tAcc1 = tmem + 384;
  const uint32_t fmt = p.in_dtype == kBF16 ? 1u : 0u;
  const uint32_t idesc_s = make_idesc_f16(fmt, 0, 0, 128, kBwdCols);
  const uint32_t idesc_a = make_idesc_f16(fmt, 0, 1, 128, 128);
  if (!mbar_wait_bounded(smem_u32(&sh.resident), item & 1, abort_flag)) {
    raise_status(status, abort_flag, kTimeoutTmaFull);
    return false;
  }
  for (int it = -1; it < w.iters; ++it) {
    if (it + 1 < w.iters) {          // over the P and dS of two steps before
      const int n = step + it + 1, j = n - 2;
      if (!mbar_wait_bounded(smem_u32(&sh.st_full[next.s]), next.ph, abort_flag) ||
          (j >= 0 && !mbar_wait_bounded(smem_u32(&sh.st_empty[j % kBwdStages]), (j / kBwdStages) & 1, abort_flag))) {
        raise_status(status, abort_flag, kTimeoutTmaFull);
        return false;
      }
      tc_fence_after();
      const uint32_t t = sT + next.s * 2 * kBwdTile, d = tmem + (n & 1) * 128;
      bwd_mma_scores(d, sR0, t, idesc_s);
      bwd_mma_scores(d + kBwdCols, sR1, t + kBwdTile, idesc_s);
      umma_commit(smem_u32(&sh.s_full[n & 1]));
      if (it + 2 == w.iters) umma_commit(smem_u32(&sh.res_empty));
      next.advance(kBwdStages);
    }
    if (it >= 0) {
      const int n = step + it;
      if ((it == 0 && !mbar_wait_bounded(smem_u32(&sh.acc_empty), (item & 1) ^ 1, abort_flag)) ||
          !mbar_wait_bounded(smem_u32(&sh.p_full[n & 1]), (n >> 1) & 1, abort_flag)) {
        raise_status(status, abort_flag, kTimeoutTmemEmpty);
        return false;
      }
      tc_fence_after();
      const uint32_t t = sT + cur.s * 2 * kBwdTile;
      const uint32_t tP = tmem + (n & 1) * 128;
      if (KV) bwd_mma_accumulate(tAcc0, tP, t + kBwdTile, idesc_a, it > 0);
      bwd_mma_accumulate(tAcc1, tP + kBwdCols, t, idesc_a, it > 0);
      umma_commit(smem_u32(&sh.st_empty[cur.s]));
      cur.advance(kBwdStages);
    }
  }
  step += w.iters;
  return true;
}

// A row warp's part: probabilities and dS of every step, then the accumulators' rows.
template <bool KV>
__device__ __forceinline__ bool bwd_rows(const AttnParams& p, const BwdItem& w, int group, int quarter, uint32_t tmem,
                                         AttnBwdShared& sh, RingPos& rp, int& step, float my_lse, float my_delta,
                                         volatile int* abort_flag, int* status) {
  const int lane = threadIdx.x & 31;
  const int row = quarter * 32 + lane;               // this thread's key / query; its half of the columns
  const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
  for (int it = 0; it < w.iters; ++it, ++step) {
    bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&sh.s_full[step & 1]), (step >> 1) & 1, abort_flag));
    // lse and delta of a step came with its stage
    if (ok && KV) ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&sh.st_full[rp.s]), rp.ph, abort_flag));
    if (!ok) {
      if (lane == 0) raise_status(status, abort_flag, kTimeoutTmemFull);
      return false;
    }
    tc_fence_after();
    const uint32_t tS = tmem + (step & 1) * 128 + lane_off;
    const int c = group * 32;
    uint32_t rs[32], rd[32], pk[16], dk[16];
    tmem_ld_32x32(tS + c, rs);
    tmem_ld_32x32(tS + kBwdCols + c, rd);
    tmem_ld_wait();
    // causal: query >= key; distance of these columns from this item's first row
    const int off = p.causal ? (w.i0 + it) * kBwdCols + c - w.blk * 128 : 0;
    const int first = KV && p.causal ? row - off : 0;
    const int last = !KV && p.causal ? row - off : 31;
    bwd_probabilities<KV>(rs, rd, sh.lse[rp.s] + c, sh.delta[rp.s] + c, my_lse, my_delta, first, last, p, pk, dk);
    // two to a column, over scores that this thread has read
    if (KV) tmem_st_32x16(tS + c, pk);
    tmem_st_32x16(tS + kBwdCols + c, dk);
    tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&sh.p_full[step & 1]));
    rp.advance(kBwdStages);
  }
  const int j = step - 1;
  if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&sh.st_empty[j % kBwdStages]), (j / kBwdStages) & 1, abort_flag))) {
    if (lane == 0) raise_status(status, abort_flag, kTimeoutTmemFull);
    return false;
  }
  tc_fence_after();
  const long long r = (long long)w.blk * 128 + row;
  const int d0 = group * 64;                         // this thread's half of the head dimension
  const uint32_t tAcc = tmem + 256 + lane_off + d0;
  uint16_t* out = KV ? reinterpret_cast<uint16_t*>(p.dk) + w.b * p.dk_sb + r * p.dk_ss + w.h * p.dk_sh + d0
                     : reinterpret_cast<uint16_t*>(p.dq) + w.b * p.dq_sb + r * p.dq_ss + w.h * p.dq_sh + d0;
  uint32_t ra[32], rb[32];
  if (KV) {
    uint16_t* dv = reinterpret_cast<uint16_t*>(p.dv) + w.b * p.dv_sb + r * p.dv_ss + w.h * p.dv_sh + d0;
    tmem_ld_32x32(tAcc, ra);
    tmem_ld_32x32(tAcc + 32, rb);
    tmem_ld_wait();
    att_store_out64(dv, ra, rb, 1.f, p.in_dtype);
  }
  tmem_ld_32x32(tAcc + 128, ra);
  tmem_ld_32x32(tAcc + 160, rb);
  tmem_ld_wait();
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(&sh.acc_empty));
  att_store_out64(out, ra, rb, 1.f, p.in_dtype);
  return true;
}

__global__ void __launch_bounds__(kAttThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                const __grid_constant__ CUtensorMap tmQ64, const __grid_constant__ CUtensorMap tmK64,
                const __grid_constant__ CUtensorMap tmV64, const __grid_constant__ CUtensorMap tmDO64,
                const __grid_constant__ AttnParams p, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ AttnBwdShared sh;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5;
  volatile int* abort_flag = &sh.abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&sh.resident), 1);
    mbar_init(smem_u32(&sh.res_empty), 1);
    mbar_init(smem_u32(&sh.acc_empty), 8);
    for (int s = 0; s < kBwdStages; ++s) {
      mbar_init(smem_u32(&sh.st_full[s]), 1);
      mbar_init(smem_u32(&sh.st_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&sh.s_full[s]), 1);
      mbar_init(smem_u32(&sh.p_full[s]), 8);
    }
    sh.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 5) {
    tmem_alloc(smem_u32(&sh.tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem_base;

  BwdItem w;
  int step = 0, item = 0;
  bool ok = true;
  if (warp == 4) {
    if (elect_one()) {
      const BwdMaps keys = {&tmK, &tmV, &tmQ64, &tmDO64}, queries = {&tmQ, &tmDO, &tmK64, &tmV64};
      RingPos rp;
      for (int r = 0; ok && bwd_item(p, r, w); ++r) {
        if (w.iters == 0) continue;
        ok = w.kv ? bwd_produce<true>(keys, p, w, item, base, sh, rp, step, abort_flag, status)
                  : bwd_produce<false>(queries, p, w, item, base, sh, rp, step, abort_flag, status);
        ++item;
      }
      if (!ok || *abort_flag) {        // the copies in flight land before shared memory is released
        for (int k = max(0, item - 2); k < item; ++k) mbar_wait_budget_only(smem_u32(&sh.resident), k & 1);
        for (int j = max(0, step - kBwdStages); j < step; ++j)
          mbar_wait_budget_only(smem_u32(&sh.st_full[j % kBwdStages]), (j / kBwdStages) & 1);
      }
    }
  } else if (warp == 5) {
    if (elect_one()) {
      RingPos next, cur;               // stages of the scores' step and of the accumulating step
      for (int r = 0; ok && bwd_item(p, r, w); ++r) {
        if (w.iters == 0) continue;
        ok = w.kv ? bwd_issue<true>(p, w, item, base, tmem, sh, next, cur, step, abort_flag, status)
                  : bwd_issue<false>(p, w, item, base, tmem, sh, next, cur, step, abort_flag, status);
        ++item;
      }
    }
  } else {
    int group = 0, quarter = 0;
    att_row_role(warp, group, quarter);
    const int row = quarter * 32 + (threadIdx.x & 31);
    RingPos rp;
    for (int r = 0; ok && bwd_item(p, r, w); ++r) {
      if (w.iters == 0) continue;
      if (w.kv) {
        ok = bwd_rows<true>(p, w, group, quarter, tmem, sh, rp, step, 0.f, 0.f, abort_flag, status);
      } else {
        const long long at = ((long long)w.b * p.H + w.h) * p.Sq + w.blk * 128 + row;
        ok = bwd_rows<false>(p, w, group, quarter, tmem, sh, rp, step, p.lse[at], p.delta[at], abort_flag, status);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// Tensor map of a token-major tensor [B][S][H][128] with element strides (sb, ss, sh).
static bool att_tmap(CUtensorMap* tm, const void* ptr, int dtype, int B, int S, int H, long long sb,
                     long long ss, long long sh, uint32_t rows = 128) {
  uint64_t dims[4] = {(uint64_t)kAttD, (uint64_t)H, (uint64_t)S, (uint64_t)B};
  uint64_t strides[3] = {(uint64_t)sh * 2, (uint64_t)ss * 2, (uint64_t)sb * 2};
  uint32_t box[4] = {64, 1, rows, 1};
  return lbhost::encode_tmap(tm, dtype, 4, ptr, dims, strides, box, nullptr, 128);
}

static bool att_layout_ok(const void* ptr, long long sb, long long ss, long long sh) {
  return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && sb % 8 == 0 && ss % 8 == 0 && sh % 8 == 0;
}

}  // namespace lb

extern "C" {

// q, k, v, o: [B][S][H][128] views, strides in elements (batch, token, head); head dim dense.
// lse: fp32 [B][H][Sq] (log2 domain), written when not null.  dtype: 0 fp16, 1 bf16.
// Returns -2 when the shape is not covered (head dim != 128 is the caller's check; sequence
// lengths must be multiples of 128, causal needs Sq == Sk).
int lb_attention_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int H,
                     int Sq, int Sk, const long long* qs, const long long* ks, const long long* vs,
                     const long long* os, float scale, int causal, int dtype, void* stream_) {
  using namespace lb;
  if (B < 1 || H < 1 || Sq < 128 || Sk < 128 || Sq % 128 || Sk % 128) return -2;
  if (causal && Sq != Sk) return -2;
  if (dtype != kF16 && dtype != kBF16) return -2;
  if (!att_layout_ok(q, qs[0], qs[1], qs[2]) || !att_layout_ok(k, ks[0], ks[1], ks[2]) ||
      !att_layout_ok(v, vs[0], vs[1], vs[2]) || !att_layout_ok(o, os[0], os[1], os[2])) return -1;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  CUtensorMap tq, tk, tv;
  if (!att_tmap(&tq, q, dtype, B, Sq, H, qs[0], qs[1], qs[2]) ||
      !att_tmap(&tk, k, dtype, B, Sk, H, ks[0], ks[1], ks[2]) ||
      !att_tmap(&tv, v, dtype, B, Sk, H, vs[0], vs[1], vs[2])) return -1;
  AttnParams p;
  memset(&p, 0, sizeof(p));
  p.B = B; p.H = H; p.Sq = Sq; p.Sk = Sk; p.causal = causal; p.in_dtype = dtype;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.o = o; p.o_sb = os[0]; p.o_ss = os[1]; p.o_sh = os[2]; p.lse = lse;
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
    configured = true;
  }
  // one query tile per CTA where all of them fit on the device at once, else two
  const int nqb = Sq / 128, tiles = (long long)nqb * H * B <= lbhost::sm_count() ? 1 : 2;
  attn_fwd_kernel<<<dim3(H, B, (nqb + tiles - 1) / tiles), kAttThreads, kFwdSmem, stream>>>(tq, tk, tv, p, tiles,
                                                                                       lbhost::status_word());
  return (int)cudaGetLastError();
}

// Gradients of lb_attention_fwd.  o, dout: [B][Sq][H][128]; lse from the forward call; delta:
// fp32 workspace [B][H][Sq], overwritten.  dq, dk, dv are written (not accumulated).
int lb_attention_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout,
                     const float* lse, float* delta, void* dq, void* dk, void* dv, int B, int H, int Sq,
                     int Sk, const long long* qs, const long long* ks, const long long* vs,
                     const long long* os, const long long* dos, const long long* dqs,
                     const long long* dks, const long long* dvs, float scale, int causal, int dtype,
                     void* stream_) {
  using namespace lb;
  if (B < 1 || H < 1 || Sq < 128 || Sk < 128 || Sq % 128 || Sk % 128) return -2;
  if (causal && Sq != Sk) return -2;
  if (dtype != kF16 && dtype != kBF16) return -2;
  if (!att_layout_ok(q, qs[0], qs[1], qs[2]) || !att_layout_ok(k, ks[0], ks[1], ks[2]) ||
      !att_layout_ok(v, vs[0], vs[1], vs[2]) || !att_layout_ok(o, os[0], os[1], os[2]) ||
      !att_layout_ok(dout, dos[0], dos[1], dos[2]) || !att_layout_ok(dq, dqs[0], dqs[1], dqs[2]) ||
      !att_layout_ok(dk, dks[0], dks[1], dks[2]) || !att_layout_ok(dv, dvs[0], dvs[1], dvs[2]))
    return -1;
  if ((reinterpret_cast<uintptr_t>(lse) & 15) || (reinterpret_cast<uintptr_t>(delta) & 15)) return -1;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  CUtensorMap tq, tk, tv, tdo, tq64, tk64, tv64, tdo64;
  if (!att_tmap(&tq, q, dtype, B, Sq, H, qs[0], qs[1], qs[2]) ||
      !att_tmap(&tk, k, dtype, B, Sk, H, ks[0], ks[1], ks[2]) ||
      !att_tmap(&tv, v, dtype, B, Sk, H, vs[0], vs[1], vs[2]) ||
      !att_tmap(&tdo, dout, dtype, B, Sq, H, dos[0], dos[1], dos[2]) ||
      !att_tmap(&tq64, q, dtype, B, Sq, H, qs[0], qs[1], qs[2], kBwdCols) ||
      !att_tmap(&tk64, k, dtype, B, Sk, H, ks[0], ks[1], ks[2], kBwdCols) ||
      !att_tmap(&tv64, v, dtype, B, Sk, H, vs[0], vs[1], vs[2], kBwdCols) ||
      !att_tmap(&tdo64, dout, dtype, B, Sq, H, dos[0], dos[1], dos[2], kBwdCols)) return -1;
  {
    const long long rows = (long long)H * Sq;          // of a batch entry
    const int exact = rows * H < (1ll << 32);          // range of the fast division
    const dim3 blocks((unsigned)((rows + 63) / 64), (unsigned)B);
    const FastDiv heads((uint32_t)H);
    if (dtype == kBF16)
      attn_delta_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(
          (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta, heads, exact, H, Sq, scale, os[0], os[1], os[2],
          dos[0], dos[1], dos[2]);
    else
      attn_delta_kernel<__half><<<blocks, 256, 0, stream>>>((const __half*)o, (const __half*)dout, delta, heads, exact, H, Sq,
                                                            scale, os[0], os[1], os[2], dos[0], dos[1], dos[2]);
  }
  AttnParams p;
  memset(&p, 0, sizeof(p));
  p.B = B; p.H = H; p.Sq = Sq; p.Sk = Sk; p.causal = causal; p.in_dtype = dtype;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.lse = const_cast<float*>(lse); p.delta = delta;
  p.dq = dq; p.dq_sb = dqs[0]; p.dq_ss = dqs[1]; p.dq_sh = dqs[2];
  p.dk = dk; p.dk_sb = dks[0]; p.dk_ss = dks[1]; p.dk_sh = dks[2];
  p.dv = dv; p.dv_sb = dvs[0]; p.dv_ss = dvs[1]; p.dv_sh = dvs[2];
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(attn_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdSmem);
    configured = true;
  }
  const long long items = (long long)H * B * (Sk / 128 + Sq / 128);
  if (items > (1ll << 30)) return -2;
  const int grid = (int)std::min<long long>(items, lbhost::sm_count());
  attn_bwd_kernel<<<grid, kAttThreads, kBwdSmem, stream>>>(
      tq, tk, tv, tdo, tq64, tk64, tv64, tdo64, p, lbhost::status_word());
  return (int)cudaGetLastError();
}

}  // extern "C"
