// Chunked causal prefill attention over the paged pool, two query heads of a key head per CTA (tcgen05 + TMEM + TMA).
//
// What bounds it: per 128 queries x 128 keys the exponentials take 1024 cycles of an SM (16 a cycle) and the two products of a
// 128-wide head 768 (their operands pass shared memory at 128 bytes a cycle). With one tile per CTA and one softmax thread per row
// these follow one another, with a single warp per scheduler to hide every latency: 4600 cycles. Here a CTA has the tiles of two
// query heads that share a key head, so keys and values are brought once for both, and the products of one head run under the
// softmax of the other:
//
//   warp 0     TMA producer: both Q tiles once, then K and V tiles of 128 keys (8 pool blocks of 16) into rings of two
//   warp 1     MMA issuer, per key tile and head t: O_t += P_t V (P_t from TMEM), then S_t = Q_t K^T of the next key tile
//   warps 2-5  softmax of head 0, one thread per query row; warps 6-9 of head 1. The row is taken from TMEM, and the weights go
//              back there as bf16 pairs over the first half of its scores: no pass through shared memory, whose room the second Q
//              tile needs. Running maximum with lazy rescaling as in attention_tc.cu.
//
// TMEM: S_0 | S_1 | O_0 | O_1, 128 + 128 + D + D columns. A commit behind S_t of key tile j + 1 also covers O_t of key tile j, so one
// barrier per head and direction is all that the two sides exchange. Every wait is bounded and reports through the status word.
// Measured on B200, one head per CTA before (us a layer, 32 query and 8 key heads of 128): 8 prompts of 1024 tokens 158 (265),
// portions of 2048 tokens over contexts to 12000 on average 240 (384), 820 TFLOP/s of causal products; 64 heads of 64, 4 x 2048
// tokens with windows of 128 in every other layer 227 (383). Against 64 bits both are off by the same 2.34e-3 (4000 keys).
#include "api.h"
#include "attention_tc2.cuh"
#include "common.cuh"

namespace mx {

constexpr int kT2Rows = 128, kT2Keys = 128, kT2Block = 16, kT2Threads = 320;
constexpr float kT2Rescale = 8.0f;                    // log2 units
enum : int { kErrT2Producer = 411, kErrT2Mma = 412, kErrT2Softmax = 413 };

__device__ __forceinline__ void t2_mma_tmem_a(uint32_t d, uint32_t a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred P;\n\tsetp.ne.b32 P, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, P;\n\t}" ::"r"(d), "r"(a), "l"(desc_b), "r"(idesc), "r"(accumulate)
               : "memory");
}
__device__ __forceinline__ float t2_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int D>
__global__ void __launch_bounds__(kT2Threads, 1)
paged_prefill_tc2_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const PrefillTc2Params p) {
  constexpr int DC = D / 64;                          // 64-column (128-byte) sub-tiles per row
  constexpr int SUB = 128 * 128;                      // bytes of one [128 rows][64 cols] sub-tile
  constexpr int TILE = DC * SUB;
  constexpr int O_COL = 2 * kT2Keys;
  extern __shared__ uint8_t t2_smem[];
  uint8_t* q_sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(t2_smem) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* k_sm = q_sm + 2 * TILE;
  uint8_t* v_sm = k_sm + 2 * TILE;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(v_sm + 2 * TILE);
  uint64_t *k_full = q_full + 1, *k_empty = k_full + 2, *v_full = k_empty + 2, *v_empty = v_full + 2;   // [2] each: ring stages
  uint64_t *s_full = v_empty + 2, *p_full = s_full + 2, *o_full = p_full + 2;                            // [2] each: heads
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(o_full + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // ---- which tile: those with the most keys (late tokens) of all heads first
  const int groups = p.num_seqs * (p.Hq / 2);
  const int tile = p.tiles_per_seq - 1 - static_cast<int>(blockIdx.x) / groups;
  const int sh = static_cast<int>(blockIdx.x) % groups;
  const int hq0 = (sh % (p.Hq / 2)) * 2, s = sh / (p.Hq / 2);
  const int hkv = hq0 / (p.Hq / p.Hkv);
  const int q0 = p.cu_q[s], q_len = p.cu_q[s + 1] - q0;
  const int tok0 = tile * kT2Rows;
  if (tok0 >= q_len) return;                          // (whole CTA, before any barrier or TMEM use)
  const int ctx = p.context_lens[s];
  const int pos_base = ctx - q_len;                   // absolute position of query token 0
  const int rows_valid = min(kT2Rows, q_len - tok0);
  const int kv_end = pos_base + tok0 + rows_valid;    // one past the last visible key
  int kv_begin = p.window > 0 ? max(0, pos_base + tok0 - p.window + 1) : 0;
  kv_begin = (kv_begin / kT2Keys) * kT2Keys;
  const int n_tiles = (kv_end - kv_begin + kT2Keys - 1) / kT2Keys;
  const int last_block = (ctx - 1) / kT2Block;        // last pool block the sequence owns

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_full[i], 1);
    }
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_ptr, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_ptr;
  pdl_trigger();
  pdl_wait();                                         // q and the newest keys come from the previous kernels of the step

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    const int* table = p.block_tables + static_cast<size_t>(s) * p.max_blocks;
    const uint64_t pol_q = l2_policy_evict_first(), pol_kv = l2_policy_evict_last();
    if (lane == 0) {
      mbar_expect_tx(q_full, 2 * TILE);
      for (int t = 0; t < 2; ++t)
        for (int c = 0; c < DC; ++c)
          tma_load_2d(q_sm + t * TILE + c * SUB, &map_q, q_full, (hq0 + t) * D + c * 64, q0 + tok0, pol_q);
    }
    for (int j = 0; j < n_tiles; ++j) {
      const int st = j & 1;
      const uint32_t phase = static_cast<uint32_t>(j >> 1) & 1u;
      // one pool block per lane; blocks past the sequence's last one repeat it (masked keys, but the values that meet a weight of
      // zero must be finite)
      int row0 = 0;
      if (lane < kT2Keys / kT2Block) row0 = (table[min(kv_begin / kT2Block + j * (kT2Keys / kT2Block) + lane, last_block)] * p.Hkv + hkv) * kT2Block;
      bool ok = true;
      for (int kv = 0; kv < 2 && ok; ++kv) {
        uint64_t* full = kv ? v_full : k_full;
        if (lane == 0) {
          ok = mbar_wait(kv ? &v_empty[st] : &k_empty[st], phase ^ 1u, p.status, kErrT2Producer);
          if (ok) mbar_expect_tx(&full[st], TILE);
        }
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        if (ok && lane < kT2Keys / kT2Block) {
          uint8_t* dst = (kv ? v_sm : k_sm) + st * TILE + lane * (kT2Block * 128);
          for (int c = 0; c < DC; ++c) tma_load_2d(dst + c * SUB, kv ? &map_v : &map_k, &full[st], c * 64, row0, pol_kv);
        }
        __syncwarp();
      }
      if (!ok) break;
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc_qk = umma_idesc_bf16(kT2Keys, false, false);   // N = keys
      constexpr uint32_t idesc_pv = umma_idesc_bf16(D, false, true);          // N = D, V is MN-major as it sits in the pool
      bool ok = mbar_wait(q_full, 0, p.status, kErrT2Mma);
      auto scores = [&](int t, int j) {               // S_t = Q_t K_j^T
        const uint32_t qa = smem_u32(q_sm + t * TILE), kb = smem_u32(k_sm + (j & 1) * TILE);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk >> 2) * SUB + (kk & 3) * 32;
          umma_bf16(tmem + t * kT2Keys, umma_desc_k_sw128(qa + off), umma_desc_k_sw128(kb + off), idesc_qk, kk > 0 ? 1u : 0u);
        }
      };
      if (ok) ok = mbar_wait(&k_full[0], 0, p.status, kErrT2Mma);
      if (ok) {
        tc_fence_after_sync();
        scores(0, 0);
        umma_commit(&s_full[0]);
        scores(1, 0);
        umma_commit(&k_empty[0]);
        umma_commit(&s_full[1]);
      }
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int st = j & 1, sn = st ^ 1;
        const uint32_t phase = static_cast<uint32_t>(j >> 1) & 1u;
        if (!mbar_wait(&v_full[st], phase, p.status, kErrT2Mma)) break;
        if (j + 1 < n_tiles && !mbar_wait(&k_full[sn], static_cast<uint32_t>((j + 1) >> 1) & 1u, p.status, kErrT2Mma)) break;
        for (int t = 0; t < 2 && ok; ++t) {
          ok = mbar_wait(&p_full[t], static_cast<uint32_t>(j) & 1u, p.status, kErrT2Mma);
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t vb = smem_u32(v_sm + st * TILE);
#pragma unroll
          for (int kk = 0; kk < kT2Keys / 16; ++kk)
            t2_mma_tmem_a(tmem + O_COL + t * D, tmem + t * kT2Keys + kk * 8, umma_desc_mn_sw128(vb + kk * (16 * 128), SUB, 1024), idesc_pv,
                          (j > 0 || kk > 0) ? 1u : 0u);
          if (t == 1) umma_commit(&v_empty[st]);
          if (j + 1 < n_tiles) {
            scores(t, j + 1);                         // (behind O_t in issue order: it overwrites the weights that O_t reads)
            if (t == 1) umma_commit(&k_empty[sn]);
            umma_commit(&s_full[t]);
          } else {
            umma_commit(&o_full[t]);
          }
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax + epilogue
    const int q4 = warp & 3, t = (warp - 2) >> 2;     // TMEM lanes of this warp: 32 q4 ..; its head
    const int row = q4 * 32 + lane;                   // query row == TMEM lane
    const uint32_t s_addr = tmem + (static_cast<uint32_t>(q4 * 32) << 16) + t * kT2Keys;
    const uint32_t o_addr = tmem + (static_cast<uint32_t>(q4 * 32) << 16) + O_COL + t * D;
    const int qpos = pos_base + tok0 + row;           // absolute position of this row's token
    float m_used = -INFINITY;                         // the maximum the stored exponentials refer to (scaled, log2 units)
    float l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_tiles; ++j) {
      ok = mbar_wait(&s_full[t], static_cast<uint32_t>(j) & 1u, p.status, kErrT2Softmax);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t sv[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(s_addr + c * 32, sv[c]);
      tmem_ld_wait();
      const int key0 = kv_begin + j * kT2Keys;
      // only tiles that cross the diagonal, the window's edge or the end need the mask
      if (key0 + kT2Keys - 1 > pos_base + tok0 || (p.window > 0 && key0 < pos_base + tok0 + kT2Rows - p.window)) {
        const int hi = qpos - key0 + 1, lo = p.window > 0 ? qpos - p.window + 1 - key0 : 0;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i < lo || c * 32 + i >= hi) sv[c][i] = 0xff800000u;
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 32; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) mx[c] = fmaxf(mx[c], __uint_as_float(sv[c][i]));
      const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2;
      // lazy rescaling: keep the old reference maximum unless the row grew past it by 2^8
      float alpha = 1.0f;
      bool rescale = false;
      if (top > m_used + kT2Rescale || m_used == -INFINITY) {
        if (top > -INFINITY) {
          alpha = m_used == -INFINITY ? 0.0f : t2_exp2(m_used - top);
          rescale = m_used != -INFINITY;
          m_used = top;
        }
      }
      if (__any_sync(0xffffffffu, rescale)) {         // (O of the key tile before is complete: see s_full)
#pragma unroll 1
        for (int c = 0; c < D; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32(o_addr + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
          tmem_st_32x32(o_addr + c, r);
        }
        tmem_st_wait();
      }
      l *= alpha;
      // P = exp2(s - m) as bf16 pairs over the first 64 columns of the row's scores
      const float neg = m_used == -INFINITY ? 0.f : -m_used;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int c = half * 2 + (i >> 4), e = (i & 15) * 2;
          const float a = t2_exp2(fmaf(__uint_as_float(sv[c][e]), p.scale_log2, neg));         // exp2(-inf) = 0 for masked keys
          const float b = t2_exp2(fmaf(__uint_as_float(sv[c][e + 1]), p.scale_log2, neg));
          sum[i & 1] += a;
          sum[2 + (i & 1)] += b;
          pk[i] = pack_bf16(a, b);
        }
        tmem_st_32x32(s_addr + half * 32, pk);
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[t]);
    }
    // ---- epilogue: O / l -> out
    if (ok) {
      ok = mbar_wait(&o_full[t], 0, p.status, kErrT2Softmax);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      tc_fence_after_sync();
      float osc = 1.0f;
      if (p.sinks != nullptr) {
        const float sk = p.sinks[hq0 + t] * 1.4426950408889634f, m2 = fmaxf(m_used, sk);
        osc = m_used > -INFINITY ? exp2f(m_used - m2) : 0.f;
        l = l * osc + exp2f(sk - m2);
      }
      const float inv = l > 0.f ? osc / l : 0.f;
      __nv_bfloat16* dst = p.out + static_cast<size_t>(q0 + tok0 + row) * p.Hq * D + (hq0 + t) * D;
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(o_addr + c, r);
        tmem_ld_wait();
        if (row < rows_valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 pk;
            pk.x = pack_bf16(__uint_as_float(r[i]) * inv, __uint_as_float(r[i + 1]) * inv);
            pk.y = pack_bf16(__uint_as_float(r[i + 2]) * inv, __uint_as_float(r[i + 3]) * inv);
            pk.z = pack_bf16(__uint_as_float(r[i + 4]) * inv, __uint_as_float(r[i + 5]) * inv);
            pk.w = pack_bf16(__uint_as_float(r[i + 6]) * inv, __uint_as_float(r[i + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c + i) = pk;
          }
        }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

template <int D>
static int launch_prefill_tc2(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const PrefillTc2Params& p, int grid,
                              cudaStream_t stream) {
  constexpr int smem = 6 * (D / 64) * 128 * 128 + 1024 + 256;
  static_assert(smem <= 227 * 1024, "shared memory");
  auto kern = paged_prefill_tc2_kernel<D>;
  // function attributes are per device: a process that drives several GPUs sets them on each
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    prefer_max_shared(kern);
    configured[dev] = true;
  }
  return static_cast<int>(launch_kernel(kern, dim3(grid), dim3(kT2Threads), smem, stream, mq, mk, mv, p));
}

int prefill_tc2_launch(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const PrefillTc2Params& p, int D, int grid,
                       cudaStream_t stream) {
  return D == 128 ? launch_prefill_tc2<128>(mq, mk, mv, p, grid, stream) : launch_prefill_tc2<64>(mq, mk, mv, p, grid, stream);
}

}  // namespace mx
