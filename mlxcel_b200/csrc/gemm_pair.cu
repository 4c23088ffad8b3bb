// Dense bf16 GEMM on pairs of SMs, for many token rows (prompt portions): out[M, N] = epilogue(x[M, K] @ w[N, K]^T).
//
// The tile of one SM, 128 tokens x 256 weight rows, makes the tensor core read 48 KB of shared memory per 64 of K, 384 cycles at
// 128 bytes each, for 256 cycles of products: it cannot pass two thirds of the peak. Two SMs of a TPC that share one tile of
// 256 x 256 (tcgen05 cta_group::2) each hold their own 128 tokens and HALF of the weight rows, 32 KB per 64 of K: 256 cycles.
//
//   cluster = 2 CTAs, persistent, one pair per TPC. Warps of a CTA:
//   warp 0     TMA producer: this CTA's 128 token rows and its half of the weight rows into a ring of 64-wide K slices; the
//              bytes of both CTAs are counted on the LEADER's (even CTA's) barrier.
//   warp 1     leader: one thread issues tcgen05.mma (M = 256, N = 256) for both SMs and commits to both CTAs' barriers
//   warps 2-5  epilogue: this CTA's 128 rows of the accumulator (one TMEM lane = one thread = one token), double-buffered
// Gated: the two halves of the weight rows are 128 gate and 128 up rows, so columns c and 128 + c of a row are a pair.
//
// Measured on B200 (us, single-SM tiles of gemm.cu in brackets; same bits in both): M 8192: N 4096 K 4096 209 (275), N 6144 321
// (374), N 4096 K 14336 837 (869); M 2048: N 4096 K 4096 85 (120), N 6144 121 (164), N 28672 391 (487); M 512: N 4096 K 4096 39
// (64), N 28672 116 (152), N 5120 K 2880 31 (51). Long runs end at 1150 to 1300 TFLOP/s, where the power cap holds them; at few
// tiles the epilogue counts as much as the operands (a thread's whole 64-byte pieces of its row against 16-byte ones).
#include <cooperative_groups.h>

#include "api.h"
#include "common.cuh"
#include "gemm_pair.cuh"

namespace mx {

constexpr int kGpBK = 64;
constexpr int kGpStages = 6;
constexpr int kGpHalf = 128 * kGpBK * 2;            // bytes of one operand slice of one CTA
constexpr int kGpStageBytes = 2 * kGpHalf;
constexpr int kGpThreads = 192;
constexpr int kGpSmem = kGpStages * kGpStageBytes + 1024 /* alignment */ + 256;

__device__ __forceinline__ uint32_t gp_leader(const void* p) {          // the leader's copy of a shared-memory location
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
__device__ __forceinline__ void gp_tma_load(void* dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, uint64_t policy) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint"
               " [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1), "l"(policy)
               : "memory");
}
__device__ __forceinline__ void gp_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred P;\n\tsetp.ne.b32 P, %4, 0;\n\t"
               "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, P;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
               : "memory");
}
__device__ __forceinline__ void gp_commit(uint64_t* bar) {               // arrives on this barrier of BOTH CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}
__device__ __forceinline__ void gp_arrive(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// mbar_wait with acquire at cluster scope: the arrivals come from the other SM too.
__device__ __forceinline__ bool gp_wait(uint64_t* bar, uint32_t parity, int* status, int code) {
  const unsigned long long t0 = globaltimer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 128; ++i) {
      uint32_t ok;
      asm volatile("{\n\t.reg .pred P;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\tselp.u32 %0, 1, 0, P;\n\t}"
                   : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
      if (ok) return true;
    }
    if (*reinterpret_cast<volatile int*>(status) != 0) return false;
    if (globaltimer_ns() - t0 > kWaitLimitNs) {
      atomicCAS(status, 0, code);
      return false;
    }
  }
}

__device__ __forceinline__ float gp_act(int epilogue, float g, float u, float alpha, float limit) {
  float z = g;
  if (epilogue == MX_EPI_GEGLU) {
    z = 2.0f * 0.7978845608028654f * (g + 0.044715f * g * g * g);
  } else if (epilogue == MX_EPI_CLIPPED_SWIGLU) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit) + 1.0f;
    z = alpha * g;
  }
  return __fdividef(g, 1.0f + __expf(-z)) * u;
}

template <bool GLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGpThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const GemmPairParams p) {
  constexpr int FEATS = GLU ? 128 : 256;              // output features of a tile
  extern __shared__ uint8_t gp_smem[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gp_smem) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(ring + kGpStages * kGpStageBytes);   // leader: both CTAs' slices landed
  uint64_t* empty_bar = full_bar + kGpStages;         // the products that read the stage are done
  uint64_t* tmem_full = empty_bar + kGpStages;
  uint64_t* tmem_empty = tmem_full + 2;               // leader: both CTAs' epilogues have read the accumulator
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank());
  const int pair = static_cast<int>(blockIdx.x) >> 1, pairs = static_cast<int>(gridDim.x) >> 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = p.tiles_m * p.tiles_n;

  // tile t -> first token row and first weight row (feature): panels of `raster` row tiles x all column tiles, row tile fastest, so
  // that a panel's tokens stay in L2 while the weights pass once per panel
  auto place = [&](int t, int& m0, int& f0) {
    const int per_panel = p.raster * p.tiles_n, g = t / per_panel, r = t - g * per_panel;
    const int rows = min(p.raster, p.tiles_m - g * p.raster);
    m0 = (g * p.raster + r % rows) * 256;
    f0 = (r / rows) * FEATS;
  };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_x);
    tma_prefetch_desc(&map_w);
    for (int s = 0; s < kGpStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 8);                   // four epilogue warps of each CTA
    }
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before_sync();
  cluster.sync();                                     // the other CTA's barriers are there
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_ptr;
  pdl_trigger();

  if (warp == 0) {
    if (lane == 0) {
      const uint64_t keep = l2_policy_evict_last(), stream = l2_policy_evict_first();
      const int num_kb = (p.K + kGpBK - 1) / kGpBK;
      const uint32_t bars = gp_leader(full_bar);
      auto load_w = [&](int s, int kb, int f0) {
        const int row = GLU ? (rank == 0 ? f0 : p.glu_offset + f0) : f0 + rank * 128;
        gp_tma_load(ring + s * kGpStageBytes + kGpHalf, &map_w, bars + 8 * s, kb * kGpBK, row, stream);
      };
      auto load_x = [&](int s, int kb, int m0) {
        gp_tma_load(ring + s * kGpStageBytes, &map_x, bars + 8 * s, kb * kGpBK, m0 + rank * 128, keep);
      };
      // weights are nobody's output, unless the call says so: the first ring of them is under way before the previous kernel has ended
      int pre = 0;
      if (!p.w_fresh && pair < tiles) {
        int m0, f0;
        place(pair, m0, f0);
        pre = min(kGpStages, num_kb);
        for (int s = 0; s < pre; ++s) {
          if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * kGpStageBytes);
          load_w(s, s, f0);
        }
      }
      pdl_wait();
      int stage = 0, seq = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; ok && t < tiles; t += pairs) {
        int m0, f0;
        place(t, m0, f0);
        for (int kb = 0; kb < num_kb; ++kb, ++seq) {
          if (seq >= pre) {
            if (!gp_wait(&empty_bar[stage], phase ^ 1u, p.status, kErrProducerWait)) {
              ok = false;
              break;
            }
            if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * kGpStageBytes);
            load_w(stage, kb, f0);
          }
          load_x(stage, kb, m0);
          if (++stage == kGpStages) stage = 0, phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0 && lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(256, false, false, 256);
      const int num_kb = (p.K + kGpBK - 1) / kGpBK;
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int t = pair; ok && t < tiles; t += pairs) {
        if (!gp_wait(&tmem_empty[acc], acc_phase ^ 1u, p.status, kErrMmaWaitTmem)) break;
        tc_fence_after_sync();
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!gp_wait(&full_bar[stage], phase, p.status, kErrMmaWaitFull)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(ring + stage * kGpStageBytes), sb = sa + kGpHalf;
#pragma unroll
          for (int kk = 0; kk < kGpBK / 16; ++kk)
            gp_mma(tmem + acc * 256, umma_desc_k_sw128(sa + kk * 32), umma_desc_k_sw128(sb + kk * 32), idesc, (kb > 0 || kk > 0) ? 1u : 0u);
          gp_commit(&empty_bar[stage]);
          if (++stage == kGpStages) stage = 0, phase ^= 1u;
        }
        if (!ok) break;
        gp_commit(&tmem_full[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t done = gp_leader(tmem_empty);
    int acc = 0;
    uint32_t acc_phase = 0;
    pdl_wait();                                       // bias, residual and sums of squares may be the previous kernel's
    for (int t = pair; t < tiles; t += pairs) {
      int m0, f0;
      place(t, m0, f0);
      const int m = m0 + rank * 128 + row;
      const bool live = m < p.M;
      float scale = 1.f;
      if (p.ssq_in != nullptr) {                      // deferred RMSNorm of the input rows, summed while the products run
        const int parts = reinterpret_cast<const int*>(p.ssq_in)[0], ld = reinterpret_cast<const int*>(p.ssq_in)[1];
        float ss = 0.f;
        if (live)
          for (int i = 0; i < parts; ++i) ss += __ldcg(p.ssq_in + 8 + static_cast<size_t>(i) * ld + m);
        scale = rsqrtf(ss * p.ssq_inv_dim + p.ssq_eps);
      }
      const bool ok = gp_wait(&tmem_full[acc], acc_phase, p.status, kErrEpilogueWait);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after_sync();
      const uint32_t taddr = tmem + (static_cast<uint32_t>(q * 32) << 16) + acc * 256;
      const int valid = p.N - f0;                     // (N is a multiple of 8: 16-byte pieces are in or out as a whole)
      const __nv_bfloat16* res = p.residual != nullptr && live ? p.residual + static_cast<size_t>(m) * p.ldr + f0 : nullptr;
      __nv_bfloat16* out = p.out + static_cast<size_t>(live ? m : 0) * p.ldo + f0;
      float ssq = 0.f;
#pragma unroll 1
      for (int c = 0; c < FEATS; c += 32) {
        uint4 rs[4];
        if (!GLU && res != nullptr) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            rs[i] = c + i * 8 < valid ? *reinterpret_cast<const uint4*>(res + c + i * 8) : make_uint4(0, 0, 0, 0);
        }
        uint32_t r[32];
        [[maybe_unused]] uint32_t u[32];
        tmem_ld_32x32(taddr + c, r);
        if constexpr (GLU) tmem_ld_32x32(taddr + 128 + c, u);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int f = c + i * 8;
          if (f >= valid) break;
          float o[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = __uint_as_float(r[i * 8 + j]) * scale;
          if (p.bias != nullptr) {
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] += __bfloat162float(p.bias[f0 + f + j]);
          }
          if constexpr (GLU) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float up = __uint_as_float(u[i * 8 + j]) * scale;
              if (p.bias != nullptr) up += __bfloat162float(p.bias[p.glu_offset + f0 + f + j]);
              o[j] = gp_act(p.epilogue, o[j], up, p.glu_alpha, p.glu_limit);
            }
          } else if (res != nullptr) {
            const uint32_t w4[4] = {rs[i].x, rs[i].y, rs[i].z, rs[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) o[2 * j] += bf16_lo(w4[j]), o[2 * j + 1] += bf16_hi(w4[j]);
          }
          const uint4 pk = make_uint4(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]), pack_bf16(o[4], o[5]), pack_bf16(o[6], o[7]));
          if (!GLU && p.ssq_out != nullptr) {
            const uint32_t w4[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) ssq += bf16_lo(w4[j]) * bf16_lo(w4[j]) + bf16_hi(w4[j]) * bf16_hi(w4[j]);
          }
          if (live) *reinterpret_cast<uint4*>(out + f) = pk;
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) gp_arrive(done + 8 * acc);
      if (!GLU && p.ssq_out != nullptr) {
        const int ld = reinterpret_cast<const int*>(p.ssq_out)[1];
        if (live) p.ssq_out[8 + static_cast<size_t>(f0 / 256) * ld + m] = ssq;
        if (t == 0 && rank == 0 && threadIdx.x == 64) reinterpret_cast<int*>(p.ssq_out)[0] = p.tiles_n;
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  tc_fence_before_sync();
  cluster.sync();                                     // nothing more arrives from or is read in the other CTA
  if (warp == 1) {
    tc_fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// Whether the pair kernel takes a call and is the faster one. Both kernels run in waves of whole tiles, 256 rows here and 128 in the
// single-SM kernel, so a ragged M or a last wave that is nearly empty can cost more than the pairing gives. A wave of single-SM
// tiles takes at least 1.25 times a wave of pair tiles (5 waves against 4 at M 543, N 28672: 143 us against 154; 4 against 3 at M
// 300: 118 against 118); gated it takes about as long (8192 x 14336, K 4096: 1575 against 1644; 5 against 4 waves at M 543: 155
// against 134), as the single-SM kernel's gated epilogue has half the outputs to write.
static bool pair_is_faster(int M, int N, bool glu, int sms) {
  if (M <= 256 || (!glu && N <= 128)) return false;
  const int feats = glu ? 128 : 256;
  const long long n = (N + feats - 1) / feats, pairs = sms / 2;
  const long long waves = ((M + 255) / 256 * n + pairs - 1) / pairs, single = ((M + 127) / 128 * n + sms - 1) / sms;
  return waves * 100 <= single * (glu ? 104 : 125);
}
bool gemm_pair_wanted(const GemmPairParams& p, bool glu, int sms) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.residual);
  return p.N % 8 == 0 && p.ldo % 8 == 0 && p.ldr % 8 == 0 && (a & 15) == 0 && p.status != nullptr && pair_is_faster(p.M, p.N, glu, sms);
}

int gemm_pair_launch(const CUtensorMap& map_x, const CUtensorMap& map_w, GemmPairParams p, bool glu, int sms, cudaStream_t stream) {
  const int feats = glu ? 128 : 256;
  p.tiles_m = (p.M + 255) / 256;
  p.tiles_n = (p.N + feats - 1) / feats;
  p.raster = 8;
  const long long tiles = static_cast<long long>(p.tiles_m) * p.tiles_n;
  const int pairs = static_cast<int>(tiles < sms / 2 ? tiles : sms / 2);
  auto kern = glu ? gemm_pair_kernel<true> : gemm_pair_kernel<false>;
  // function attributes are per device: a process that drives several GPUs sets them on each
  static bool configured[2][64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!configured[glu][dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kGpSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    prefer_max_shared(kern);
    configured[glu][dev] = true;
  }
  return static_cast<int>(launch_kernel(kern, dim3(2 * pairs), dim3(kGpThreads), kGpSmem, stream, map_x, map_w, p));
}

}  // namespace mx

extern "C" int mx_gemm_on_pairs(int M, int N, int glu) { return N % 8 == 0 && mx::pair_is_faster(M, N, glu != 0, mx::device_sm_count()); }
