// Grouped 4-bit weight-streaming matrix products for mixture-of-experts decode: a few token rows per expert, straight from
// the checkpoint's packed layout.
//
// Bound by the bytes of the packed weights (0.53 to 0.56 per weight) if the SM can unpack them fast enough: at the copy
// bandwidth an SM has to take 42 weights per cycle, so issue slots and the latency between dependent instructions are what
// is scarce, and everything is laid out around them (reference: gather_qmm for SwitchGLU, src/models/switch_layers.rs:98-220;
// overlays/cuda/.../quantized/qmm/qmv.cu):
//
//   grid  = (K split, output-feature blocks, local experts); a block whose expert got no rows returns as soon as it knows, and
//           where few experts are in use nothing of its weights has been asked for by then (mx_qstream_ahead).
//   warp  = one 16-row A tile of mma.sync m16n8k16: 16 features, or 8 features x (gate row, up row) when gated, so that a gate
//           value and its up value meet in one lane. Every warp brings its own rows by cp.async into a ring of its own (64
//           bytes = 128 weights of a row a stage, XOR-swizzled pieces), so no barrier stands between the stages.
//   A     = a quad of lanes reads 64 weights of a row at once (32 where groups are that small), two MMA steps a 32-bit word.
//           affine: the code pairs (i, i + 4) of a word become bf16 pairs 16 + code with one shift and one lop3 (the code
//           lands on mantissa bits 3..6 of 16.0), and the activations are staged in that pair order; exact, no rounded weight
//           exists. mxfp4: the hardware e2m1x2 -> f16x2 conversion (activations as fp16).
//   B     = up to 8 * NT token rows staged in shared memory per K slab, one 16-byte read = two steps.
//   C     = per scale group a fresh fp32 accumulator, folded into the running sum with the group's scale; affine adds
//           (bias - 16 scale) * sum(x), the sums taken in fp32 when x is staged.
//   K     = split over the CTAs of a cluster where the row tiles of the experts in use leave SMs idle; the partial tiles meet
//           over distributed shared memory in rank order (deterministic), without a workspace.
//
// Measured on B200 (mxfp4, 128 experts of 2880 x 2880, top 4 of 128 rows): gate/up 393 us and down 211 us, 44 % of the copy
// bandwidth; 1312 us for the two with the lanes of a quad reading the same 16 bytes and picking their codes by byte permutes.
// 8 rows 97 and 56 us, 1 row 39 and 26 us. Counters at 128 rows: issue slots 73 %, integer pipe 69 %, LSU wavefronts 44 %, DRAM 35 %.
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include "api.h"
#include "common.cuh"
#include "mma_sync.cuh"

namespace mx {

constexpr int kQsWarps = 8;
constexpr int kQsThreads = kQsWarps * 32;
constexpr int kQsBlockK = 128;       // weights of a row per stage
constexpr int kQsRowBytes = kQsBlockK / 2;
constexpr int kQsMaxSplit = 8;       // CTAs of a cluster along K

struct QsParams {
  const __nv_bfloat16* xs;        // [rows, K]: rows of expert e are [offsets[e], offsets[e + 1])
  const uint8_t* w;               // [E, N, K / 2] bytes, code 2i in the low nibble of byte i
  const uint8_t* scales;          // affine: bf16 [E, N, K / group]; mxfp4: e8m0 bytes
  const uint8_t* biases;          // affine only
  const __nv_bfloat16* lin_bias;  // [E, N] or null
  const int* offsets;             // [E + 1]
  __nv_bfloat16* out;             // [rows, n_out]
  int N, K, n_out, epi;
  int k_per_cta;                  // multiple of 128
  int ahead;                      // the first stages are loaded before it is known whether the expert has rows
  float alpha, limit;
};

template <int MODE, int NT>
struct QsShape {
  static constexpr int kTok = 8 * NT;
  static constexpr int kSlabK = NT == 1 ? (MODE == 0 ? 1024 : 1536) : 512;
  static constexpr int kXStride = kSlabK * 2 + 64;               // bytes; 64 mod 128: conflict-free 16-byte reads
  static constexpr int kRows = kQsWarps * 16;                    // tile rows of a CTA
  static constexpr int kStages = 4;
  static constexpr int kScaleRow = MODE == 0 ? 32 : 8;           // bytes of a row's scales in a stage (affine: 16 scales, 16 biases)
  static constexpr int kStageBytes = 16 * (kQsRowBytes + kScaleRow);
  static constexpr int kRingBytes = kQsWarps * kStages * kStageBytes;
  static constexpr int kXBytes = kTok * kXStride;
  static constexpr int kSumBytes = MODE == 0 ? (kSlabK / 32) * kTok * 4 : 0;
  static constexpr int kPartStride = kRows + 4;                  // floats; the 8 x 4 fragment writes hit 32 banks
  static constexpr int kPartBytes = kTok * kPartStride * 4;      // (takes the ring's place once it is drained)
  static constexpr int kSmem = kXBytes + kSumBytes + (kRingBytes > kPartBytes ? kRingBytes : kPartBytes);
  static constexpr int kResident = NT == 1 ? 3 : 2;              // CTAs an SM: registers and shared memory are sized for it
};

__device__ __forceinline__ float qs_e8m0(uint32_t s) {
  if (s == 255) return __uint_as_float(0x7fc00000u);
  if (s == 0) return __uint_as_float(0x00400000u);
  return __uint_as_float(s << 23);
}
__device__ __forceinline__ uint32_t qs_and_or(uint32_t a, uint32_t mask, uint32_t bits) { return (a & mask) | bits; }

template <int MODE>
__device__ __forceinline__ void qs_unpack(uint32_t w, uint32_t (&v)[4]) {
  if (MODE == 0) {
    v[0] = qs_and_or(w << 3, 0x00780078u, 0x41804180u);   // codes 0, 4
    v[1] = qs_and_or(w >> 1, 0x00780078u, 0x41804180u);   // codes 1, 5
    v[2] = qs_and_or(w >> 5, 0x00780078u, 0x41804180u);   // codes 2, 6
    v[3] = qs_and_or(w >> 9, 0x00780078u, 0x41804180u);   // codes 3, 7
  } else {
    asm("{ .reg .b8 a, b, c, d;\n mov.b32 {a, b, c, d}, %4;\n"
        " cvt.rn.f16x2.e2m1x2 %0, a;\n cvt.rn.f16x2.e2m1x2 %1, b;\n"
        " cvt.rn.f16x2.e2m1x2 %2, c;\n cvt.rn.f16x2.e2m1x2 %3, d;\n }"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(w));
  }
}

template <int MODE>
__device__ __forceinline__ void qs_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if (MODE == 0)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The first product of a group: accumulator zero.
template <int MODE>
__device__ __forceinline__ void qs_mma0(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if (MODE == 0)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ uint64_t qs_pair(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float2 qs_unpair(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ void qs_fma2(uint64_t& c, uint64_t a, uint64_t b) {   // two fp32 multiply-adds
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

__device__ __forceinline__ float qs_glu(int epi, float g, float u, float alpha, float limit) {
  if (epi == MX_EPI_SWIGLU) return g / (1.f + __expf(-g)) * u;
  if (epi == MX_EPI_GEGLU) {
    const float c = 0.7978845608028654f * (g + 0.044715f * g * g * g);
    return 0.5f * g * (1.f + tanhf(c)) * u;
  }
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g / (1.f + __expf(-alpha * g)) * (u + 1.f);
}

// MODE 0 affine, 1 mxfp4. NT: 8-token column tiles of a pass. LG: log2 of the scale group (5 for mxfp4).
template <int MODE, int NT, int LG>
__global__ void __launch_bounds__(kQsThreads, QsShape<MODE, NT>::kResident) qstream_kernel(const QsParams p) {
  using S = QsShape<MODE, NT>;
  constexpr int SZ = MODE == 0 ? 2 : 1;                           // bytes of a scale
  constexpr int UNIT = LG == 5 ? 32 : 64;                         // weights a quad reads of a row at once, all of one group
  constexpr int WORDS = UNIT / 32;                                // of them a lane's 32-bit words
  constexpr int RING = S::kStages * S::kStageBytes;
  extern __shared__ __align__(128) uint8_t smem[];
  uint8_t* xs_s = smem;
  float* sum_s = reinterpret_cast<float*>(smem + S::kXBytes);
  uint8_t* ring_all = smem + S::kXBytes + S::kSumBytes;
  float* part = reinterpret_cast<float*>(ring_all);

  namespace cg = cooperative_groups;
  const int splits = static_cast<int>(gridDim.x);                 // cluster = the CTAs along K of one row block
  const int split = static_cast<int>(blockIdx.x);
  const int e = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = lane >> 2, q = lane & 3;
  const bool gated = p.epi >= MX_EPI_SWIGLU;
  const int feats = gated ? 8 : 16;                               // output features of a tile
  const int f_cta = static_cast<int>(blockIdx.y) * (S::kRows / 16) * feats;
  const int k_begin = split * p.k_per_cta, k_end = min(p.K, k_begin + p.k_per_cta);
  const size_t ebase = static_cast<size_t>(e) * p.N;

  // the lane's rows r and r + 8 (rows past the last feature read row 0; their results go nowhere)
  const uint8_t* w_row[2];                                        // at this lane's 16-byte piece of the range's first stage
  uint32_t s_off[2];                                              // byte of the first scale of the range
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int f = f_cta + warp * feats + r + (gated ? 0 : 8 * h);
    const size_t n = ebase + (f < p.n_out ? (gated && h ? p.n_out + f : f) : 0);
    w_row[h] = p.w + n * (static_cast<size_t>(p.K) >> 1) + (k_begin >> 1) + q * 16;
    s_off[h] = (static_cast<uint32_t>(n) * static_cast<uint32_t>(p.K >> LG) + static_cast<uint32_t>(k_begin >> LG)) * SZ;
  }
  const uint32_t ring = smem_u32(ring_all) + warp * RING;
  const uint32_t w_dst = r * kQsRowBytes + ((q ^ (LG == 5 ? (r >> 1) & 3 : r & 2)) << 4);
  const uint32_t s_dst = 16 * kQsRowBytes + r * S::kScaleRow;

  // One stage: 128 weights and their scales of the warp's rows; what lies past the range is zero-filled. The scales come as
  // the aligned 32-bit words around them.
  int ld_k = 0;                                                   // from k_begin
  uint32_t ld_st = 0;
  auto load = [&]() {
    const int kn = k_end - k_begin - ld_k;
    if (kn > 0) {
      const uint32_t need = static_cast<uint32_t>(min(kn, kQsBlockK) >> LG) * SZ;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const bool in = q * 32 < kn;
        cp_async16(ring + ld_st + w_dst + h * 8 * kQsRowBytes, w_row[h] + (in ? ld_k >> 1 : 0), in);
        const uint32_t off = s_off[h] + static_cast<uint32_t>(ld_k >> LG) * SZ, at = off & ~3u;
        const uint32_t dst = ring + ld_st + s_dst + h * 8 * S::kScaleRow;
        auto word = [&](const uint8_t* base, uint32_t i, uint32_t d) {
          const bool ok = at + i * 4 < off + need;
          cp_async_small<4>(d, base + (ok ? at + i * 4 : 0u), ok);
        };
        if (MODE == 1) {
          if (q < 2) word(p.scales, q, dst + q * 4);
        } else if (LG == 5) {
          if (q < 3) {
            word(p.scales, q, dst + q * 4);
            word(p.biases, q, dst + 16 + q * 4);
          }
        } else {
          word(q < 2 ? p.scales : p.biases, q & 1, dst + (q >> 1) * 16 + (q & 1) * 4);
        }
      }
    }
    ld_k += kQsBlockK;
    ld_st = ld_st + S::kStageBytes == RING ? 0 : ld_st + S::kStageBytes;
    cp_async_commit();
  };
  if (p.ahead) {                                                  // weights are nobody's output: before the wait
#pragma unroll
    for (int i = 0; i < S::kStages - 1; ++i) load();
  }
  pdl_wait();
  pdl_trigger();

  const int row0 = p.offsets[e], m_e = p.offsets[e + 1] - row0;
  if (m_e <= 0) {                                                 // (the same for every CTA of the cluster)
    cp_async_wait<0>();
    return;
  }
  if (!p.ahead) {
#pragma unroll
    for (int i = 0; i < S::kStages - 1; ++i) load();
  }
  for (int t0 = 0; t0 < m_e; t0 += S::kTok) {
    const int toks = min(S::kTok, m_e - t0);
    const int nt = (toks + 7) >> 3;
    if (t0 > 0) {                                                 // another pass over the weights
      __syncthreads();                                            // (the ring served as the partial tile)
      ld_k = 0, ld_st = 0;
#pragma unroll
      for (int i = 0; i < S::kStages - 1; ++i) load();
    }
    uint64_t acc[NT][2];                                          // (rows r, r + 8: tokens 2q, 2q + 1)
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = 0;

    uint32_t st_off = 0;                                          // the stage in use
    for (int k_slab = k_begin; k_slab < k_end; k_slab += S::kSlabK) {
      const int ks = min(S::kSlabK, k_end - k_slab);
      const int ks_pad = (ks + kQsBlockK - 1) & ~(kQsBlockK - 1);
      __syncthreads();                                            // the previous slab is consumed
      // ---- stage the slab: 8 activations per item, items of a token back to back
      const int per_tok = ks_pad >> 3, items = toks * per_tok;
      const __nv_bfloat16* xg = p.xs + static_cast<size_t>(row0 + t0) * p.K + k_slab;
      constexpr int kBatch = NT >= 3 ? 4 : 2;
      for (int i0 = threadIdx.x & ~31; i0 < items; i0 += kQsThreads * kBatch) {
        uint4 v[kBatch];
        int tk[kBatch], ck[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
          const int i = i0 + j * kQsThreads + lane;
          tk[j] = i < items ? i / per_tok : -1;
          ck[j] = i - (tk[j] < 0 ? 0 : tk[j]) * per_tok;
          v[j] = make_uint4(0, 0, 0, 0);
          if (tk[j] >= 0 && ck[j] * 8 < ks) v[j] = *reinterpret_cast<const uint4*>(xg + static_cast<size_t>(tk[j]) * p.K + ck[j] * 8);
        }
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
          if (i0 + j * kQsThreads >= items) break;                // (the same for the whole warp)
          if (MODE == 0) {
            float s = bf16_lo(v[j].x) + bf16_hi(v[j].x) + bf16_lo(v[j].y) + bf16_hi(v[j].y) + bf16_lo(v[j].z) + bf16_hi(v[j].z) +
                      bf16_lo(v[j].w) + bf16_hi(v[j].w);
            s += __shfl_xor_sync(0xffffffffu, s, 1);              // sums of a group's activations: 4, 8 or 16 items of 8
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if (LG >= 6) s += __shfl_xor_sync(0xffffffffu, s, 4);
            if (LG >= 7) s += __shfl_xor_sync(0xffffffffu, s, 8);
            if (tk[j] >= 0 && (ck[j] & ((1 << LG) / 8 - 1)) == 0) sum_s[(ck[j] >> (LG - 3)) * S::kTok + tk[j]] = s;
            const uint4 u = v[j];
            v[j] = make_uint4(__byte_perm(u.x, u.z, 0x5410), __byte_perm(u.x, u.z, 0x7632), __byte_perm(u.y, u.w, 0x5410),
                              __byte_perm(u.y, u.w, 0x7632));
          } else {
            const __half2 h[4] = {__floats2half2_rn(bf16_lo(v[j].x), bf16_hi(v[j].x)), __floats2half2_rn(bf16_lo(v[j].y), bf16_hi(v[j].y)),
                                  __floats2half2_rn(bf16_lo(v[j].z), bf16_hi(v[j].z)), __floats2half2_rn(bf16_lo(v[j].w), bf16_hi(v[j].w))};
            v[j] = *reinterpret_cast<const uint4*>(h);
          }
          // (a lane of a 64-weight unit takes items 2q, 2q + 1: they go 64 bytes apart, four lanes side by side)
          const int pos = UNIT == 32 ? ck[j] : (ck[j] & ~7) + (ck[j] & 1) * 4 + ((ck[j] >> 1) & 3);
          if (tk[j] >= 0) *reinterpret_cast<uint4*>(xs_s + tk[j] * S::kXStride + pos * 16) = v[j];
        }
      }
      __syncthreads();
      // ---- the warp walks the slab's blocks
      const uint8_t* xb = xs_s + r * S::kXStride + q * 16;
      const float* xsum = sum_s + 2 * q;
      for (int k0 = k_slab; k0 < k_slab + ks; k0 += kQsBlockK) {
        cp_async_wait<S::kStages - 2>();
        __syncwarp();
        load();                                                   // (into the slot of the block before this one)
        uint8_t* st = ring_all + warp * RING + st_off;
        st_off = st_off + S::kStageBytes == RING ? 0 : st_off + S::kStageBytes;
        if (LG < 7 && k0 + kQsBlockK > p.K) {
          // A last block that is not full: behind the row's own scales its words hold the next row's, and a NaN or an infinity
          // there would spoil this row even times the zeros of the missing weights. (Cleared in place, with the offsets indexed so
          // that they are kept in local memory for this branch: masks in registers cost 1 to 3 %, exact fetches 4 to 10 %.)
          if (q < 2) {
            uint8_t* row = st + 16 * kQsRowBytes + (q * 8 + r) * S::kScaleRow;
            const uint32_t first = s_off[q] + static_cast<uint32_t>((k0 - k_begin) >> LG) * SZ;
            for (uint32_t i = (first & 3) + ((p.K - k0) >> LG) * SZ; i < (MODE == 0 ? 12u : 8u); ++i) {
              row[i] = 0;
              if (MODE == 0) row[16 + i] = 0;
            }
          }
          __syncwarp();
        }
        // the block's scales of the lane's rows
        uint32_t sw[2][2], bw[2][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t* row = reinterpret_cast<const uint32_t*>(st + 16 * kQsRowBytes + (h * 8 + r) * S::kScaleRow);
          const uint2 a = *reinterpret_cast<const uint2*>(row);
          const uint32_t sh = ((s_off[h] + static_cast<uint32_t>((k0 - k_begin) >> LG) * SZ) & 3) * 8;
          sw[h][0] = __funnelshift_r(a.x, a.y, sh);
          if (MODE == 0) {
            const uint2 b = *reinterpret_cast<const uint2*>(row + 4);
            bw[h][0] = __funnelshift_r(b.x, b.y, sh);
            if (LG == 5) {
              sw[h][1] = __funnelshift_r(a.y, row[2], sh);
              bw[h][1] = __funnelshift_r(b.y, row[6], sh);
            }
          }
        }
#pragma unroll
        for (int g = 0; g < (kQsBlockK >> LG); ++g) {             // scale groups
          float d[NT][4];
#pragma unroll
          for (int i = 0; i < (1 << LG) / 32; ++i) {              // the lane's words of the group
            const int wi = g * ((1 << LG) / 32) + i, u = wi / WORDS, w = wi % WORDS;
            const uint32_t piece = LG == 5 ? ((u ^ ((r >> 1) & 3)) << 4) + q * 4
                                           : (((u * 2 + (q >> 1)) ^ (r & 2)) << 4) + (q & 1) * 8 + w * 4;
            const uint8_t* wr = st + r * kQsRowBytes + piece;
            uint32_t a[4], c[4];
            qs_unpack<MODE>(*reinterpret_cast<const uint32_t*>(wr), a);
            qs_unpack<MODE>(*reinterpret_cast<const uint32_t*>(wr + 8 * kQsRowBytes), c);
#pragma unroll
            for (int n = 0; n < NT; ++n)
              if (NT == 1 || n < nt) {
                const uint4 b = *reinterpret_cast<const uint4*>(xb + n * 8 * S::kXStride + wi * 64);
                if (i == 0) qs_mma0<MODE>(d[n], a[0], c[0], a[1], c[1], b.x, b.y);
                else qs_mma<MODE>(d[n], a[0], c[0], a[1], c[1], b.x, b.y);
                qs_mma<MODE>(d[n], a[2], c[2], a[3], c[3], b.z, b.w);
              }
          }
          float s[2], c[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (MODE == 0) {
              s[h] = g & 1 ? bf16_hi(sw[h][g >> 1]) : bf16_lo(sw[h][g >> 1]);
              c[h] = fmaf(-16.f, s[h], g & 1 ? bf16_hi(bw[h][g >> 1]) : bf16_lo(bw[h][g >> 1]));
            } else {
              s[h] = qs_e8m0((sw[h][0] >> (8 * g)) & 255u);
            }
          }
          const uint64_t s0 = qs_pair(s[0], s[0]), s1 = qs_pair(s[1], s[1]);
#pragma unroll
          for (int n = 0; n < NT; ++n)
            if (NT == 1 || n < nt) {
              if (MODE == 0) {
                const uint64_t x2 = *reinterpret_cast<const uint64_t*>(xsum + g * S::kTok + n * 8);
                qs_fma2(acc[n][0], qs_pair(c[0], c[0]), x2);
                qs_fma2(acc[n][1], qs_pair(c[1], c[1]), x2);
              }
              qs_fma2(acc[n][0], s0, qs_pair(d[n][0], d[n][1]));
              qs_fma2(acc[n][1], s1, qs_pair(d[n][2], d[n][3]));
            }
        }
        xb += kQsBlockK * 2;
        xsum += (kQsBlockK >> LG) * S::kTok;
      }
    }
    cp_async_wait<0>();

    // ---- partial tile: [token][tile row], through shared memory so that features store back to back
    __syncthreads();                                              // every warp is through with its ring
#pragma unroll
    for (int n = 0; n < NT; ++n)
      if (NT == 1 || n < nt) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 v = qs_unpair(acc[n][h]);
          float* to = part + (n * 8 + 2 * q) * S::kPartStride + warp * 16 + r + h * 8;
          to[0] = v.x;
          to[S::kPartStride] = v.y;
        }
      }
    cg::cluster_group cluster = cg::this_cluster();
    if (splits > 1) cluster.sync(); else __syncthreads();
    const int cta_feats = (S::kRows / 16) * feats;
    for (int i = split * kQsThreads + static_cast<int>(threadIdx.x); i < toks * cta_feats; i += splits * kQsThreads) {
      const int t = i / cta_feats, fl = i - t * cta_feats, f = f_cta + fl;
      if (f >= p.n_out) continue;
      const int row = gated ? (fl >> 3) * 16 + (fl & 7) : fl;
      float a = 0.f, b = 0.f;
      for (int c = 0; c < splits; ++c) {
        const float* src = (splits > 1 ? cluster.map_shared_rank(part, c) : part) + t * S::kPartStride + row;
        a += src[0];
        if (gated) b += src[8];
      }
      if (p.lin_bias) {
        a += __bfloat162float(p.lin_bias[ebase + f]);
        if (gated) b += __bfloat162float(p.lin_bias[ebase + p.n_out + f]);
      }
      if (gated) a = qs_glu(p.epi, a, b, p.alpha, p.limit);
      p.out[static_cast<size_t>(row0 + t0 + t) * p.n_out + f] = __float2bfloat16(a);
    }
    if (splits > 1) cluster.sync();                               // the partial tiles have been read
  }
}

template <int MODE, int NT, int LG>
inline cudaError_t qs_launch(const QsParams& p, int E, int in_use, int rows_used, cudaStream_t stream) {
  using S = QsShape<MODE, NT>;
  auto kern = qstream_kernel<MODE, NT, LG>;
  // function attributes are per device: a process that drives several GPUs sets them on each
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!configured[dev]) {
    const cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem);
    if (err != cudaSuccess) return err;
    prefer_max_shared(kern);
    configured[dev] = true;
  }
  const int feats = (p.epi >= MX_EPI_SWIGLU ? 8 : 16) * (S::kRows / 16);
  const int blocks = (p.n_out + feats - 1) / feats;
  QsParams a = p;
  // Split K over 2, 4 or 8 CTAs while all of the experts in use still fit at two CTAs an SM (clusters stay inside a GPC, which
  // leaves some SMs out: 48 clusters of 6 took twice the time of 32 clusters of 8, hence powers of two and 256, not 296), down
  // to two stages of work a CTA.
  int splits = 1;
  const int nblk = (p.K + kQsBlockK - 1) / kQsBlockK;
  while (splits < kQsMaxSplit && static_cast<long long>(blocks) * in_use * splits * 2 <= 256 && nblk / (splits * 2) >= 2) splits *= 2;
  a.k_per_cta = (nblk + splits - 1) / splits * kQsBlockK;
  splits = (p.K + a.k_per_cta - 1) / a.k_per_cta;
  a.ahead = mx_qstream_ahead(E, rows_used, static_cast<long long>(splits) * blocks * E, S::kResident * device_sm_count());
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(splits, blocks, E);
  cfg.blockDim = dim3(kQsThreads);
  cfg.dynamicSmemBytes = S::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = splits;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, a);
}

template <int MODE, int LG>
inline cudaError_t qs_dispatch(const QsParams& p, int E, int rows_used, cudaStream_t stream) {
  const int in_use = rows_used < E ? (rows_used > 0 ? rows_used : 1) : E;   // at most so many experts have rows
  const int hint = static_cast<int>(2ll * rows_used / E);   // (an expert's share varies: twice the average nearly always fits a pass)
  if (hint <= 8) return qs_launch<MODE, 1, LG>(p, E, in_use, rows_used, stream);
  if (hint <= 16) return qs_launch<MODE, 2, LG>(p, E, in_use, rows_used, stream);
  return qs_launch<MODE, 4, LG>(p, E, in_use, rows_used, stream);
}

}  // namespace mx

// Whether the first three stages are requested ahead of the dependent-launch wait, before the offsets can be read. An expert
// without rows then has 3 of its stages read for nothing (3 of 23 for rows of 2880, twice that with K split in two), so this is
// left to calls that expect rows nearly everywhere, and to those whose blocks are all on the GPU at once (`ctas` of at most
// `resident`), where the wait is what counts: 6 to 8 rows on 8 experts of 1408, 17 / 19. Top 4 of 128 mxfp4 experts of 2880, gate/up and down (us), ahead / behind:
// 1 row 62 and 46 / 39 and 26, 8 rows 115 and 69 / 97 and 56, 32 rows 250 and 134 / 246 and 131, 64 rows 333 and 176 / 333 and
// 177, 128 rows 391 and 210 / 393 and 212; 128 affine experts of 768, groups of 32, 512 rows in all: 127 and 56 / 130 and 57.
extern "C" int mx_qstream_ahead(int E, int rows_used, long long ctas, int resident) {
  return rows_used >= 2ll * E || ctas <= resident ? 1 : 0;
}

// xs [rows, K]; w [E, N, K/8] MLX-packed 4-bit (N = 2 * n_out rows, gate then up, when `epi` is a gated activation, else
// N = n_out). mode: 0 affine (bf16 scales and biases per `group`), 1 mxfp4 (e8m0 scales per 32). offsets: device [E + 1] rows
// of every expert. rows_used: how many rows are expected in all (any number is served; an expert with more than a pass holds
// has its weights read again). Returns -9 for shapes it does not cover.
extern "C" int mx_qstream(const void* xs, const void* w, const void* scales, const void* biases, const void* lin_bias, const int* offsets,
                          void* out, int E, int rows_used, int n_out, int K, int group, int mode, int epi, float alpha, float limit,
                          void* stream_) {
  using namespace mx;
  if (E <= 0 || n_out <= 0) return 0;
  if (K <= 0 || K % 32 || (group != 32 && group != 64 && group != 128) || K % group || (mode != 0 && mode != 1)) return -9;
  if (mode == 0 && biases == nullptr) return -9;
  if (mode == 1 && group != 32) return -9;
  if (E > 65535 || n_out > (1 << 21)) return -9;
  const bool gated = epi >= MX_EPI_SWIGLU;
  if (!gated && epi != MX_EPI_NONE && epi != MX_EPI_BIAS) return -9;
  // scales are fetched as aligned 32-bit words at 32-bit offsets: whole words, below 4 GB
  const unsigned long long scale_bytes = static_cast<unsigned long long>(E) * (gated ? 2 : 1) * n_out * (K / group) * (mode == 0 ? 2 : 1);
  if (scale_bytes % 4 || scale_bytes >> 32) return -9;
  if ((reinterpret_cast<uintptr_t>(xs) | reinterpret_cast<uintptr_t>(w)) & 15) return -9;
  if ((reinterpret_cast<uintptr_t>(scales) | reinterpret_cast<uintptr_t>(biases)) & 3) return -9;
  QsParams p;
  p.xs = static_cast<const __nv_bfloat16*>(xs);
  p.w = static_cast<const uint8_t*>(w);
  p.scales = static_cast<const uint8_t*>(scales);
  p.biases = static_cast<const uint8_t*>(biases);
  p.lin_bias = static_cast<const __nv_bfloat16*>(lin_bias);
  p.offsets = offsets;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.N = gated ? 2 * n_out : n_out, p.K = K, p.k_per_cta = 0;
  p.n_out = n_out, p.epi = epi, p.alpha = alpha, p.limit = limit;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (mode == 1) return static_cast<int>(qs_dispatch<1, 5>(p, E, rows_used, stream));
  if (group == 32) return static_cast<int>(qs_dispatch<0, 5>(p, E, rows_used, stream));
  if (group == 64) return static_cast<int>(qs_dispatch<0, 6>(p, E, rows_used, stream));
  return static_cast<int>(qs_dispatch<0, 7>(p, E, rows_used, stream));
}
