// BF16 GEMM  D = alpha * A . B + beta * C  on the 5th-generation tensor cores (tcgen05).
//
// Operator semantics follow Matmul / MatmulExecutor of the reference
// (crates/cleandl/src/execgraph/ops/matmul.rs:61-68, 1092-1183), which hands the problem to
// cuBLASLt; the kernel itself is written for sm_100a from scratch.  (The reference's own, disabled,
// tcgen05 kernel is crates/cleandl/rust-kernels/src/sky_matmul/tcgen05_bf16.rs.)
//
// Kernel structure (one persistent CTA per SM, 320 threads):
//   warp 0      TMA producer: loads a 128 x 64 A tile and a 256 x 64 B tile per stage into
//               128-byte-swizzled shared memory (4-stage ring, 48 KiB per stage).
//   warp 1      MMA issuer: one elected thread issues 4 tcgen05.mma (M128 N256 K16) per stage into
//               one of two 256-column f32 accumulators in TMEM; tcgen05.commit releases the stage
//               and, after the last K block, publishes the accumulator.
//   warps 2-9   epilogue: tcgen05.ld the accumulator (one row per thread, 32 columns at a time),
//               apply alpha / beta*C, convert and store straight to global memory.  The second
//               accumulator lets the epilogue of tile i overlap the main loop of tile i+1.
// Both operands may be K-major (K contiguous) or MN-major (M or N contiguous); that covers
// forward (A row-major, B row-major), dgrad (B transposed view) and wgrad (A transposed view)
// without copies.  M/N/K tails rely on TMA zero fill for loads and on predicated stores.
#include "gemm_rows.cuh"
#include "host.h"
#include "ops.h"
#include "ptx.cuh"

#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>

namespace cdl {
namespace gemm {

constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BK = 64;
constexpr int STAGES = 4;
constexpr int A_BYTES = BM * BK * 2;  // 16 KiB
constexpr int B_BYTES = BN * BK * 2;  // 32 KiB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int THREADS = 320;  // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue (two per TMEM lane quadrant)
constexpr int EPI_WARPS = 8;
constexpr int TMEM_COLS = 512;
// L2 budget for A plus one raster panel of B (see the raster_w computation on the host).
#ifndef CDL_GEMM_RASTER_BUDGET_MB
#define CDL_GEMM_RASTER_BUDGET_MB 96
#endif
constexpr size_t SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + 256;

struct Barriers {
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_word;
};

// 32 consecutive columns of one output row, all operands 32-byte aligned: C read, fused
// SwiGLU or plain conversion, 256-bit stores.
__device__ __forceinline__ void store_chunk_wide(const Params& p, float (&v)[32], int b, int row,
                                                 int col0) {
  const long long r64 = row;
  if (p.c_mode == 1) {
    const __nv_bfloat16* cp = static_cast<const __nv_bfloat16*>(p.c) + b * p.c_batch + r64 * p.ldc + col0;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      uint32_t w[8];
      ld_global_v8(cp + g * 16, w);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[g * 16 + 2 * j] += p.beta * bf16_lo(w[j]);
        v[g * 16 + 2 * j + 1] += p.beta * bf16_hi(w[j]);
      }
    }
  } else if (p.c_mode == 2) {
    const float* cp = static_cast<const float*>(p.c) + b * p.c_batch + r64 * p.ldc + col0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      uint32_t w[8];
      ld_global_v8(cp + g * 8, w);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[g * 8 + j] += p.beta * __uint_as_float(w[j]);
    }
  }
  if (p.epi_mode != 0) {
    __nv_bfloat16* dp = static_cast<__nv_bfloat16*>(p.d) + r64 * p.ldd + col0;
    __nv_bfloat16* op = p.out2 + r64 * p.ld_out2 + col0;
    const __nv_bfloat16* a0 = p.aux0 + r64 * p.ld_aux0 + col0;
    const __nv_bfloat16* a1 = p.aux1 + r64 * p.ld_aux1 + col0;  // only dereferenced in mode 2
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      uint32_t w0[8], w1[8], q1[8], q2[8];
      ld_global_v8(a0 + g * 16, w0);
      if (p.epi_mode == 2) ld_global_v8(a1 + g * 16, w1);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float o1[2], o2[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float rr = v[g * 16 + 2 * j + e];
          const float x0 = e ? bf16_hi(w0[j]) : bf16_lo(w0[j]);
          if (p.epi_mode == 1) {
            o1[e] = rr;
            o2[e] = rr * fast_sigmoid(rr) * x0;
          } else {
            const float x1 = e ? bf16_hi(w1[j]) : bf16_lo(w1[j]);
            const float sg = fast_sigmoid(x0);
            o1[e] = x0 * sg * rr;
            o2[e] = rr * x1 * (sg + x0 * sg * (1.0f - sg));
          }
        }
        q1[j] = pack_bf16x2(o1[0], o1[1]);
        q2[j] = pack_bf16x2(o2[0], o2[1]);
      }
      st_global_v8(dp + g * 16, q1);
      st_global_v8(op + g * 16, q2);
    }
  } else if (p.out_f32) {
    float* dp = static_cast<float*>(p.d) + b * p.d_batch + r64 * p.ldd + col0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      uint32_t w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = __float_as_uint(v[g * 8 + j]);
      st_global_v8(dp + g * 8, w);
    }
  } else {
    __nv_bfloat16* dp = static_cast<__nv_bfloat16*>(p.d) + b * p.d_batch + r64 * p.ldd + col0;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      uint32_t w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = pack_bf16x2(v[g * 16 + 2 * j], v[g * 16 + 2 * j + 1]);
      st_global_v8(dp + g * 16, w);
    }
  }
}

// Epilogue of one accumulator for the calling warp: thread `lane` owns output row `row`
// (TMEM lane = its lane inside the warp's quadrant); t_row addresses column 0 of the accumulator
// at the warp's first lane.  Applies alpha / beta * C, converts and stores 128 columns (the warp's half of the tile).
__device__ __forceinline__ void store_tile_rows(const Params& p, uint32_t t_row, int b, int row,
                                                int col_base) {
  const bool row_ok = row < p.M;
#pragma unroll 1
  for (int ch = 0; ch < BN / 64; ++ch) {
    const int col0 = col_base + ch * 32;
    if (col0 >= p.N) break;  // warp-uniform
    uint32_t r[32];
    tmem_ld32(t_row + ch * 32, r);
    tmem_wait_ld(r);
    if (row_ok) {
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = p.alpha * __uint_as_float(r[j]);
      if (p.wide && !p.atomic_out && col0 + 32 <= p.N) {
        // Fast path: every row involved is 32-byte aligned, so each thread moves whole 32-byte
        // sectors with 256-bit accesses (a thread owns a row, so narrower accesses would touch
        // every sector twice).
        store_chunk_wide(p, v, b, row, col0);
        continue;
      }
      if (p.c_mode == 1) {
        const __nv_bfloat16* cp = static_cast<const __nv_bfloat16*>(p.c) +
                                  b * p.c_batch + static_cast<long long>(row) * p.ldc + col0;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if (p.c_vec && col0 + g * 8 + 8 <= p.N) {
            const uint4 q = *reinterpret_cast<const uint4*>(cp + g * 8);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              v[g * 8 + 2 * j] += p.beta * bf16_lo(w[j]);
              v[g * 8 + 2 * j + 1] += p.beta * bf16_hi(w[j]);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (col0 + g * 8 + j < p.N)
                v[g * 8 + j] += p.beta * __bfloat162float(cp[g * 8 + j]);
          }
        }
      } else if (p.c_mode == 2) {
        const float* cp = static_cast<const float*>(p.c) + b * p.c_batch +
                          static_cast<long long>(row) * p.ldc + col0;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          if (p.c_vec && col0 + g * 4 + 4 <= p.N) {
            const float4 q = *reinterpret_cast<const float4*>(cp + g * 4);
            v[g * 4 + 0] += p.beta * q.x;
            v[g * 4 + 1] += p.beta * q.y;
            v[g * 4 + 2] += p.beta * q.z;
            v[g * 4 + 3] += p.beta * q.w;
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (col0 + g * 4 + j < p.N) v[g * 4 + j] += p.beta * cp[g * 4 + j];
          }
        }
      }
      if (p.epi_mode != 0) {
        // sigmoid via ex2 / rcp approximations, as in the reference's fused epilogues
        // (crates/cleandl/rust-kernels/src/sky_matmul/tcgen05_bf16.rs:851-877).
        __nv_bfloat16* dp = static_cast<__nv_bfloat16*>(p.d) + static_cast<long long>(row) * p.ldd + col0;
        __nv_bfloat16* op = p.out2 + static_cast<long long>(row) * p.ld_out2 + col0;
        const __nv_bfloat16* a0 = p.aux0 + static_cast<long long>(row) * p.ld_aux0 + col0;
        const __nv_bfloat16* a1 = p.epi_mode == 2 ? p.aux1 + static_cast<long long>(row) * p.ld_aux1 + col0 : nullptr;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if (col0 + g * 8 + 8 <= p.N) {  // N % 8 == 0 is checked on the host
            const uint4 q0 = *reinterpret_cast<const uint4*>(a0 + g * 8);
            const uint32_t w0[4] = {q0.x, q0.y, q0.z, q0.w};
            uint32_t w1[4] = {0, 0, 0, 0};
            if (p.epi_mode == 2) {
              const uint4 q1 = *reinterpret_cast<const uint4*>(a1 + g * 8);
              w1[0] = q1.x; w1[1] = q1.y; w1[2] = q1.z; w1[3] = q1.w;
            }
            float o1[8], o2[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float r = v[g * 8 + j];
              const float x0 = (j & 1) ? bf16_hi(w0[j >> 1]) : bf16_lo(w0[j >> 1]);
              if (p.epi_mode == 1) {
                const float sg = fast_sigmoid(r);
                o1[j] = r;
                o2[j] = r * sg * x0;
              } else {
                const float x1 = (j & 1) ? bf16_hi(w1[j >> 1]) : bf16_lo(w1[j >> 1]);
                const float sg = fast_sigmoid(x0);
                o1[j] = x0 * sg * r;
                o2[j] = r * x1 * (sg + x0 * sg * (1.0f - sg));
              }
            }
            uint4 qa, qb;
            qa.x = pack_bf16x2(o1[0], o1[1]); qa.y = pack_bf16x2(o1[2], o1[3]);
            qa.z = pack_bf16x2(o1[4], o1[5]); qa.w = pack_bf16x2(o1[6], o1[7]);
            qb.x = pack_bf16x2(o2[0], o2[1]); qb.y = pack_bf16x2(o2[2], o2[3]);
            qb.z = pack_bf16x2(o2[4], o2[5]); qb.w = pack_bf16x2(o2[6], o2[7]);
            *reinterpret_cast<uint4*>(dp + g * 8) = qa;
            *reinterpret_cast<uint4*>(op + g * 8) = qb;
          }
        }
      } else if (p.atomic_out) {
        // K-sliced accumulation: D (f32, already holding C) += alpha * partial.  Several slices
        // of a tile add concurrently, so the order of the f32 additions is not fixed.
        float* dp = static_cast<float*>(p.d) + b * p.d_batch +
                    static_cast<long long>(row) * p.ldd + col0;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          if (p.d_vec && col0 + g * 4 + 4 <= p.N) {
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dp + g * 4),
                         "f"(v[g * 4]), "f"(v[g * 4 + 1]), "f"(v[g * 4 + 2]), "f"(v[g * 4 + 3])
                         : "memory");
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (col0 + g * 4 + j < p.N) atomicAdd(dp + g * 4 + j, v[g * 4 + j]);
          }
        }
      } else if (p.out_f32) {
        float* dp = static_cast<float*>(p.d) + b * p.d_batch +
                    static_cast<long long>(row) * p.ldd + col0;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          if (p.d_vec && col0 + g * 4 + 4 <= p.N) {
            *reinterpret_cast<float4*>(dp + g * 4) =
                make_float4(v[g * 4], v[g * 4 + 1], v[g * 4 + 2], v[g * 4 + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (col0 + g * 4 + j < p.N) dp[g * 4 + j] = v[g * 4 + j];
          }
        }
      } else {
        __nv_bfloat16* dp = static_cast<__nv_bfloat16*>(p.d) + b * p.d_batch +
                            static_cast<long long>(row) * p.ldd + col0;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if (p.d_vec && col0 + g * 8 + 8 <= p.N) {
            uint4 q;
            q.x = pack_bf16x2(v[g * 8 + 0], v[g * 8 + 1]);
            q.y = pack_bf16x2(v[g * 8 + 2], v[g * 8 + 3]);
            q.z = pack_bf16x2(v[g * 8 + 4], v[g * 8 + 5]);
            q.w = pack_bf16x2(v[g * 8 + 6], v[g * 8 + 7]);
            *reinterpret_cast<uint4*>(dp + g * 8) = q;
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (col0 + g * 8 + j < p.N) dp[g * 8 + j] = __float2bfloat16_rn(v[g * 8 + j]);
          }
        }
      }
    }
  }
}

// Epilogue of mode 3 for the calling warp: its 128 columns are one head.  The rotation pairs column
// i with column i + 64, so the 32-column chunks are drained in pairs (0, 2) and (1, 3); heads at or
// beyond rope_cols (the value heads of a fused qkv projection) are stored unrotated.
__device__ __forceinline__ void store_tile_rows_rope(const Params& p, uint32_t t_row, int row,
                                                     int col_base) {
  if (col_base >= p.N) return;  // warp-uniform
  const bool row_ok = row < p.M;
  const bool rotate = col_base < p.rope_cols;  // warp-uniform
  int pos = 0;
  if (row_ok && rotate) {
    if (p.rope_cu != nullptr) {
      // ragged batch: the position restarts at every sequence; rows after the last sequence keep
      // position 0 (they are padding)
      int lo_i = 0, hi_i = p.rope_nseq;  // largest b with cu[b] <= row
      while (hi_i - lo_i > 1) {
        const int mid = (lo_i + hi_i) >> 1;
        if (p.rope_cu[mid] <= row) lo_i = mid;
        else hi_i = mid;
      }
      pos = row < p.rope_cu[p.rope_nseq] ? min(row - p.rope_cu[lo_i], p.rope_seqlen - 1) : 0;
    } else {
      pos = row % p.rope_seqlen;
    }
  }
  const float* cs = p.rope_table + static_cast<long long>(pos) * 128;
  __nv_bfloat16* dp = static_cast<__nv_bfloat16*>(p.d) + static_cast<long long>(row) * p.ldd + col_base;
#pragma unroll 1
  for (int pr = 0; pr < 2; ++pr) {
    uint32_t lo[32], hi[32];
    tmem_ld32(t_row + pr * 32, lo);
    tmem_ld32(t_row + (pr + 2) * 32, hi);
    tmem_wait_ld(lo, hi);
    if (!row_ok) continue;
    uint32_t olo[16], ohi[16];
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      float c[4] = {1.f, 1.f, 1.f, 1.f}, sn[4] = {0.f, 0.f, 0.f, 0.f};
      if (rotate) {
        const float4 cv = __ldg(reinterpret_cast<const float4*>(cs + pr * 32 + g * 4));
        const float4 sv = __ldg(reinterpret_cast<const float4*>(cs + 64 + pr * 32 + g * 4));
        c[0] = cv.x; c[1] = cv.y; c[2] = cv.z; c[3] = cv.w;
        sn[0] = sv.x; sn[1] = sv.y; sn[2] = sv.z; sn[3] = sv.w;
      }
      float rl[4], rh[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float l = p.alpha * __uint_as_float(lo[g * 4 + e]), h = p.alpha * __uint_as_float(hi[g * 4 + e]);
        rl[e] = l * c[e] - h * sn[e];
        rh[e] = h * c[e] + l * sn[e];
      }
      olo[g * 2] = pack_bf16x2(rl[0], rl[1]);
      olo[g * 2 + 1] = pack_bf16x2(rl[2], rl[3]);
      ohi[g * 2] = pack_bf16x2(rh[0], rh[1]);
      ohi[g * 2 + 1] = pack_bf16x2(rh[2], rh[3]);
    }
    if (p.wide) {  // whole 32-byte sectors per access, as in store_chunk_wide
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const uint32_t wl[8] = {olo[g * 8], olo[g * 8 + 1], olo[g * 8 + 2], olo[g * 8 + 3],
                                olo[g * 8 + 4], olo[g * 8 + 5], olo[g * 8 + 6], olo[g * 8 + 7]};
        const uint32_t wh[8] = {ohi[g * 8], ohi[g * 8 + 1], ohi[g * 8 + 2], ohi[g * 8 + 3],
                                ohi[g * 8 + 4], ohi[g * 8 + 5], ohi[g * 8 + 6], ohi[g * 8 + 7]};
        st_global_v8(dp + pr * 32 + g * 16, wl);
        st_global_v8(dp + (pr + 2) * 32 + g * 16, wh);
      }
    } else {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        *reinterpret_cast<uint4*>(dp + pr * 32 + g * 8) =
            make_uint4(olo[g * 4], olo[g * 4 + 1], olo[g * 4 + 2], olo[g * 4 + 3]);
        *reinterpret_cast<uint4*>(dp + (pr + 2) * 32 + g * 8) =
            make_uint4(ohi[g * 4], ohi[g * 4 + 1], ohi[g * 4 + 2], ohi[g * 4 + 3]);
      }
    }
  }
}

// The operands of the fused SwiGLU forms come ahead of their use: a warp's next 32 rows x 32 columns of aux0 (and aux1)
// by TMA into its 4 KiB buffer (the 64-byte swizzle: a row is 64 bytes, its 16-byte chunk c at c ^ (row / 2 & 3)), the
// first ones of a tile under its products, the others under the arithmetic and the stores of those before.
struct SwigluFeed {
  const CUtensorMap* map0;
  const CUtensorMap* map1;
  uint8_t* buf;
  uint64_t* full;
  bool two;
  uint32_t phase;
  __device__ __forceinline__ void load(int lane, int row0, int col0) {
    if (lane != 0) return;
    mbar_arrive_expect_tx(full, two ? 4096 : 2048);
    tma_load_3d(buf, map0, full, col0, row0, 0);
    if (two) tma_load_3d(buf + 2048, map1, full, col0, row0, 0);
  }
  __device__ __forceinline__ void read(int lane, int which, uint32_t (&w)[16]) const {
    const uint32_t row = smem_u32(buf) + which * 2048 + lane * 64, x = (lane >> 1 & 3) << 4;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(w[4 * c]), "=r"(w[4 * c + 1]), "=r"(w[4 * c + 2]), "=r"(w[4 * c + 3])
                   : "r"(row + ((c << 4) ^ x))
                   : "memory");
  }
};

// Pairs of f32 in one register pair: one packed operation for two.
struct F32x2 {
  uint64_t v;
  __device__ __forceinline__ F32x2() {}
  __device__ __forceinline__ F32x2(float lo, float hi) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi)); }
  __device__ __forceinline__ void get(float& lo, float& hi) const { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
};
__device__ __forceinline__ F32x2 mul2(F32x2 a, F32x2 b) {
  F32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ F32x2 fma2(F32x2 a, F32x2 b, F32x2 c) {
  F32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return d;
}
__device__ __forceinline__ F32x2 tanh2(F32x2 a) {
  float lo, hi;
  a.get(lo, hi);
  asm("tanh.approx.f32 %0, %0;" : "+f"(lo));
  asm("tanh.approx.f32 %0, %0;" : "+f"(hi));
  return F32x2(lo, hi);
}
__device__ __forceinline__ uint32_t pack2(F32x2 a) {
  float lo, hi;
  a.get(lo, hi);
  return pack_bf16x2(lo, hi);
}

// The fused SwiGLU epilogues for the calling warp: 32 rows, 128 columns; the first chunk's operands are under way.
// TWO: mode 2 (d_up, d_gate), else mode 1 (gate, act).  alpha is 1.  Eight warps do this beside the products, so their
// instructions count: packed pairs take half of what single operations take.
template <bool TWO>
__device__ __forceinline__ void store_tile_rows_swiglu(const Params& p, SwigluFeed& feed, uint32_t t_row, int row,
                                                       int col_base, int lane, volatile int* abort_word) {
  if (row - lane >= p.M) return;  // warp-uniform
#pragma unroll 1
  for (int ch = 0; ch < BN / 64; ++ch) {
    const int col0 = col_base + ch * 32;
    if (col0 >= p.N) break;
    uint32_t r[32], w0[16], w1[16];
    if (!mbar_wait(feed.full, feed.phase, abort_word, 313)) return;
    feed.phase ^= 1;
    feed.read(lane, 0, w0);
    if (TWO) feed.read(lane, 1, w1);
    tmem_ld32(t_row + ch * 32, r);
    tmem_wait_ld(r);
    __syncwarp();  // the buffer has been read
    if (ch + 1 < BN / 64 && col0 + 32 < p.N) feed.load(lane, row - lane, col0 + 32);
    uint32_t q1[16], q2[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const F32x2 rr(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
      const F32x2 x0(bf16_lo(w0[j]), bf16_hi(w0[j])), half(0.5f, 0.5f);
      const F32x2 s = fma2(tanh2(mul2(TWO ? x0 : rr, half)), half, half);  // the sigmoid, as fast_sigmoid
      if (!TWO) {
        q1[j] = pack2(rr);
        q2[j] = pack2(mul2(mul2(rr, s), x0));
      } else {
        const F32x2 x1(bf16_lo(w1[j]), bf16_hi(w1[j])), one(1.0f, 1.0f), minus(-1.0f, -1.0f);
        const F32x2 xs = mul2(x0, s);
        q1[j] = pack2(mul2(xs, rr));
        q2[j] = pack2(mul2(mul2(rr, x1), fma2(xs, fma2(s, minus, one), s)));
      }
    }
    if (row < p.M) {
      __nv_bfloat16* dp = static_cast<__nv_bfloat16*>(p.d) + static_cast<long long>(row) * p.ldd + col0;
      __nv_bfloat16* op = p.out2 + static_cast<long long>(row) * p.ld_out2 + col0;
      if (p.wide && col0 + 32 <= p.N) {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          st_global_v8(dp + g * 16, reinterpret_cast<const uint32_t(&)[8]>(q1[g * 8]));
          st_global_v8(op + g * 16, reinterpret_cast<const uint32_t(&)[8]>(q2[g * 8]));
        }
      } else {
#pragma unroll
        for (int g = 0; g < 4; ++g)
          if (col0 + g * 8 + 8 <= p.N) {  // N % 8 == 0 is checked on the host
            *reinterpret_cast<uint4*>(dp + g * 8) = make_uint4(q1[g * 4], q1[g * 4 + 1], q1[g * 4 + 2], q1[g * 4 + 3]);
            *reinterpret_cast<uint4*>(op + g * 8) = make_uint4(q2[g * 4], q2[g * 4 + 1], q2[g * 4 + 2], q2[g * 4 + 3]);
          }
      }
    }
    __syncwarp();  // all lanes are at the next chunk's tensor-memory load together
  }
}

// The epilogue of D += alpha * accumulator for the calling warp: rows row0 .. row0 + 31, 128 columns.
__device__ __forceinline__ void add_tile_rows(const Params& p, const CUtensorMap* tm_d, uint8_t* buf, uint32_t t_row,
                                              int b, int row0, int col_base, int lane) {
  if (row0 >= p.M) return;  // warp-uniform; rows past M inside the box are clipped
#pragma unroll 1
  for (int ch = 0; ch < BN / 64; ++ch) {
    const int col0 = col_base + ch * 32;
    if (col0 >= p.N) break;
    uint32_t r[32];
    tmem_ld32(t_row + ch * 32, r);
    tmem_wait_ld(r);
    if (lane == 0) tma_store_wait_read<0>();  // the buffer's last reduction has read it
    __syncwarp();
    add_chunk(tm_d, buf, r, p.alpha, lane, col0, row0, b);
  }
}

__global__ void __launch_bounds__(THREADS, 1)
    gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmap_a,
                     const __grid_constant__ CUtensorMap tmap_b, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  Barriers* bars = reinterpret_cast<Barriers*>(smem + STAGES * STAGE_BYTES);
  volatile int* abort_word = &bars->abort_word;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->acc_full[i], 1);
      mbar_init(&bars->acc_empty[i], EPI_WARPS);
    }
    bars->abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  // Everything above overlaps the tail of the previous kernel of the stream; operands are read
  // (and outputs written) only from here on.
  grid_dep_wait();
  grid_dep_launch();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.num_tiles && ok; tile += gridDim.x) {
        int b, tm, tn;
        tile_coords(p, tile, b, tm, tn);
        const int m0 = tm * BM, n0 = tn * BN;
        for (int kb = 0; kb < p.k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&bars->empty[s], ph ^ 1, abort_word, 101)) {
            ok = false;
            break;
          }
          uint8_t* sa = smem + s * STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          mbar_arrive_expect_tx(&bars->full[s], STAGE_BYTES);
          const int k0 = kb * BK;
          if (p.a_mn) {
#pragma unroll
            for (int i = 0; i < BM / 64; ++i)
              tma_load_3d(sa + i * 8192, &tmap_a, &bars->full[s], m0 + i * 64, k0, b);
          } else {
            tma_load_3d(sa, &tmap_a, &bars->full[s], k0, m0, b);
          }
          if (p.b_mn) {
#pragma unroll
            for (int i = 0; i < BN / 64; ++i)
              tma_load_3d(sb + i * 8192, &tmap_b, &bars->full[s], n0 + i * 64, k0, b);
          } else {
            tma_load_3d(sb, &tmap_b, &bars->full[s], k0, n0, b);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(BM, BN, p.a_mn, p.b_mn);
      const uint32_t a_lbo = p.a_mn ? 8192u : 16u, b_lbo = p.b_mn ? 8192u : 16u;
      const uint32_t a_kstep = p.a_mn ? 2048u : 32u, b_kstep = p.b_mn ? 2048u : 32u;
      uint32_t it = 0;
      int t = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.num_tiles && ok; tile += gridDim.x, ++t) {
        const int acc = t & 1;
        const uint32_t acc_ph = (t >> 1) & 1;
        if (!mbar_wait(&bars->acc_empty[acc], acc_ph ^ 1, abort_word, 201)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < p.k_blocks; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&bars->full[s], ph, abort_word, 202)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t da = smem_desc_sw128(sa + k * a_kstep, a_lbo, 1024);
            const uint64_t db = smem_desc_sw128(sb + k * b_kstep, b_lbo, 1024);
            umma_ss(d_tmem, da, db, idesc, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit(&bars->empty[s]);
        }
        if (ok) umma_commit(&bars->acc_full[acc]);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9)
    const int quad = warp & 3;  // TMEM lane quadrant this warp may read
    const int half = (warp - 2) >> 2;  // which 128 of the tile's 256 columns
    int t = 0;
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, ++t) {
      int b, tm, tn;
      tile_coords(p, tile, b, tm, tn);
      const int acc = t & 1;
      const uint32_t acc_ph = (t >> 1) & 1;
      if (!mbar_wait(&bars->acc_full[acc], acc_ph, abort_word, 301)) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * BN + half * (BN / 2);
      if (p.epi_mode == 3) store_tile_rows_rope(p, t_row, tm * BM + quad * 32 + lane, tn * BN + half * (BN / 2));
      else store_tile_rows(p, t_row, b, tm * BM + quad * 32 + lane, tn * BN + half * (BN / 2));
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_empty[acc]);
    }
  }

  // ------------------------------------------------------------ tear-down
  __syncwarp();
  if (*abort_word != 0) {
    // Give loads that may still be in flight time to land before shared memory is released.
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (threadIdx.x == 0 && *abort_word != 0) atomicExch(p.status, *abort_word);
}

// ------------------------------------------------------------------------------------------
// CTA-pair variant: a cluster of two CTAs computes a 256 x 256 tile with tcgen05.mma.cta_group::2.
// Each CTA loads its own 128 rows of A and its own 128-column half of B (32 KiB per stage, so the
// ring is 6 deep), which halves the B traffic per SM; the pair's leader (cluster rank 0) issues
// every MMA for both CTAs and each CTA drains its own 128 accumulator rows from its own TMEM.
// Cross-CTA signalling: the peer's TMA loads complete on the leader's `full` barrier
// (cta_group::2 form of the load, barrier given as a cluster address); the leader releases
// stages and publishes accumulators with one tcgen05.commit per CTA (local and peer address); the
// peer's epilogue warps arrive on the leader's `acc_empty` barrier with a remote mbarrier.arrive.
constexpr int PAIR_STAGES = 6;
constexpr int PAIR_STAGE_BYTES = 2 * A_BYTES;  // A 128 x 64 and half of B 128 x 64
constexpr int PAIR_M = 2 * BM;
constexpr int PAIR_BARRIER_BYTES = 512;
// One kernel per kind of store.  All of them in one, with the buffers that the plain ones do not need (they take room
// from the L1, through which C is read), cost those 0.2 to 0.9 us (2048 x 5632 x
// 256 12.3 instead of 11.9, with a bf16 C 18.8 instead of 18.0).
enum PairStore { STORE, STORE_ADD, STORE_SWIGLU };  // D in any form, D += by TMA, the SwiGLU forms whose operands TMA brings
constexpr int pair_staging(int kind) { return kind == STORE ? 0 : EPI_WARPS * CHUNK_BYTES; }  // a buffer per epilogue warp
constexpr size_t pair_smem_bytes(int kind) {
  return 1024 + PAIR_STAGES * PAIR_STAGE_BYTES + pair_staging(kind) + PAIR_BARRIER_BYTES;
}

// Work units are handed out at run time: a cluster's first unit is its index, every further one
// comes from a global counter, so a cluster that finds its SMs late (another kernel, e.g. a
// collective, holds them) takes less work instead of holding its fixed share back to the end.
// The leader's producer thread draws the unit for step t and publishes it in slot t % SCHED_SLOTS
// of both CTAs' rings: locally with a store and an arrival on sched_full, in the peer with one
// st.async that carries the value and completes the peer's sched_full (armed by the peer's
// producer thread with expect-tx).  No role can be SCHED_SLOTS units ahead of another (6 stages of
// operands and 2 accumulators bound the distance), so slots are reused without a release barrier.
constexpr int SCHED_SLOTS = 16;
constexpr uint32_t SCHED_DONE = 0xffffffffu;
struct PairBarriers {
  uint64_t full[PAIR_STAGES];
  uint64_t empty[PAIR_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t sched_full[SCHED_SLOTS];
  uint64_t extra_full[EPI_WARPS];  // the SwiGLU epilogue's operands, a warp's next chunk
  uint32_t unit_ring[SCHED_SLOTS];
  uint32_t tmem_base;
  int abort_word;
};
static_assert(sizeof(PairBarriers) <= PAIR_BARRIER_BYTES, "barriers fit behind the staging buffers");

template <int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
    gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmap_a,
                          const __grid_constant__ CUtensorMap tmap_b,
                          const __grid_constant__ CUtensorMap tmap_e0,
                          const __grid_constant__ CUtensorMap tmap_e1, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* staging = smem + PAIR_STAGES * PAIR_STAGE_BYTES;
  PairBarriers* bars = reinterpret_cast<PairBarriers*>(staging + pair_staging(KIND));
  volatile int* abort_word = &bars->abort_word;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int cluster_id = blockIdx.x >> 1;
  const int num_clusters = gridDim.x >> 1;
  // Work unit = (tile, K slice); slices exist only in the accumulate-in-place form.
  const int num_units = p.num_tiles * p.split_k;
  // Unit numbering with K slices: tiles are taken in chunks of one wave (as many tiles as the
  // grid has clusters); within a chunk all tiles of K slice 0 come first, then all of slice 1, ...
  // The clusters that run at the same time then work on neighbouring tiles of ONE slice and share
  // its A and B panels through L2, and the chunk's slices follow each other while the chunk's
  // part of D (19 MB at 74 tiles) is still in L2.  Weight gradient 2048 x 5632 x 16384 (251 MB of
  // operands, 46 MB of f32 output read and written): numbered tile by tile (a wave = three slices
  // of ~25 tiles, which share nothing) 693 MB read + 42 MB written; slice by slice over all tiles
  // 525 + 75 MB (every slice pass brings all of D back).
  auto unit_range = [&](int unit, int& tile, int& kb0, int& kb1) {
    int slice;
    if (p.split_k == 1) {
      tile = unit;
      slice = 0;
    } else {
      const int per_chunk = num_clusters * p.split_k;
      const int chunk = unit / per_chunk;
      const int r = unit - chunk * per_chunk;
      const int first = chunk * num_clusters;
      const int in_chunk = p.num_tiles - first < num_clusters ? p.num_tiles - first : num_clusters;
      slice = r / in_chunk;
      tile = first + (r - slice * in_chunk);
    }
    kb0 = static_cast<int>(static_cast<long long>(slice) * p.k_blocks / p.split_k);
    kb1 = static_cast<int>(static_cast<long long>(slice + 1) * p.k_blocks / p.split_k);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < PAIR_STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->acc_full[i], 1);
      mbar_init(&bars->acc_empty[i], 2 * EPI_WARPS);  // epilogue warps of both CTAs (leader's copy is used)
    }
    for (int i = 0; i < SCHED_SLOTS; ++i) mbar_init(&bars->sched_full[i], 1);
    for (int i = 0; i < EPI_WARPS; ++i) mbar_init(&bars->extra_full[i], 1);
    bars->abort_word = 0;
    fence_mbar_init();
    // the peer's slots wait for the leader's 4-byte st.async
    if (rank != 0)
      for (int i = 0; i < SCHED_SLOTS; ++i) mbar_arrive_expect_tx(&bars->sched_full[i], 4);
  }
  if (warp == 1) {
    tmem_alloc_pair(&bars->tmem_base, TMEM_COLS);
    tmem_relinquish_pair();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anything signals across the pair
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  if (!p.early) grid_dep_wait();  // set-up above overlaps the previous kernel's tail; global memory from here on
  grid_dep_launch();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      // The leader's producer also hands out the units (see PairBarriers).  Every cluster with a
      // valid first unit draws from the counter after each unit it takes, until a draw runs past
      // the last unit; the launch's last draw puts the counter back to zero.
      const int fetchers = num_clusters < num_units ? num_clusters : num_units;
      const unsigned total_draws = static_cast<unsigned>((num_units > num_clusters ? num_units - num_clusters : 0) + fetchers);
      uint32_t unit_u = cluster_id < num_units ? static_cast<uint32_t>(cluster_id) : SCHED_DONE;
      unsigned drawn = 0;  // the draw for the next step, under way while this step's tiles load
      for (int t = 0; ok; ++t) {
        const int slot = t % SCHED_SLOTS;
        if (rank == 0) {
          if (t > 0) {
            if (p.sched_counter != nullptr) {
              unit_u = static_cast<unsigned>(num_clusters) + drawn < static_cast<unsigned>(num_units)
                           ? static_cast<uint32_t>(num_clusters) + drawn
                           : SCHED_DONE;
              if (drawn + 1 == total_draws) atomicExch(p.sched_counter, 0u);
            } else {  // fixed round-robin assignment
              const long long u = static_cast<long long>(cluster_id) + static_cast<long long>(t) * num_clusters;
              unit_u = u < num_units ? static_cast<uint32_t>(u) : SCHED_DONE;
            }
          }
          bars->unit_ring[slot] = unit_u;
          mbar_arrive(&bars->sched_full[slot]);
          st_async_u32(mapa_shared(smem_u32(&bars->unit_ring[slot]), 1), unit_u,
                       mapa_shared(smem_u32(&bars->sched_full[slot]), 1));
          if (unit_u != SCHED_DONE && p.sched_counter != nullptr) drawn = atomicAdd(p.sched_counter, 1u);
        } else {
          if (!mbar_wait(&bars->sched_full[slot], (t / SCHED_SLOTS) & 1, abort_word, 112)) break;
          unit_u = bars->unit_ring[slot];
          mbar_arrive_expect_tx(&bars->sched_full[slot], 4);  // armed again for step t + SCHED_SLOTS
        }
        if (unit_u == SCHED_DONE) break;
        const int unit = static_cast<int>(unit_u);
        int tile, kb0, kb1, b, tm, tn;
        unit_range(unit, tile, kb0, kb1);
        tile_coords(p, tile, b, tm, tn);
        const int m0 = tm * PAIR_M + static_cast<int>(rank) * BM;
        const int n0 = tn * BN + static_cast<int>(rank) * (BN / 2);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % PAIR_STAGES;
          const uint32_t ph = (it / PAIR_STAGES) & 1;
          if (!mbar_wait(&bars->empty[s], ph ^ 1, abort_word, 111)) {
            ok = false;
            break;
          }
          uint8_t* sa = smem + s * PAIR_STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          // Bytes of both CTAs land on the leader's barrier.
          if (rank == 0) mbar_arrive_expect_tx(&bars->full[s], 2 * PAIR_STAGE_BYTES);
          const uint32_t full_leader = mapa_shared(smem_u32(&bars->full[s]), 0);
          const int k0 = kb * BK;
          if (p.a_mn) {
#pragma unroll
            for (int i = 0; i < BM / 64; ++i)
              tma_load_3d_pair(sa + i * 8192, &tmap_a, full_leader, m0 + i * 64, k0, b);
          } else {
            tma_load_3d_pair(sa, &tmap_a, full_leader, k0, m0, b);
          }
          if (p.b_mn) {
#pragma unroll
            for (int i = 0; i < BN / 128; ++i)
              tma_load_3d_pair(sb + i * 8192, &tmap_b, full_leader, n0 + i * 64, k0, b);
          } else {
            tma_load_3d_pair(sb, &tmap_b, full_leader, k0, n0, b);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = make_idesc_bf16(PAIR_M, BN, p.a_mn, p.b_mn);
      const uint32_t a_lbo = p.a_mn ? 8192u : 16u, b_lbo = p.b_mn ? 8192u : 16u;
      const uint32_t a_kstep = p.a_mn ? 2048u : 32u, b_kstep = p.b_mn ? 2048u : 32u;
      uint32_t it = 0;
      int t = 0;
      bool ok = true;
      for (; ok; ++t) {
        const int slot = t % SCHED_SLOTS;
        if (!mbar_wait(&bars->sched_full[slot], (t / SCHED_SLOTS) & 1, abort_word, 213)) break;
        const uint32_t unit_u = bars->unit_ring[slot];
        if (unit_u == SCHED_DONE) break;
        const int unit = static_cast<int>(unit_u);
        int tile, kb0, kb1;
        unit_range(unit, tile, kb0, kb1);
        const int acc = t & 1;
        const uint32_t acc_ph = (t >> 1) & 1;
        if (!mbar_wait(&bars->acc_empty[acc], acc_ph ^ 1, abort_word, 211)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % PAIR_STAGES;
          const uint32_t ph = (it / PAIR_STAGES) & 1;
          if (!mbar_wait(&bars->full[s], ph, abort_word, 212)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s * PAIR_STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t da = smem_desc_sw128(sa + k * a_kstep, a_lbo, 1024);
            const uint64_t db = smem_desc_sw128(sb + k * b_kstep, b_lbo, 1024);
            umma_ss_pair(d_tmem, da, db, idesc, (kb != kb0 || k != 0) ? 1u : 0u);
          }
          const uint32_t e = smem_u32(&bars->empty[s]);
          umma_commit_pair(e);                  // own producer
          umma_commit_pair(mapa_shared(e, 1));  // the peer's producer
        }
        if (ok) {
          const uint32_t f = smem_u32(&bars->acc_full[acc]);
          umma_commit_pair(f);
          umma_commit_pair(mapa_shared(f, 1));
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..9, both CTAs)
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    uint8_t* buf = staging + (warp - 2) * CHUNK_BYTES;
    SwigluFeed feed{&tmap_e0, &tmap_e1, buf, &bars->extra_full[warp - 2], p.epi_mode == 2, 0};
    if (p.early == 2) grid_dep_wait();
    int t = 0;
    for (;; ++t) {
      const int slot = t % SCHED_SLOTS;
      if (!mbar_wait(&bars->sched_full[slot], (t / SCHED_SLOTS) & 1, abort_word, 312)) break;
      const uint32_t unit_u = bars->unit_ring[slot];
      if (unit_u == SCHED_DONE) break;
      const int unit = static_cast<int>(unit_u);
      int tile, kb0, kb1, b, tm, tn;
      unit_range(unit, tile, kb0, kb1);
      tile_coords(p, tile, b, tm, tn);
      const int acc = t & 1;
      const uint32_t acc_ph = (t >> 1) & 1;
      const int row = tm * PAIR_M + static_cast<int>(rank) * BM + quad * 32 + lane;
      const int col = tn * BN + half * (BN / 2);
      if (KIND == STORE_SWIGLU && row - lane < p.M && col < p.N) feed.load(lane, row - lane, col);  // under the products
      if (!mbar_wait(&bars->acc_full[acc], acc_ph, abort_word, 311)) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * BN + half * (BN / 2);
      if constexpr (KIND == STORE_ADD) {
        add_tile_rows(p, &tmap_e0, buf, t_row, b, row - lane, col, lane);
      } else if constexpr (KIND == STORE_SWIGLU) {
        if (p.epi_mode == 1) store_tile_rows_swiglu<false>(p, feed, t_row, row, col, lane, abort_word);
        else store_tile_rows_swiglu<true>(p, feed, t_row, row, col, lane, abort_word);
      } else {
        if (p.epi_mode == 3) store_tile_rows_rope(p, t_row, row, col);
        else store_tile_rows(p, t_row, b, row, col);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&bars->acc_empty[acc]), 0));
    }
    if (KIND == STORE_ADD && lane == 0) tma_store_wait<0>();
  }

  // ------------------------------------------------------------ tear-down
  __syncwarp();
  if (*abort_word != 0) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer may still signal into this CTA's shared memory until here
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
  if (threadIdx.x == 0 && *abort_word != 0) atomicExch(p.status, *abort_word);
  if (p.early) grid_dep_wait();
}

// Splits a [rows, cols] (or batched) bf16 view into major-ness and leading dimension.
struct OperandLayout {
  int mn_major;     // 1 when the non-contraction dimension is the contiguous one
  long long ld;     // stride of the other dimension, elements
  long long batch;  // batch stride, elements
};

static int32_t analyze_operand(const char* name, const cdl_tensor* t, bool contraction_is_last,
                               OperandLayout* out) {
  const int r = t->rank;
  const long long rows = t->shape[r - 2], cols = t->shape[r - 1];
  const long long s_row = t->stride[r - 2], s_col = t->stride[r - 1];
  const bool aligned_base = (reinterpret_cast<uintptr_t>(t->ptr) & 15) == 0;
  out->batch = r == 3 ? t->stride[0] : 0;
  const bool batch_ok = r != 3 || t->shape[0] <= 1 || (out->batch % 8 == 0 && out->batch > 0);
  // A dimension of extent 1 has no meaningful stride, so either reading may apply; take the
  // first one whose leading dimension TMA can describe.
  const bool last_contig = s_col == 1 || cols == 1;
  const bool first_contig = s_row == 1 || rows == 1;
  if (!last_contig && !first_contig)
    return fail(CDL_ERR_INVALID,
                "matmul operand %s must have a contiguous dimension (strides [%lld, %lld])", name,
                s_row, s_col);
  auto round8 = [](long long v) { return (v + 7) / 8 * 8; };
  const long long ld_last = rows == 1 ? round8(cols) : s_row;   // rows are ld_last apart
  const long long ld_first = cols == 1 ? round8(rows) : s_col;  // columns are ld_first apart
  const bool last_ok = last_contig && ld_last % 8 == 0 && ld_last >= cols;
  const bool first_ok = first_contig && ld_first % 8 == 0 && ld_first >= rows;
  if (!aligned_base || !batch_ok || (!last_ok && !first_ok))
    return fail(CDL_ERR_UNSUPPORTED,
                "matmul operand %s: TMA needs a 16-byte aligned base, leading dimension and batch "
                "stride (ptr %p, strides [%lld, %lld] elements, batch stride %lld)",
                name, t->ptr, s_row, s_col, out->batch);
  const bool use_last = last_ok;
  out->ld = use_last ? ld_last : ld_first;
  // contraction_is_last: the operand is A [M, K]; otherwise it is B [K, N].
  const bool k_contig = contraction_is_last ? use_last : !use_last;
  out->mn_major = k_contig ? 0 : 1;
  return CDL_OK;
}

// K slices (1, 2, 4 or 8) of the cluster kernel (gemm_cluster.cu) for a problem, or 0: the 256 x 256
// tiles of the pair kernel (128 x 256 up to 128 rows).  Both times are estimated, in microseconds, and
// the cluster kernel taken where it saves 5 %.
//   wide tiles: launch and set-up; 0.28 us per K block (a quarter more when every pair loads); a store
//     that grows with the part of the tile that exists, four times as dear where an f32 C is added to, and
//     dearer for columns beyond the last 32 and with a bf16 C; and, for a pair's further tiles, the longer of
//     their products and the store.  Where TMA adds into D the store is short, and the time of the additions at
//     the memory (0.39 us per MB of D) joins as a 2.5-norm (fitted to 160 shapes: 0.6 % from the best on average).
//   cluster: launch, exchange and store (more for more slices, less for fewer rows) and the longest of
//     one CTA's K blocks (0.23 us), the K blocks of the CTAs that share an SM (0.22 us) and all blocks
//     over all SMs (0.28 us; 0.25 us where D is reduced into; more for rows of B under 128 bytes); CTAs
//     beyond one per SM add their own launch and store.  Tiles that one CTA per SM walks: the products of the
//     SM that has most of them, and all stores over all SMs.  The GPCs hold 14 clusters of 8 and 33 of 4 CTAs
//     that have an SM to themselves: more than that run in two turns.
//   either: the time of its bytes at 6.5 TB/s where they exceed 100 MB.
// Fitted to 1550 shapes (8 to 2488 rows, N 8 to 32768, K 8 to 16384, batches to 64, C none, bf16 and f32)
// and corrected on 1067 more (16 to 8192 rows): there 0.5 % from the best choice on average and over 8 % slower
// than the wide tiles in 2, 10 % at worst.  In microseconds, wide -> cluster: 64 x 5632 x 2048 36.1 -> 12.0 (4
// slices), 256 x 2048 x 2048 15.4 -> 9.2 (4), 512 x 5632 x 2048 31.8 -> 16.9 (2); the other way at 2048 x 2048 x 2048, 17.2 against
// 19.1, and for narrow outputs, where a wide tile's loads and store shrink with N: 128 x 32 x 64 3.4
// against 5.0, 59 x (1024 x 32 x 128) 8.4 against 12.0, D += A^T B 200 x 32 x 4096 7.0 against 10.6; D += A^T B
// 512 x 5632 x 5632, whose 176 tiles of 128 x 128 leave most SMs waiting for two, 30.6 against 42.6, and 2048 x 3072 x 5616, 384 tiles
// to walk in turns of 148, 56 against 91.
static int choose_cluster_splits(long long batch, long long M, long long N, long long K, bool adds_f32,
                                 bool adds_bf16, bool may_slice, bool reduces, bool tma_adds) {
  auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  auto part = [](long long n, int tile) { return static_cast<double>(n < tile ? n : tile) / tile; };
  const double kb = static_cast<double>(up(K, BK));
  const double sms = sm_count();
  const double megabytes = 1e-6 * batch * (2.0 * (M + N) * K + (adds_f32 ? 8.0 : adds_bf16 ? 4.0 : 2.0) * M * N);
  const double hbm = megabytes > 100.0 ? 3.5 + megabytes / 6.5 : 0.0;
  const bool one_cta = M <= BM;
  const long long wide_tiles = batch * (one_cta ? 1 : up(M, PAIR_M)) * up(N, BN);
  const long long wide_slots = one_cta ? sm_count() : sm_count() / 2;
  const double ragged = N % 32 != 0 && N > 32 ? 0.8 : 0.0;
  const double filled = part(N, BN) * part(M, one_cta ? BM : PAIR_M);
  double best = 1e30;
  for (int s = 1; s <= (may_slice && !one_cta ? 8 : 1) && (s == 1 || s * 8 <= kb); ++s) {
    const long long units = wide_tiles * s;
    const double busy = units < wide_slots ? static_cast<double>(units) / wide_slots : 1.0;
    const double loop = 0.275 * (1.0 + 0.23 * busy) * kb / s;
    double store, step;
    if (tma_adds) {
      // the additions' way to memory runs under the products and is felt where it is the longer
      const double way = 0.39 * 4e-6 * batch * M * N;
      const double own = 4.3 + loop + 2.8 * filled + static_cast<double>(up(units, wide_slots) - 1) * fmax(1.2, loop + 3.0);
      best = fmin(best, 0.95 * fmax(pow(pow(own, 2.5) + pow(way, 2.5), 0.4), hbm));
      continue;
    }
    if (!adds_f32) {
      store = 1.6 * filled + (!adds_bf16 ? ragged : N % 32 == 0 || N < 32 ? 2.2 : N < 128 ? 3.3 : 5.0);
      step = fmax(fmax(1.2, loop + 0.6), 2.7 * filled);
    } else if (s == 1) {
      store = 0.6 + ragged + (6.2 + 0.7 * busy) * filled;
      step = fmax(fmax(1.2, loop + 0.6), 8.5 * filled);
    } else {
      store = 0.35 + 4.6 * filled;
      step = loop + 20.0 * filled;
    }
    const double t = (one_cta ? 3.45 : 4.3) + loop + store + static_cast<double>(up(units, wide_slots) - 1) * step;
    best = fmin(best, 0.95 * fmax(t, hbm));
  }
  const long long tiles = batch * up(M, 128) * up(N, CLUSTER_TILE_N);
  if (tiles > (1 << 20)) return 0;
  const double rows = part(M, 128), per_sm = static_cast<double>(tiles) / sms;
  const double fixed[4] = {3.3 + 1.55 * rows, 4.25 + 1.55 * rows, 5.45 + 0.75 * rows, 4.1 + 2.2 * rows};
  const double crowded[4] = {2.1, 3.15, 4.05, 5.55}, short_rows = N < 32 ? 2.0 : N < 64 ? 1.3 : 1.0;
  int splits = 0;
  for (int i = 0; i < 4 && (1 << i) <= kb; ++i) {
    const long long ctas = tiles << i;
    const double per_cta = kb / (1 << i);
    double t = fixed[i] + fmax(fmax(0.23 * per_cta, ctas > sm_count() ? 0.22 * up(ctas, sm_count()) * per_cta : 0.0),
                               (reduces ? 0.25 : 0.28) * short_rows * per_sm * kb);
    if (ctas > sm_count()) t += (crowded[i] + (adds_bf16 ? 0.8 : 0.0)) * (static_cast<double>(ctas) / sms - 1.0);
    else if ((i == 2 && tiles > sm_count() / 4 - 4) || (i == 3 && tiles > sm_count() / 8 - 4)) t *= 2.0;
    if (i == 3) t += 0.13 * static_cast<double>(tiles < 14 ? tiles : 14);
    if (adds_f32) t += reduces ? 0.3 * per_sm : 0.2 + 1.2 * rows;
    if (adds_bf16) t += 0.8 * rows;
    // From two tiles per SM on, unsplit additions into D are walked by one CTA per SM.
    if (reduces && i == 0 && tiles >= 2 * sm_count())
      t = 4.3 + 2.2 * per_sm + 0.24 * kb * static_cast<double>(up(tiles, sm_count()));
    t = fmax(t, hbm);
    if (t < best) {
      best = t;
      splits = 1 << i;
    }
  }
  return splits;
}

// K slices of a CTA-pair product that adds into D.
// time ~ waves * (K slice + a fixed per-unit cost of epilogue / ramp).  The fixed part is worth
// ~6 K blocks without slices and ~10 with them, whose additions into D are reductions at the L2
// (fitted to 47 shapes, 64 to 16384 deep; mean distance from the best slice count 0.4 %, worst
// 6 %; with 6 for both 1.3 % and 25 %: 2048 x 5632 x 2048 takes 53 us whole and 66 us in two
// slices, 2048 x 6144 x 16384 285 whole and 299 in three).
static int choose_pair_slices(long long tiles, int k_blocks, long long clusters) {
  int best_s = 1;
  double best_cost = 1e30;
  for (int sp = 1; sp <= 8 && sp * 8 <= k_blocks; ++sp) {
    const long long waves = (tiles * sp + clusters - 1) / clusters;
    const double cost = static_cast<double>(waves) * (static_cast<double>(k_blocks) / sp + (sp == 1 ? 6.0 : 10.0));
    if (cost < best_cost * 0.97) {
      best_cost = cost;
      best_s = sp;
    }
  }
  return best_s;
}

}  // namespace gemm

static int32_t check_epi_operand(const char* name, const cdl_tensor* t, long long M, long long N) {
  if (!t || t->rank != 2 || t->shape[0] != M || t->shape[1] != N || t->dtype != CDL_BF16 ||
      t->stride[1] != 1 || t->stride[0] % 8 != 0 || (reinterpret_cast<uintptr_t>(t->ptr) & 15) != 0)
    return fail(CDL_ERR_INVALID,
                "matmul (fused SwiGLU): %s must be bf16 [%lld, %lld] with 16-byte aligned rows", name, M, N);
  return CDL_OK;
}

int32_t matmul_execute(const cdl_tensor* a, const cdl_tensor* b, const cdl_tensor* c,
                       const cdl_tensor* d, float alpha, float beta, cudaStream_t stream,
                       const cdl_matmul_options* opts, void* scratch, size_t scratch_bytes, int early) {
  return matmul_execute_epi(a, b, c, d, alpha, beta, 0, nullptr, nullptr, nullptr, stream, opts, nullptr, scratch,
                            scratch_bytes, early);
}

int32_t matmul_execute_epi(const cdl_tensor* a, const cdl_tensor* b, const cdl_tensor* c,
                           const cdl_tensor* d, float alpha, float beta, int epi_mode,
                           const cdl_tensor* aux0, const cdl_tensor* aux1, const cdl_tensor* out2,
                           cudaStream_t stream, const cdl_matmul_options* opts, const RopeEpilogue* rope,
                           void* scratch, size_t scratch_bytes, int early) {
  using namespace gemm;
  const int variant = opts ? opts->variant : CDL_GEMM_AUTO;
  if (variant < CDL_GEMM_AUTO || variant > CDL_GEMM_CTA_PAIR)
    return fail(CDL_ERR_INVALID, "matmul: unknown kernel variant %d", variant);
  if (!a || !b || !d) return fail(CDL_ERR_INVALID, "matmul: a, b and d are required");
  if (a->rank != b->rank || (a->rank != 2 && a->rank != 3) || d->rank != a->rank)
    return fail(CDL_ERR_INVALID,
                "matmul operands must all have rank 2 or all rank 3 (got rank %d, %d, %d)",
                a->rank, b->rank, d->rank);
  const bool f32_inputs = a->dtype == CDL_F32 && b->dtype == CDL_F32;
  if (!f32_inputs && (a->dtype != CDL_BF16 || b->dtype != CDL_BF16))
    return fail(CDL_ERR_INVALID, "matmul inputs must be f32 or bf16 and of one type (got %s x %s)",
                dtype_name(a->dtype), dtype_name(b->dtype));
  if (f32_inputs && epi_mode != 0)
    return fail(CDL_ERR_UNSUPPORTED, "matmul (fused SwiGLU): inputs must be bf16");
  if (d->dtype != CDL_BF16 && d->dtype != CDL_F32)
    return fail(CDL_ERR_INVALID, "matmul output must be f32 or bf16");
  const int r = a->rank;
  const long long batch = r == 3 ? a->shape[0] : 1;
  const long long M = a->shape[r - 2], K = a->shape[r - 1], N = b->shape[r - 1];
  if (b->shape[r - 2] != K)
    return fail(CDL_ERR_INVALID, "matmul contraction dimensions differ: a is [.., %lld, %lld], b is [.., %lld, %lld]",
                M, K, (long long)b->shape[r - 2], N);
  if (r == 3 && (b->shape[0] != batch || d->shape[0] != batch))
    return fail(CDL_ERR_INVALID, "matmul batch dimensions differ");
  if (d->shape[r - 2] != M || d->shape[r - 1] != N)
    return fail(CDL_ERR_INVALID, "matmul output shape must be [%lld, %lld]", M, N);
  if (d->stride[r - 1] != 1 && N > 1)
    return fail(CDL_ERR_INVALID, "matmul output must be row-major with a contiguous last dimension");
  const bool use_c = c != nullptr && beta != 0.0f;
  if (use_c) {
    if (c->rank != r || c->shape[r - 2] != M || c->shape[r - 1] != N ||
        (r == 3 && c->shape[0] != batch))
      return fail(CDL_ERR_INVALID, "matmul c must have the output's shape");
    if (c->dtype != CDL_BF16 && c->dtype != CDL_F32)
      return fail(CDL_ERR_INVALID, "matmul c must be f32 or bf16");
    if (c->stride[r - 1] != 1 && N > 1)
      return fail(CDL_ERR_INVALID, "matmul c must have a contiguous last dimension");
  }
  if (batch == 0 || M == 0 || N == 0) return CDL_OK;  // empty output: nothing to do
  if (K == 0) return fail(CDL_ERR_INVALID, "matmul: K is zero");
  if (M > INT32_MAX || N > INT32_MAX || K > INT32_MAX || batch > 65535)
    return fail(CDL_ERR_UNSUPPORTED, "matmul dimension too large");

  // f32 inputs, and bf16 operands TMA cannot describe (unaligned pointer or leading dimension):
  // the general kernel (gemm_general.cu).  Operands without any contiguous dimension
  // stay rejected, as in the reference.
  if (f32_inputs) return matmul_general_execute(a, b, c, d, alpha, beta, scratch, scratch_bytes, stream);
  OperandLayout la, lb;
  for (int which = 0; which < 2; ++which) {
    const int32_t rc = which == 0 ? analyze_operand("a", a, true, &la) : analyze_operand("b", b, false, &lb);
    if (rc == CDL_ERR_UNSUPPORTED && epi_mode == 0)
      return matmul_general_execute(a, b, c, d, alpha, beta, scratch, scratch_bytes, stream);
    CDL_CHECK(rc);
  }

  // Kernel choice, unless the caller's options name a variant: clusters that share a tile's K range where
  // that is estimated to be faster, else CTA pairs (256 x 256 tiles) whenever the problem has more
  // than one 128-row slab.
  // The weight-gradient form D = C + A^T B, f32 in place, may add K slices into D with atomics.
  const bool adds_f32 = use_c && c->dtype == CDL_F32;
  const bool may_slice = adds_f32 && d->dtype == CDL_F32 && c->ptr == d->ptr && beta == 1.0f &&
                         !(opts && opts->deterministic != 0);
  // In the cluster kernel it adds every element once, by vector reductions where D's rows allow them.
  const bool reduces = may_slice && N % 4 == 0 && (reinterpret_cast<uintptr_t>(d->ptr) & 15) == 0 &&
                       (M == 1 || (d->stride[r - 2] % 4 == 0 && c->stride[r - 2] == d->stride[r - 2])) &&
                       (r == 2 || (d->stride[0] % 4 == 0 && c->stride[0] == d->stride[0]));
  // In the pair kernel TMA adds, where it can describe D.
  const bool tma_adds = M > BM && adds_f32 && d->dtype == CDL_F32 && c->ptr == d->ptr && beta == 1.0f &&
                        (reinterpret_cast<uintptr_t>(d->ptr) & 15) == 0 && d->stride[r - 2] % 4 == 0 &&
                        d->stride[r - 2] >= N && c->stride[r - 2] == d->stride[r - 2] &&
                        (r == 2 || batch == 1 ||
                         (d->stride[0] % 4 == 0 && d->stride[0] > 0 && c->stride[0] == d->stride[0]));
  auto splits_of = [&](bool tma) {
    return choose_cluster_splits(batch, M, N, K, adds_f32, use_c && !adds_f32, may_slice, reduces, tma);
  };
  int cluster_splits = variant == CDL_GEMM_AUTO ? splits_of(tma_adds) : 0;
  // The error of a sum in the tensor core grows with its length: a shorter store is no reason for fewer K slices (129 x
  // 384 x 640 whole instead of in four slices: 4.7e-7 off, not 1.3e-7).  One in a thousand weight gradients.
  if (variant == CDL_GEMM_AUTO && cluster_splits == 0 && tma_adds) {
    const int sliced = splits_of(false);
    const long long tiles = batch * ((M + PAIR_M - 1) / PAIR_M) * ((N + BN - 1) / BN);
    if (sliced > (may_slice ? choose_pair_slices(tiles, static_cast<int>((K + BK - 1) / BK), sm_count() / 2) : 1))
      cluster_splits = sliced;
  }
  const bool use_cluster = cluster_splits > 0;
  const bool use_pair = !use_cluster && (variant == CDL_GEMM_AUTO ? M > BM : variant == CDL_GEMM_CTA_PAIR);
  const int tile_m = use_pair ? PAIR_M : BM;
  const int tile_n = use_cluster ? CLUSTER_TILE_N : BN;
  const uint32_t b_box_rows = use_pair ? BN / 2 : tile_n;

  CUtensorMap tm_a, tm_b;
  {
    // Innermost-first dims: K-major operand = [K, M|N, batch]; MN-major = [M|N, K, batch].
    const uint64_t bs_a = static_cast<uint64_t>(batch > 1 ? la.batch : la.ld * (la.mn_major ? K : M)) * 2;
    const uint64_t bs_b = static_cast<uint64_t>(batch > 1 ? lb.batch : lb.ld * (lb.mn_major ? K : N)) * 2;
    uint64_t da[3], sa[3], db[3], sb[3];
    uint32_t ba[3], bb[3];
    if (la.mn_major) {
      da[0] = M; da[1] = K; ba[0] = 64; ba[1] = 64;
    } else {
      da[0] = K; da[1] = M; ba[0] = 64; ba[1] = BM;
    }
    da[2] = batch; ba[2] = 1; sa[0] = 0; sa[1] = la.ld * 2; sa[2] = bs_a;
    if (lb.mn_major) {
      db[0] = N; db[1] = K; bb[0] = 64; bb[1] = 64;
    } else {
      db[0] = K; db[1] = N; bb[0] = 64; bb[1] = b_box_rows;
    }
    db[2] = batch; bb[2] = 1; sb[0] = 0; sb[1] = lb.ld * 2; sb[2] = bs_b;
    CDL_CHECK(encode_tmap(&tm_a, a->ptr, CDL_BF16, 3, da, sa, ba, true));
    CDL_CHECK(encode_tmap(&tm_b, b->ptr, CDL_BF16, 3, db, sb, bb, true));
  }

  Params p;
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.K = static_cast<int>(K);
  p.batch = static_cast<int>(batch);
  p.num_m_tiles = static_cast<int>((M + tile_m - 1) / tile_m);
  p.num_n_tiles = static_cast<int>((N + tile_n - 1) / tile_n);
  const long long tiles = batch * p.num_m_tiles * p.num_n_tiles;
  if (tiles > INT32_MAX) return fail(CDL_ERR_UNSUPPORTED, "matmul: too many tiles");
  p.num_tiles = static_cast<int>(tiles);
  p.k_blocks = static_cast<int>((K + BK - 1) / BK);
  {
    // Raster panels: all M tiles of `raster_w` N tiles run together, so the panel's B columns
    // (raster_w * 256 * K elements) and, when it fits next to them, all of A are served from L2
    // while the panel lasts.  With a long K (the weight-gradient shapes: K = tokens) eight B
    // column panels plus A exceed the L2's 126 MB and both get evicted and re-read from HBM, so
    // the panel is narrowed until A and the panel's B fit a budget of 96 MB.
    const double a_bytes = 2.0 * static_cast<double>(M) * K;
    const double b_panel = 2.0 * BN * static_cast<double>(K);
    const double budget = static_cast<double>(CDL_GEMM_RASTER_BUDGET_MB) * 1024 * 1024;
    int w = RASTER_W;
    if (a_bytes <= 0.75 * budget)
      while (w > 2 && a_bytes + w * b_panel > budget) --w;
    p.raster_w = w;
  }
  p.a_mn = la.mn_major;
  p.b_mn = lb.mn_major;
  p.out_f32 = d->dtype == CDL_F32;
  p.c_mode = !use_c ? 0 : (c->dtype == CDL_BF16 ? 1 : 2);
  p.d = d->ptr;
  p.c = use_c ? c->ptr : nullptr;
  p.ldd = M > 1 ? d->stride[r - 2] : N;
  p.ldc = use_c ? (M > 1 ? c->stride[r - 2] : N) : 0;
  p.d_batch = r == 3 ? d->stride[0] : 0;
  p.c_batch = use_c && r == 3 ? c->stride[0] : 0;
  auto vec_ok = [](const void* ptr, long long ld, long long bstride, size_t es) {
    return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && (ld * es) % 16 == 0 &&
           (bstride * es) % 16 == 0;
  };
  p.d_vec = vec_ok(p.d, p.ldd, p.d_batch, dtype_size(d->dtype));
  p.c_vec = use_c ? vec_ok(p.c, p.ldc, p.c_batch, dtype_size(c->dtype)) : 0;
  p.alpha = alpha;
  p.beta = use_c ? beta : 0.0f;
  p.split_k = use_cluster ? cluster_splits : 1;
  p.sched_counter = nullptr;
  p.atomic_out = 0;
  p.tma_add = 0;
  p.early = (early & EARLY_PRODUCTS) ? (use_pair ? 2 : 0) : early > 0 ? 1 : 0;
  p.epi_mode = 0;
  p.aux0 = p.aux1 = nullptr;
  p.out2 = nullptr;
  p.ld_aux0 = p.ld_aux1 = p.ld_out2 = 0;
  p.rope_table = nullptr;
  p.rope_cu = nullptr;
  p.rope_seqlen = p.rope_cols = p.rope_nseq = 0;
  if (epi_mode == 3) {
    if (!rope || !rope->table || rope->seqlen <= 0 || rope->rot_cols < 0 || rope->rot_cols % 128 != 0 ||
        rope->rot_cols > N || (rope->cu_seqlens != nullptr && rope->num_seqs <= 0))
      return fail(CDL_ERR_INVALID, "matmul (RoPE epilogue): table, seqlen > 0 and rot_cols (a multiple of 128, "
                  "at most N) are required");
    if (r != 2 || use_c || d->dtype != CDL_BF16 || N % 128 != 0 || !p.d_vec ||
        (reinterpret_cast<uintptr_t>(rope->table) & 15) != 0)
      return fail(CDL_ERR_INVALID, "matmul (RoPE epilogue): rank 2, no C operand, bf16 output with 16-byte "
                  "aligned rows, N %% 128 == 0 and a 16-byte aligned table are required");
    p.epi_mode = 3;
    p.rope_table = rope->table;
    p.rope_cu = rope->cu_seqlens;
    p.rope_seqlen = rope->seqlen;
    p.rope_cols = rope->rot_cols;
    p.rope_nseq = rope->num_seqs;
  } else if (epi_mode != 0) {
    if (r != 2 || use_c || alpha != 1.0f || d->dtype != CDL_BF16 || N % 8 != 0 || !p.d_vec)
      return fail(CDL_ERR_INVALID,
                  "matmul (fused SwiGLU): rank 2, alpha 1, no C operand, bf16 output with 16-byte aligned rows "
                  "and N %% 8 == 0 are required");
    CDL_CHECK(check_epi_operand("aux0", aux0, M, N));
    CDL_CHECK(check_epi_operand("out2", out2, M, N));
    if (epi_mode == 2) CDL_CHECK(check_epi_operand("aux1", aux1, M, N));
    p.epi_mode = epi_mode;
    p.aux0 = static_cast<const __nv_bfloat16*>(aux0->ptr);
    p.ld_aux0 = aux0->stride[0];
    p.out2 = static_cast<__nv_bfloat16*>(out2->ptr);
    p.ld_out2 = out2->stride[0];
    if (epi_mode == 2) {
      p.aux1 = static_cast<const __nv_bfloat16*>(aux1->ptr);
      p.ld_aux1 = aux1->stride[0];
    }
  }
  {
    auto al32 = [](const void* ptr, long long ld, long long bstride, size_t es) {
      return (reinterpret_cast<uintptr_t>(ptr) & 31) == 0 && (ld * es) % 32 == 0 &&
             (bstride * es) % 32 == 0;
    };
    bool w = al32(p.d, p.ldd, p.d_batch, dtype_size(d->dtype));
    if (use_c) w = w && al32(p.c, p.ldc, p.c_batch, dtype_size(c->dtype));
    if (p.epi_mode == 1 || p.epi_mode == 2) {
      w = w && al32(p.aux0, p.ld_aux0, 0, 2) && al32(p.out2, p.ld_out2, 0, 2);
      if (p.epi_mode == 2) w = w && al32(p.aux1, p.ld_aux1, 0, 2);
    }
    p.wide = w ? 1 : 0;
  }
  p.status = device_status_ptr();
  if (!p.status) return fail(CDL_ERR_CUDA, "cannot resolve the device status word");

  // D += alpha * A^T B by TMA reductions (every element added to once per K slice).
  CUtensorMap tm_e0 = tm_a, tm_e1 = tm_a;  // (valid maps where none is used)
  const bool adds_in_place = adds_f32 && p.out_f32 && c->ptr == d->ptr && beta == 1.0f && p.ldc == p.ldd &&
                             p.c_batch == p.d_batch;
  if (use_pair && tma_adds) {
    const uint64_t dims[3] = {static_cast<uint64_t>(N), static_cast<uint64_t>(M), static_cast<uint64_t>(batch)};
    const uint64_t strides[3] = {0, static_cast<uint64_t>(p.ldd) * 4,
                                 static_cast<uint64_t>(batch > 1 ? p.d_batch : p.ldd * M) * 4};
    const uint32_t box[3] = {32, 32, 1};
    CDL_CHECK(encode_tmap(&tm_e0, p.d, CDL_F32, 3, dims, strides, box, true));
    p.tma_add = 1;
  }
  // (rows that overlap, one row for all of M for instance, are read by the store itself)
  const bool feeds = use_pair && (p.epi_mode == 1 || p.epi_mode == 2) && aux0->stride[0] >= N &&
                     (p.epi_mode == 1 || aux1->stride[0] >= N);
  if (feeds) {
    const cdl_tensor* aux[2] = {aux0, aux1};
    for (int i = 0; i < p.epi_mode; ++i) {
      const uint64_t ld = static_cast<uint64_t>(aux[i]->stride[0]) * 2;
      const uint64_t dims[3] = {static_cast<uint64_t>(N), static_cast<uint64_t>(M), 1};
      const uint64_t strides[3] = {0, ld, ld * M};
      const uint32_t box[3] = {32, 32, 1};
      CDL_CHECK(encode_tmap(i ? &tm_e1 : &tm_e0, aux[i]->ptr, CDL_BF16, 3, dims, strides, box, false, true));
    }
  }

  if (use_cluster) {
    // D += A^T B: every element is added to once, by a reduction at the L2, instead of read, added to and
    // written: 2048 x 5632 x 256 29 us instead of 34 (25 as a walk), 512 x 1536 x 256 5.6 instead of 7.7.  (The pair
    // kernel's tiles with TMA reductions: 25.9; with a thread's own reductions along its row 42.)
    if (reduces) {
      p.atomic_out = 1;
      p.c_mode = 0;
    }
    ProfileScope ps(PROF_GEMM, 2.0 * static_cast<double>(batch) * M * N * K, stream);
    return gemm_cluster_launch(tm_a, tm_b, p, early, stream);
  }

  static std::once_flag attr_once[64];
  static int max_clusters[64] = {};
  int dev = 0;
  CDL_CUDA(cudaGetDevice(&dev));
  cudaError_t attr_err = cudaSuccess;
  std::call_once(attr_once[dev & 63], [&] {
    attr_err = cudaFuncSetAttribute(gemm_bf16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(SMEM_BYTES));
    auto pair = [&](auto kernel, int kind) {
      if (attr_err == cudaSuccess)
        attr_err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(pair_smem_bytes(kind)));
    };
    pair(gemm_bf16_pair_kernel<STORE>, STORE);
    pair(gemm_bf16_pair_kernel<STORE_ADD>, STORE_ADD);
    pair(gemm_bf16_pair_kernel<STORE_SWIGLU>, STORE_SWIGLU);
    // How many CTA pairs the device can hold at once (GPCs with an odd SM count lose one SM).
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(sm_count() & ~1));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = pair_smem_bytes(STORE);
    if (attr_err == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&n, gemm_bf16_pair_kernel<STORE>, &cfg) == cudaSuccess && n > 0)
      max_clusters[dev & 63] = n;
    else
      max_clusters[dev & 63] = sm_count() / 2;
    (void)cudaGetLastError();
  });
  if (attr_err != cudaSuccess)
    return fail(CDL_ERR_CUDA, "cudaFuncSetAttribute failed: %s", cudaGetErrorString(attr_err));

  // K slicing for the accumulate-in-place form (D = C, f32, beta = 1: the weight-gradient GEMM,
  // whose output is small and whose K is long).  Slices add into D with atomics, which removes
  // the tile-count quantisation (e.g. 192 tiles on 74 CTA pairs = 2.6 waves) at the price of an
  // unordered f32 sum; the caller's `deterministic` option turns it off.
  if (use_pair && adds_in_place) {
    if (!(opts && opts->deterministic != 0)) {
      const int best_s = choose_pair_slices(p.num_tiles, p.k_blocks, max_clusters[dev & 63]);
      if (best_s > 1) {
        p.split_k = best_s;
        p.atomic_out = 1;
        p.c_mode = 0;  // D already holds C; the slices only add
        // Only one K slice of the operands is live at a time (units are numbered slice by slice
        // within a chunk of tiles): the raster panel may be as wide as that slice allows.
        const double a_slice = 2.0 * static_cast<double>(M) * K / best_s;
        const double b_panel_slice = 2.0 * BN * static_cast<double>(K) / best_s;
        const double budget = static_cast<double>(CDL_GEMM_RASTER_BUDGET_MB) * 1024 * 1024;
        int w = RASTER_W;
        if (a_slice <= 0.75 * budget)
          while (w > 2 && a_slice + w * b_panel_slice > budget) --w;
        p.raster_w = w;
      }
    }
  }

  ProfileScope ps(PROF_GEMM, 2.0 * static_cast<double>(batch) * M * N * K, stream);
  if (use_pair) {
    const long long units = static_cast<long long>(p.num_tiles) * p.split_k;
    const int clusters = units < max_clusters[dev & 63] ? static_cast<int>(units) : max_clusters[dev & 63];
    p.sched_counter = units > clusters ? sched_counter_for(gemm_counter_kind(early), dev, stream) : nullptr;
    auto run = [&](auto kernel, int kind) {
      return launch_pdl(kernel, dim3(2 * clusters), dim3(THREADS), pair_smem_bytes(kind), stream, tm_a, tm_b, tm_e0, tm_e1, p);
    };
    CDL_CUDA(p.tma_add ? run(gemm_bf16_pair_kernel<STORE_ADD>, STORE_ADD)
             : feeds   ? run(gemm_bf16_pair_kernel<STORE_SWIGLU>, STORE_SWIGLU)
                       : run(gemm_bf16_pair_kernel<STORE>, STORE));
  } else {  // (this one always waits at its start)
    const int grid = p.num_tiles < sm_count() ? p.num_tiles : sm_count();
    CDL_CUDA(launch_pdl(gemm_bf16_kernel, dim3(grid), dim3(THREADS), SMEM_BYTES, stream, tm_a, tm_b, p));
  }
  CDL_CUDA(cudaGetLastError());
  return CDL_OK;
}

}  // namespace cdl

extern "C" {

int32_t cdl_b200_matmul(const cdl_tensor* a, const cdl_tensor* b, const cdl_tensor* c,
                        const cdl_tensor* d, float alpha, float beta, void* scratch,
                        size_t scratch_bytes, cdl_stream stream) {
  return cdl::matmul_execute(a, b, c, d, alpha, beta, static_cast<cudaStream_t>(stream), nullptr, scratch,
                             scratch_bytes);
}

int32_t cdl_b200_matmul_opt(const cdl_tensor* a, const cdl_tensor* b, const cdl_tensor* c,
                            const cdl_tensor* d, float alpha, float beta,
                            const cdl_matmul_options* options, void* scratch, size_t scratch_bytes,
                            cdl_stream stream) {
  return cdl::matmul_execute(a, b, c, d, alpha, beta, static_cast<cudaStream_t>(stream), options, scratch,
                             scratch_bytes);
}

int32_t cdl_b200_matmul_candidates(const cdl_tensor* a, const cdl_tensor* b, const cdl_tensor* d,
                                   cdl_matmul_options* out, int32_t capacity, int32_t* count) {
  using namespace cdl;
  if (!a || !b || !d || !count || (capacity > 0 && !out))
    return fail(CDL_ERR_INVALID, "matmul_candidates: a, b, d, count (and out) are required");
  cdl_matmul_options list[6];
  int n = 0;
  list[n++] = {CDL_GEMM_AUTO, 0};  // the heuristic's choice, which may be the cluster form (it has no name of its own)
  const bool tensor_core = a->dtype == CDL_BF16 && b->dtype == CDL_BF16 && a->rank >= 2 &&
                           a->rank == b->rank && [&] {
                             gemm::OperandLayout la, lb;
                             const bool ok = gemm::analyze_operand("a", a, true, &la) == CDL_OK &&
                                             gemm::analyze_operand("b", b, false, &lb) == CDL_OK;
                             last_error().clear();
                             return ok;
                           }();
  if (tensor_core) {
    const long long M = a->shape[a->rank - 2];
    const bool accumulates = d->dtype == CDL_F32;  // the weight-gradient form may slice K
    if (accumulates) list[n++] = {CDL_GEMM_AUTO, 1};
    const int first = M > gemm::BM ? CDL_GEMM_CTA_PAIR : CDL_GEMM_ONE_CTA;
    const int second = first == CDL_GEMM_CTA_PAIR ? CDL_GEMM_ONE_CTA : CDL_GEMM_CTA_PAIR;
    list[n++] = {first, 0};
    if (accumulates && first == CDL_GEMM_CTA_PAIR) list[n++] = {first, 1};
    list[n++] = {second, 0};
    if (accumulates && second == CDL_GEMM_CTA_PAIR) list[n++] = {second, 1};
  }
  *count = n;
  for (int i = 0; i < n && i < capacity; ++i) out[i] = list[i];
  return CDL_OK;
}

int32_t cdl_b200_matmul_swiglu_gate(const cdl_tensor* a, const cdl_tensor* b, const cdl_tensor* up,
                                    const cdl_tensor* gate_out, const cdl_tensor* act_out,
                                    cdl_stream stream) {
  return cdl::matmul_execute_epi(a, b, nullptr, gate_out, 1.0f, 0.0f, 1, up, nullptr, act_out,
                                 static_cast<cudaStream_t>(stream), nullptr, nullptr);
}

int32_t cdl_b200_matmul_rope(const cdl_tensor* a, const cdl_tensor* b, const cdl_tensor* cos_sin,
                             int32_t rot_heads, int32_t seqlen, const cdl_tensor* cu_seqlens,
                             const cdl_tensor* d, cdl_stream stream) {
  using namespace cdl;
  const char* op = "matmul (RoPE epilogue)";
  if (!cos_sin || cos_sin->rank != 2 || cos_sin->dtype != CDL_F32 || cos_sin->shape[1] != 128 ||
      cos_sin->stride[1] != 1 || cos_sin->stride[0] != 128 || seqlen <= 0 || cos_sin->shape[0] < seqlen)
    return fail(CDL_ERR_INVALID, "%s: cos_sin must be packed f32 [>= seqlen, 128] (head_dim 128)", op);
  if (rot_heads < 0) return fail(CDL_ERR_INVALID, "%s: rot_heads must not be negative", op);
  if (cu_seqlens && (cu_seqlens->rank != 1 || cu_seqlens->dtype != CDL_I32 || cu_seqlens->stride[0] != 1 ||
                     cu_seqlens->shape[0] < 2))
    return fail(CDL_ERR_INVALID, "%s: cu_seqlens must be a packed i32 vector of num_seqs + 1 entries", op);
  RopeEpilogue rope{static_cast<const float*>(cos_sin->ptr), seqlen, rot_heads * 128,
                    cu_seqlens ? static_cast<const int*>(cu_seqlens->ptr) : nullptr,
                    cu_seqlens ? static_cast<int>(cu_seqlens->shape[0] - 1) : 0};
  return matmul_execute_epi(a, b, nullptr, d, 1.0f, 0.0f, 3, nullptr, nullptr, nullptr,
                            static_cast<cudaStream_t>(stream), nullptr, &rope);
}

int32_t cdl_b200_matmul_swiglu_dgrad(const cdl_tensor* a, const cdl_tensor* b, const cdl_tensor* gate,
                                     const cdl_tensor* up, const cdl_tensor* d_up_out,
                                     const cdl_tensor* d_gate_out, cdl_stream stream) {
  return cdl::matmul_execute_epi(a, b, nullptr, d_up_out, 1.0f, 0.0f, 2, gate, up, d_gate_out,
                                 static_cast<cudaStream_t>(stream), nullptr, nullptr);
}

int32_t cdl_b200_matmul_scratch_bytes(const cdl_tensor* a, const cdl_tensor* b,
                                      const cdl_tensor* d, size_t* bytes_out) {
  using namespace cdl;
  if (bytes_out) *bytes_out = 0;
  if (!a || !b || !d || !bytes_out || (a->rank != 2 && a->rank != 3) || b->rank != a->rank || d->rank != a->rank ||
      a->dtype != b->dtype || (a->dtype != CDL_F32 && a->dtype != CDL_BF16) || a->shape[a->rank - 1] != b->shape[a->rank - 2])
    return CDL_OK;  // (the call itself says what is wrong)
  if (a->dtype == CDL_BF16) {
    gemm::OperandLayout la, lb;
    const int32_t ra = gemm::analyze_operand("a", a, true, &la), rb = gemm::analyze_operand("b", b, false, &lb);
    last_error().clear();
    if (ra == CDL_ERR_INVALID || rb == CDL_ERR_INVALID || (ra == CDL_OK && rb == CDL_OK)) return CDL_OK;
  }
  *bytes_out = matmul_general_scratch_bytes(a, b, d);
  return CDL_OK;
}

}  // extern "C"
