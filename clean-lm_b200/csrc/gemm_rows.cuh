// What the bf16 GEMM kernels share: the problem description and the row-wise epilogue of the kernels
// whose K slices meet inside a thread-block cluster (gemm_cluster.cu, gemm_general.cu).
#pragma once
#include "ptx.cuh"

namespace cdl {
namespace gemm {

constexpr int RASTER_W = 8;  // N tiles per raster panel (upper bound; see Params::raster_w)

struct Params {
  int M, N, K, batch;
  int num_m_tiles, num_n_tiles, num_tiles, k_blocks;
  int raster_w;        // N tiles per raster panel, 1 .. RASTER_W
  int a_mn, b_mn;      // 1 = operand is MN-major (M or N contiguous)
  int out_f32, c_mode; // c_mode: 0 none, 1 bf16, 2 f32
  void* d;
  const void* c;
  long long ldd, ldc, d_batch, c_batch;  // in elements
  int d_vec, c_vec;                      // 1 = rows are 16-byte aligned, vector access allowed
  float alpha, beta;
  int split_k;     // K slices per tile (pair kernel: accumulate-in-place form only; cluster kernels: CTAs
                   // per cluster); 1 = none
  int sum_blocks;  // gemm_general.cu: K blocks that one tensor-core accumulator sums up
  int atomic_out;  // 1 = add alpha * partial into D with red.global.add (D already holds C)
  int tma_add;     // 1 = the pair kernel adds by TMA reductions (add_chunk)
  // Fused SwiGLU epilogues (bf16 [M, N] operands, 16-byte aligned rows):
  //   1: D = G (the product),           out2 = SiLU(G) * aux0           (aux0 = up projection)
  //   2: D = SiLU(aux0) * R,            out2 = R * aux1 * dSiLU(aux0)   (R = product, aux0 = gate, aux1 = up)
  int wide;  // 1 = D, C and the fused operands all have 32-byte aligned rows: 256-bit accesses
  int epi_mode;
  const __nv_bfloat16* aux0;
  const __nv_bfloat16* aux1;
  __nv_bfloat16* out2;
  long long ld_aux0, ld_aux1, ld_out2;
  // Epilogue mode 3, rotate-half RoPE on the heads (128 columns each) below rope_cols:
  //   d[r, h 128 + i]      = x[i] cos(pos, i) - x[i + 64] sin(pos, i)
  //   d[r, h 128 + i + 64] = x[i + 64] cos(pos, i) + x[i] sin(pos, i)        (i < 64)
  // with x the product's row, pos = r % rope_seqlen, or r - cu_seqlens[b] for the sequence b that
  // holds row r of a ragged batch; the table is f32 [positions, 128] = cos | sin.
  const float* rope_table;
  const int* rope_cu;  // cu_seqlens of a ragged batch (device), or nullptr
  int rope_seqlen, rope_cols, rope_nseq;
  // Pair kernel: counter of the work units handed out beyond every cluster's first one (zero
  // between launches; one counter per device and stream).
  unsigned int* sched_counter;
  int* status;
  // 1 = starts before the kernel ahead of it has finished (see grid_dep_wait); 2 (CTA pairs) = the same, but what the
  // epilogue reads comes from that kernel: the epilogue waits for it.
  int early;
};

__device__ __forceinline__ void tile_coords(const Params& p, int tile, int& b, int& m, int& n) {
  const int per_batch = p.num_m_tiles * p.num_n_tiles;
  b = tile / per_batch;
  int r = tile - b * per_batch;
  const int panel_tiles = p.raster_w * p.num_m_tiles;
  const int panel = r / panel_tiles;
  const int first_n = panel * p.raster_w;
  const int width = min(p.raster_w, p.num_n_tiles - first_n);
  r -= panel * panel_tiles;
  m = r / width;
  n = first_n + (r - m * width);
}

// sigmoid(x) = 0.5 + 0.5 tanh(x / 2): one MUFU operation per element (tanh.approx, relative error
// about 2^-11, below the bf16 rounding of the outputs).  The reference's fused epilogues use
// rcp.approx(1 + ex2.approx(-x log2 e)) (crates/cleandl/rust-kernels/src/sky_matmul/
// tcgen05_bf16.rs:851-854), two MUFU operations; at 16 per clock per SM the 65536 elements of a
// 256 x 256 tile then cost half the time of the tile's main loop, and the epilogue warps, not the
// tensor pipe, set the pace of the fused GEMMs.
__device__ __forceinline__ float fast_sigmoid(float x) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * x));
  return fmaf(0.5f, t, 0.5f);
}

// gemm_cluster.cu.  p.split_k = 1, 2, 4 or 8; tensor maps with boxes of 128 rows (K-major operands) or
// 64 x 64 (MN-major).
constexpr int CLUSTER_TILE_N = 128;
int32_t gemm_cluster_launch(const CUtensorMap& tm_a, const CUtensorMap& tm_b, const Params& p,
                            int early, cudaStream_t stream);

// ------------------------------------------------------------------ D += alpha * accumulator
// A warp's 32 rows x 32 columns of an f32 accumulator go to D as one TMA reduction from a 4 KiB buffer of shared
// memory (tensor map of D: [N, M, batch], boxes of 32 x 32, the 128-byte swizzle, under which the rows' 16-byte
// stores meet no bank twice).  A thread owns a row of the accumulator, so its own accesses to D take 32 lines
// per instruction and, where C is read first, a round trip to HBM per 32 columns; the reduction is one
// instruction, nothing waits for it, and the L2 adds whole lines.  Every element is added to once per K slice.
constexpr int CHUNK_BYTES = 32 * 32 * 4;
__device__ __forceinline__ void add_chunk(const CUtensorMap* tm_d, uint8_t* buf, const uint32_t (&r)[32], float alpha,
                                          int lane, int col0, int row0, int b) {
  const uint32_t row = smem_u32(buf) + lane * 128, x = (lane & 7) << 4;
#pragma unroll
  for (int c = 0; c < 8; ++c)
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(row + ((c << 4) ^ x)),
                 "f"(alpha * __uint_as_float(r[4 * c])), "f"(alpha * __uint_as_float(r[4 * c + 1])),
                 "f"(alpha * __uint_as_float(r[4 * c + 2])), "f"(alpha * __uint_as_float(r[4 * c + 3]))
                 : "memory");
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    tma_reduce_add_3d(tm_d, buf, col0, row0, b);
    tma_store_commit();
  }
}

// ------------------------------------------------------------------ K slices that meet in a cluster
// A cluster of `splits` CTAs holds the partial sums of one 128 x 128 tile, one K slice per CTA.  Every
// CTA leaves its partial in its own shared memory, rows PART_LD floats apart (the four extra floats put
// the eight rows a quarter-warp writes with 128-bit stores on different banks), and after a cluster
// barrier CTA `rank` adds up rows rank, rank + splits, ... in slice order: a fixed order, so results do
// not depend on timing, and no memory outside the SMs is touched.  A warp owns a row: its stores (and
// the loads of C or of the fused operands) cover whole 128-byte lines, also where a row starts off the
// 16-byte grid.
constexpr int PART_LD = 132;
constexpr int PART_BYTES = 128 * PART_LD * 4;
constexpr int MAX_SPLITS = 8;

template <int S>
__device__ __forceinline__ float4 ld_part_f4(uint32_t addr) {
  float4 v;
  if (S == 1)
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  else
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr));
  return v;
}
template <int S>
__device__ __forceinline__ float ld_part_f1(uint32_t addr) {
  float v;
  if (S == 1) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  else asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

// Stores a partial tile: thread = row (TMEM lane), `cols` columns from col0 (a multiple of 4).
template <int COLS>
__device__ __forceinline__ void store_partial(float* part, int row, int col0, const float (&v)[COLS]) {
#pragma unroll
  for (int j = 0; j < COLS; j += 4)
    *reinterpret_cast<float4*>(part + row * PART_LD + col0 + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
}

// Position of a row in its sequence, for the RoPE table (see Params::rope_cu).
__device__ __forceinline__ int rope_position(const Params& p, int row) {
  if (p.rope_cu == nullptr) return row % p.rope_seqlen;
  int lo = 0, hi = p.rope_nseq;  // largest b with cu[b] <= row
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (p.rope_cu[mid] <= row) lo = mid;
    else hi = mid;
  }
  return row < p.rope_cu[p.rope_nseq] ? min(row - p.rope_cu[lo], p.rope_seqlen - 1) : 0;
}

// A warp's share of the output: rows rank + S * (warp + W i) of the tile, for W warps in each of the
// cluster's S CTAs, BATCH of them at a time: loads of a batch are in flight together.  prefetch() brings
// the first batch's C or fused operands into registers and may run while the products are still under
// way; finish() is called between two cluster barriers.
//
// The loops over batches stay loops and every form has its own: a tile's rows are few, so what is
// executed here is executed once or twice per launch, from a cold instruction cache.  Unrolled over
// 16 rows with all forms in the row's body, a row cost 2000 clk and the store of a tile 34000; like this
// the tile takes a tenth of it.
//
// PAIR: the cluster holds S pairs of CTAs; slice s of this CTA's 128 rows lies in CTA 2 s + (its rank & 1).
// ROWS: rows off the 16-byte grid that a warp takes at a time (finish_scalar).  Four pay where a CTA has 128 rows and many K
// blocks (cluster kernel, 515 x 1030 x 2056: 21.6 -> 16.8 us); the general kernel's products, most of them small, take one
// (16 x 515 x 515 7.2 us, four 9.6; 8 x 4097 x 4097 23.8 and 25.5).
template <int S, int W, bool PAIR = false, int ROWS = 4>
struct TileOut {
  static __device__ __forceinline__ uint32_t part_of(uint32_t at, int s) {
    return S == 1 ? at : mapa_shared(at, PAIR ? 2 * s + (cluster_ctarank() & 1) : s);
  }
  static constexpr int STEP = S * W;
  static constexpr int BATCH = S == 8 ? 2 : 4;
  uint4 pre[BATCH];

  // Everything a row's vector path touches starts on the 16-byte grid (the fused forms demand it), and
  // the last four columns of the tile exist or are outside together.
  static __device__ __forceinline__ bool vec(const Params& p) {
    return p.d_vec && (p.c_mode == 0 || p.c_vec) && p.N % 4 == 0;
  }

  __device__ __forceinline__ void load_extra(const Params& p, int r0, int b, int m0, int col) {
    const int rows = min(128, p.M - m0);
    if (p.c_mode == 2) {
      const float* c = static_cast<const float*>(p.c) + b * p.c_batch + m0 * p.ldc + col;
#pragma unroll
      for (int i = 0; i < BATCH; ++i)
        if (r0 + STEP * i < rows) pre[i] = *reinterpret_cast<const uint4*>(c + (r0 + STEP * i) * p.ldc);
    } else if (p.c_mode == 1 || p.epi_mode == 1 || p.epi_mode == 2) {
      const bool aux = p.c_mode == 0;
      const __nv_bfloat16* c = aux ? p.aux0 : static_cast<const __nv_bfloat16*>(p.c) + b * p.c_batch;
      const long long ld = aux ? p.ld_aux0 : p.ldc;
#pragma unroll
      for (int i = 0; i < BATCH; ++i)
        if (r0 + STEP * i < rows) {
          const uint2 q = *reinterpret_cast<const uint2*>(c + (m0 + r0 + STEP * i) * ld + col);
          pre[i].x = q.x;
          pre[i].y = q.y;
        }
      if (p.epi_mode == 2) {
#pragma unroll
        for (int i = 0; i < BATCH; ++i)
          if (r0 + STEP * i < rows) {
            const uint2 q = *reinterpret_cast<const uint2*>(p.aux1 + (m0 + r0 + STEP * i) * p.ld_aux1 + col);
            pre[i].z = q.x;
            pre[i].w = q.y;
          }
      }
    }
  }

  __device__ __forceinline__ void prefetch(const Params& p, int rank, int warp, int b, int m0, int n0) {
    const int lane = threadIdx.x & 31;
    const int col = n0 + lane * 4;
    if (!vec(p)) return;
    if (col < p.N) load_extra(p, rank + S * warp, b, m0, col);
  }

  __device__ __forceinline__ void finish(const Params& p, const float* part, int rank, int warp, int b, int m0,
                                         int n0) {
    const int lane = threadIdx.x & 31;
    const int rows = min(128, p.M - m0);
    const uint32_t base = smem_u32(part);
    if (!vec(p)) {
      finish_scalar(p, base, rank, warp, b, m0, n0);
      return;
    }
    const int col = n0 + lane * 4;
#pragma unroll 1
    for (int r0 = rank + S * warp; r0 < rows; r0 += STEP * BATCH) {
      float v[BATCH][4];
#pragma unroll
      for (int i = 0; i < BATCH; ++i) {
        // rows past the end are read like the others (the buffer has 128) and not stored
        const uint32_t at = base + min(r0 + STEP * i, 127) * (PART_LD * 4) + lane * 16;
        float4 q[S];
#pragma unroll
        for (int s = 0; s < S; ++s) q[s] = ld_part_f4<S>(part_of(at, s));
        v[i][0] = q[0].x; v[i][1] = q[0].y; v[i][2] = q[0].z; v[i][3] = q[0].w;
#pragma unroll
        for (int s = 1; s < S; ++s) {
          v[i][0] += q[s].x; v[i][1] += q[s].y; v[i][2] += q[s].z; v[i][3] += q[s].w;
        }
      }
#pragma unroll
      for (int i = 0; i < BATCH; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j] *= p.alpha;
      if (p.epi_mode == 3 && n0 < p.rope_cols) {  // warp-uniform
        // lane l holds columns 4l .. 4l + 3 of a head; the other half of each rotated pair is on lane l ^ 16
        const float sign = lane < 16 ? -1.f : 1.f;
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
          const int row = m0 + min(r0 + STEP * i, rows - 1);
          const float* cs = p.rope_table + static_cast<long long>(rope_position(p, row)) * 128 + (lane & 15) * 4;
          const float4 c = __ldg(reinterpret_cast<const float4*>(cs));
          const float4 sn = __ldg(reinterpret_cast<const float4*>(cs + 64));
          float o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) o[j] = sign * __shfl_xor_sync(0xffffffffu, v[i][j], 16);
          v[i][0] = v[i][0] * c.x + o[0] * sn.x;
          v[i][1] = v[i][1] * c.y + o[1] * sn.y;
          v[i][2] = v[i][2] * c.z + o[2] * sn.z;
          v[i][3] = v[i][3] * c.w + o[3] * sn.w;
        }
      }
      if (col < p.N) {
        if (p.c_mode == 2) {
#pragma unroll
          for (int i = 0; i < BATCH; ++i) {
            v[i][0] += p.beta * __uint_as_float(pre[i].x);
            v[i][1] += p.beta * __uint_as_float(pre[i].y);
            v[i][2] += p.beta * __uint_as_float(pre[i].z);
            v[i][3] += p.beta * __uint_as_float(pre[i].w);
          }
        } else if (p.c_mode == 1) {
#pragma unroll
          for (int i = 0; i < BATCH; ++i) {
            v[i][0] += p.beta * bf16_lo(pre[i].x);
            v[i][1] += p.beta * bf16_hi(pre[i].x);
            v[i][2] += p.beta * bf16_lo(pre[i].y);
            v[i][3] += p.beta * bf16_hi(pre[i].y);
          }
        }
        if (p.epi_mode == 1 || p.epi_mode == 2) store_swiglu(p, v, r0, rows, m0, col);
        else if (p.atomic_out) {
          float* d = static_cast<float*>(p.d) + b * p.d_batch + m0 * p.ldd + col;
#pragma unroll
          for (int i = 0; i < BATCH; ++i)
            if (r0 + STEP * i < rows)
              asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(d + (r0 + STEP * i) * p.ldd),
                           "f"(v[i][0]), "f"(v[i][1]), "f"(v[i][2]), "f"(v[i][3])
                           : "memory");
        } else if (p.out_f32) {
          float* d = static_cast<float*>(p.d) + b * p.d_batch + m0 * p.ldd + col;
#pragma unroll
          for (int i = 0; i < BATCH; ++i)
            if (r0 + STEP * i < rows)
              *reinterpret_cast<float4*>(d + (r0 + STEP * i) * p.ldd) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
        } else {
          __nv_bfloat16* d = static_cast<__nv_bfloat16*>(p.d) + b * p.d_batch + m0 * p.ldd + col;
#pragma unroll
          for (int i = 0; i < BATCH; ++i)
            if (r0 + STEP * i < rows)
              *reinterpret_cast<uint2*>(d + (r0 + STEP * i) * p.ldd) =
                  make_uint2(pack_bf16x2(v[i][0], v[i][1]), pack_bf16x2(v[i][2], v[i][3]));
        }
        if (r0 + STEP * BATCH < rows) load_extra(p, r0 + STEP * BATCH, b, m0, col);
      }
    }
  }

  __device__ __forceinline__ void store_swiglu(const Params& p, const float (&v)[BATCH][4], int r0, int rows, int m0,
                                               int col) {
#pragma unroll
    for (int i = 0; i < BATCH; ++i) {
      const float x0[4] = {bf16_lo(pre[i].x), bf16_hi(pre[i].x), bf16_lo(pre[i].y), bf16_hi(pre[i].y)};
      const float x1[4] = {bf16_lo(pre[i].z), bf16_hi(pre[i].z), bf16_lo(pre[i].w), bf16_hi(pre[i].w)};
      float o1[4], o2[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float sg = fast_sigmoid(p.epi_mode == 1 ? v[i][j] : x0[j]);
        o1[j] = p.epi_mode == 1 ? v[i][j] : x0[j] * sg * v[i][j];
        o2[j] = p.epi_mode == 1 ? v[i][j] * sg * x0[j] : v[i][j] * x1[j] * (sg + x0[j] * sg * (1.0f - sg));
      }
      if (r0 + STEP * i < rows) {
        const long long row = m0 + r0 + STEP * i;
        *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.d) + row * p.ldd + col) =
            make_uint2(pack_bf16x2(o1[0], o1[1]), pack_bf16x2(o1[2], o1[3]));
        *reinterpret_cast<uint2*>(p.out2 + row * p.ld_out2 + col) =
            make_uint2(pack_bf16x2(o2[0], o2[1]), pack_bf16x2(o2[2], o2[3]));
      }
    }
  }

  // Rows off the 16-byte grid or a column count that is no multiple of 4 (never a fused form): lane l
  // takes columns l, l + 32, l + 64 and l + 96, so that every access of the warp is contiguous; ROWS at a
  // time, whose loads are in flight together.
  static __device__ __forceinline__ void finish_scalar(const Params& p, uint32_t base, int rank, int warp, int b,
                                                       int m0, int n0) {
    const int lane = threadIdx.x & 31;
    const int rows = min(128, p.M - m0);
    const long long at_c = b * p.c_batch + m0 * p.ldc + n0 + lane, at_d = b * p.d_batch + m0 * p.ldd + n0 + lane;
#pragma unroll 1
    for (int r0 = rank + S * warp; r0 < rows; r0 += STEP * ROWS) {
      float v[ROWS][4], c[ROWS][4];
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int r = r0 + STEP * i;
          const long long at = at_c + r * p.ldc + 32 * j;
          c[i][j] = 0.f;
          if (p.c_mode != 0 && r < rows && n0 + lane + 32 * j < p.N)
            c[i][j] = p.c_mode == 2 ? static_cast<const float*>(p.c)[at]
                                    : __bfloat162float(static_cast<const __nv_bfloat16*>(p.c)[at]);
        }
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t at = base + (min(r0 + STEP * i, 127) * PART_LD + lane + 32 * j) * 4;
          float q[S];
#pragma unroll
          for (int s = 0; s < S; ++s) q[s] = ld_part_f1<S>(part_of(at, s));
          v[i][j] = q[0];
#pragma unroll
          for (int s = 1; s < S; ++s) v[i][j] += q[s];
        }
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int r = r0 + STEP * i;
          if (r < rows && n0 + lane + 32 * j < p.N) {
            const long long at = at_d + r * p.ldd + 32 * j;
            const float x = p.c_mode != 0 ? p.alpha * v[i][j] + p.beta * c[i][j] : p.alpha * v[i][j];
            if (p.out_f32) static_cast<float*>(p.d)[at] = x;
            else static_cast<__nv_bfloat16*>(p.d)[at] = __float2bfloat16_rn(x);
          }
        }
    }
  }
};

}  // namespace gemm
}  // namespace cdl
