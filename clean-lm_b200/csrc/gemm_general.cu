// Matmul for the operands TMA cannot bring to the tensor cores as they are: bf16 pointers or leading
// dimensions off the 16-byte grid (the reference hands them to cuBLASLt, tests `unaligned_operands`,
// crates/cleandl/tests/matmul.rs:604-630) and f32 inputs (`f32_tf32_matmul`, tests/matmul.rs:243-265:
// the reference computes those with TF32 tensor cores, 10 mantissa bits; here they keep f32's 24, see below).
//
// D = alpha * A . B + beta * C, f32 accumulation.  Products of a short K are sums of plain FMAs
// (gemm_fma_kernel); the others go to the tensor cores.  128 x 128 tiles; the K range of a tile is shared by
// a cluster of 1, 2, 4 or 8 CTAs whose partial sums meet in distributed shared memory (gemm_rows.cuh).
//   warp 0       issues the tcgen05.mma (M128 N128 K16)
//   16 loader warps: a warp takes a row of 64 consecutive elements, a lane two of
//                them, with plain loads of any alignment, and writes them as bf16 into the
//                128-byte-swizzled tile the tensor core reads; the loads of the next K block are in
//                flight meanwhile
//   4 sum warps  add the tensor core's sums (of Params::sum_blocks) to the running sums
//
// f32 operands.  A f32 value is the exact sum of three bf16 values (8 significant bits each): x = h + m + l
// (the splitting of Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For
// Higher-Precision Computations", 2019).  Of the nine products of two such sums the six of h.h, h.m, m.h, m.m, h.l and l.h are
// taken; the others are below 2^-24 of the product.  bf16 products are exact in f32.  The tensor core
// truncates when it adds, so it only ever sums one K block of 64, the small terms first; the blocks
// are added with round-to-nearest.
// A value whose pieces leave bf16's range (inf, NaN, the largest and the smallest magnitudes) has no
// such sum, and where a product overflows, h.h and h.m or m.h may be infinities of either sign (1e30
// squared is one): a CTA that met such a value or a sum that is not finite computes its part of the tile
// again with plain FMAs (partial_by_fma).
// Measured error (2-norm, against f64) 5.5e-8 at K = 20, 7.8e-8 at 100 and 1.0e-7 to 1.3e-7 at 1024 .. 2048, where a
// chain of FMAs has 8.2e-8, 1.8e-7 and 5.7e-7 .. 8.1e-7.
//
// What bounds it: the loaders and the shared memory they share with the tensor core (f32: 96 KiB of
// pieces written and 192 KiB read per K block of 64), and every operand is converted again for each tile that uses it.
// With scratch for the pieces lay_out_kernel converts each operand once and gemm_pieces_kernel multiplies them by TMA;
// worth_laying_out chooses.  us without -> with scratch (FMAs on the CUDA cores): 1024 x 2048 x 1536 f32 69 -> 45
// (460), 1500 x 1027 x 2051 bf16 with odd rows 51 -> 25 (310).
#include "gemm_rows.cuh"
#include "host.h"
#include "ops.h"
#include "ptx.cuh"

#include <math.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace cdl {
namespace gemm_general {

using gemm::Params;

constexpr int TILE = 128, BK = 64;
constexpr int PIECE_BYTES = TILE * BK * 2;

// One operand: element (i, k), i an index of M or N, at ptr + batch * s_batch + i * s_mn + k * s_k.
struct Operand {
  const void* ptr;
  long long s_batch, s_mn, s_k;
  int mn;        // extent of M or N
  int mn_major;  // 1: rows of the tile run along M or N (contiguous there), 0: along K
  int pairs;     // 1: every row starts on a pair of elements and is contiguous: one load for two
};

template <typename T>
struct Traits;
template <>
struct Traits<float> {
  static constexpr int PIECES = 3, STAGES = 2;
};
template <>
struct Traits<__nv_bfloat16> {
  static constexpr int PIECES = 1, STAGES = 6;
};
constexpr int MAX_STAGES = 6;
// 21 warps leave 80 registers a thread: a loader holds its 8 rows of A and of B for the next K block.
constexpr int LOADERS = 16, ROWS = TILE / LOADERS;
constexpr int WARPS = 1 + LOADERS + 4, THREADS = WARPS * 32;
constexpr int TMEM_COLS = 512;  // two accumulators and the running sums, 128 columns each
template <typename T>
constexpr int stage_bytes() { return 2 * Traits<T>::PIECES * PIECE_BYTES; }
template <typename T>
constexpr size_t smem_bytes() { return 1024 + Traits<T>::STAGES * stage_bytes<T>() + 256; }

struct Barriers {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_word;
  int outside;  // f32: an element without an exact sum of three bf16 values, or a sum that is not finite, was met
};
static_assert(sizeof(Barriers) <= 256, "barriers fit behind the stages");

// Two elements of a row, as loaded.  Predicated loads in straight-line code: a row's loads wait for
// nothing, so all of a block's are in flight at once.
struct PairF32 { uint32_t x, y; };
struct PairBf16 { uint32_t x, y; };  // x | y << 16 (x: both elements where one load takes them)
__device__ __forceinline__ uint32_t load32_if(const void* p, int positive) {
  uint32_t v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.b32 %0, [%1];\n\t}\n"
               : "=r"(v)
               : "l"(p), "r"(positive));
  return v;
}
__device__ __forceinline__ uint32_t load16_if(const void* p, int positive) {
  uint32_t v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.u16 %0, [%1];\n\t}\n"
               : "=r"(v)
               : "l"(p), "r"(positive));
  return v;
}
__device__ __forceinline__ void load_pair_if(const float* p, PairF32& v, int positive) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %3, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t"
      "@p ld.global.v2.b32 {%0, %1}, [%2];\n\t}\n"
      : "=r"(v.x), "=r"(v.y)
      : "l"(p), "r"(positive));
}
__device__ __forceinline__ void load_pair_if(const __nv_bfloat16* p, PairBf16& v, int positive) {
  v.x = load32_if(p, positive);
  v.y = 0;
}
__device__ __forceinline__ uint32_t load_one_if(const float* p, int positive) { return load32_if(p, positive); }
__device__ __forceinline__ uint32_t load_one_if(const __nv_bfloat16* p, int positive) { return load16_if(p, positive); }
template <typename T>
struct PairOf { using type = PairF32; };
template <>
struct PairOf<__nv_bfloat16> { using type = PairBf16; };

// A loader warp's rows of one operand's tile.
template <typename T>
struct RowSource {
  const T* p;               // this lane's first element of row 0 of the next K block
  long long row_step, in_step, block_step;
  int rows, inner;          // rows, and elements of a row, that exist (K-dependent one: of the next block)
  int mn_major, pairs;
  __device__ __forceinline__ void init(const Operand& o, int batch, int mn0, int k0, int K, int w, int lane) {
    mn_major = o.mn_major;
    pairs = o.pairs;
    const int r0 = w * ROWS;
    long long i, k;
    if (mn_major) {  // rows: 64 K indices of two 64-wide panels
      i = mn0 + (r0 & ~63) + 2 * lane;
      k = k0 + (r0 & 63);
      row_step = o.s_k;
      in_step = o.s_mn;
      rows = K - static_cast<int>(k);
      inner = o.mn - (mn0 + (r0 & ~63));
    } else {
      i = mn0 + r0;
      k = k0 + 2 * lane;
      row_step = o.s_mn;
      in_step = o.s_k;
      rows = o.mn - static_cast<int>(i);
      inner = K - k0;
    }
    block_step = BK * o.s_k;
    p = static_cast<const T*>(o.ptr) + batch * o.s_batch + i * o.s_mn + k * o.s_k;
  }
  // Loads the rows of the next K block (zeros outside the operand) and moves on.
  __device__ __forceinline__ void load(typename PairOf<T>::type (&v)[ROWS], int lane) {
    // rows this lane's first and second element exist in
    const int first = 2 * lane < inner ? rows : 0, second = 2 * lane + 1 < inner ? rows : 0;
    const T* q = p;
    if (pairs && (inner >= BK || (inner & 1) == 0)) {
#pragma unroll
      for (int i = 0; i < ROWS; ++i, q += row_step) load_pair_if(q, v[i], second - i);
    } else {
#pragma unroll
      for (int i = 0; i < ROWS; ++i, q += row_step) {
        v[i].x = load_one_if(q, first - i);
        v[i].y = load_one_if(q + in_step, second - i);
      }
    }
    p += block_step;
    if (mn_major) rows -= BK;
    else inner -= BK;
  }
};

// Writes a warp's rows into the swizzled tile: row r is 128 bytes, its 16-byte chunk c at c ^ (r & 7).
// Returns false for an element that is not the sum of its bf16 pieces.
__device__ __forceinline__ bool store_rows(uint32_t tile, int lane, const PairBf16 (&v)[ROWS]) {
  const uint32_t chunk = (lane >> 2) << 4, in = (lane & 3) << 2;
#pragma unroll
  for (int i = 0; i < ROWS; ++i)
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + i * 128 + (chunk ^ ((i & 7) << 4)) + in),
                 "r"(v[i].x | (v[i].y << 16))
                 : "memory");
  return true;
}
// The pieces of two neighbours: x = h + m + l.  Returns false where that does not hold (NaN and infinities leave one).
__device__ __forceinline__ bool split_pair(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16x2(x, y);
  const float rx = x - bf16_lo(h), ry = y - bf16_hi(h);
  m = pack_bf16x2(rx, ry);
  const float tx = rx - bf16_lo(m), ty = ry - bf16_hi(m);
  l = pack_bf16x2(tx, ty);
  return bf16_lo(l) == tx && bf16_hi(l) == ty;
}
__device__ __forceinline__ bool store_rows(uint32_t tile, int lane, const PairF32 (&v)[ROWS]) {
  const uint32_t chunk = (lane >> 2) << 4, in = (lane & 3) << 2;
  bool exact = true;
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const uint32_t at = tile + i * 128 + (chunk ^ ((i & 7) << 4)) + in;
    uint32_t h, m, l;
    exact = split_pair(__uint_as_float(v[i].x), __uint_as_float(v[i].y), h, m, l) && exact;
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(h) : "memory");
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + PIECE_BYTES), "r"(m) : "memory");
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + 2 * PIECE_BYTES), "r"(l) : "memory");
  }
  return exact;
}

// ------------------------------------------------------------ plain FMAs
// A chain of FMAs over K in ascending order, both operands through shared memory FMA_K elements deep
// ([k][i], two buffers), the next FMA_K on their way in registers meanwhile.
constexpr int FMA_K = 16;
template <int N>
constexpr int fma_tile() { return FMA_K * (N + 4); }

__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// One operand's N x FMA_K elements, fetched by `THREADS_` threads (lanes walk the contiguous index) and
// written to shared memory as S.
template <typename T, typename S, int N, int THREADS_>
struct FmaSource {
  static constexpr int PER = N * FMA_K / THREADS_;
  static_assert(N * FMA_K % THREADS_ == 0 && THREADS_ % N == 0, "a thread's elements are evenly spaced");
  const T* q;           // this thread's first element of the next FMA_K
  long long step, adv;  // from element to element, from FMA_K to FMA_K
  int left_i, left_k;   // elements that exist from the first one on, along M or N and along K
  int di, dk;           // element to element, along either
  int at, dat;          // place in shared memory
  float v[PER];
  __device__ __forceinline__ void init(const Operand& o, int batch, int mn0, int k0, int k_end) {
    const int t = threadIdx.x;
    const int i = o.mn_major ? t % N : t / FMA_K, k = o.mn_major ? t / N : t % FMA_K;
    di = o.mn_major ? 0 : THREADS_ / FMA_K;
    dk = o.mn_major ? THREADS_ / N : 0;
    step = di * o.s_mn + dk * o.s_k;
    adv = FMA_K * o.s_k;
    left_i = o.mn - (mn0 + i);
    left_k = k_end - (k0 + k);
    at = k * (N + 4) + i;
    dat = dk * (N + 4) + di;
    q = static_cast<const T*>(o.ptr) + batch * o.s_batch + (mn0 + i) * o.s_mn + (k0 + k) * o.s_k;
  }
  // Zeros outside the operand.
  __device__ __forceinline__ void fetch() {
#pragma unroll
    for (int j = 0; j < PER; ++j) v[j] = j * di < left_i && j * dk < left_k ? as_f32(q[j * step]) : 0.f;
    q += adv;
    left_k -= FMA_K;
  }
  __device__ __forceinline__ void store(S* tile) const {
#pragma unroll
    for (int j = 0; j < PER; ++j) tile[at + j * dat] = static_cast<S>(v[j]);
  }
  static __device__ __forceinline__ float as_f32(float x) { return x; }
  static __device__ __forceinline__ float as_f32(__nv_bfloat16 x) { return __bfloat162float(x); }
};
// acc[i][4 c + j] += row ty * 4 + i of A times column tx * 4 + 64 c + j of B over FMA_K elements, of which `left`
// exist.  In f32 two columns at a time: packed FMAs round as single ones do.
template <int N, int C>
__device__ __forceinline__ void fma_block(const float* ta, const float* tb, int tx, int ty, int left,
                                          float (&acc)[4][4 * C]) {
  uint64_t sums[4][2 * C];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2 * C; ++j) sums[i][j] = pack_f32x2(acc[i][2 * j], acc[i][2 * j + 1]);
#pragma unroll
  for (int kk = 0; kk < FMA_K; ++kk) {
    if (kk % 4 == 0 && kk >= left) break;
    const float4 av = *reinterpret_cast<const float4*>(ta + kk * (N + 4) + ty * 4);
    const uint64_t ar[4] = {pack_f32x2(av.x, av.x), pack_f32x2(av.y, av.y), pack_f32x2(av.z, av.z), pack_f32x2(av.w, av.w)};
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const float4 bv = *reinterpret_cast<const float4*>(tb + kk * (N + 4) + tx * 4 + 64 * c);
      const uint64_t br[2] = {pack_f32x2(bv.x, bv.y), pack_f32x2(bv.z, bv.w)};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sums[i][2 * c + j]) : "l"(ar[i]), "l"(br[j]));
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2 * C; ++j) unpack_f32x2(sums[i][j], acc[i][2 * j], acc[i][2 * j + 1]);
}

// The CTA's part of the tile once more (see the top of the file), by the first 512 of its threads, 4 x 8
// sums each; 12 floats from shared memory for 32 FMAs, which is what bounds it.  1024 x 2048 x 1536 with one
// value of 1e-35, or only such: 409 us (74 without; 64 x 64 tiles of FMAs alone 457; thread by thread from
// global memory 5080, B transposed 18080); 2048 x 256 x 2048, all: 118 (33; 142; 1256).  `smem` is the start of the operand stages as an offset into shared memory: a pointer argument
// would be loaded from as a generic address.  The partial tile goes there, the operands' tiles behind it.
constexpr int REDO_THREADS = 512, REDO_FLOATS = 2 * fma_tile<TILE>();
static_assert(gemm::PART_BYTES + 2 * REDO_FLOATS * sizeof(float) <= Traits<float>::STAGES * 6 * PIECE_BYTES,
              "the FMA tiles fit behind the partial tile");
__device__ __noinline__ void partial_by_fma(const Operand oa, const Operand ob, int b, int m0, int n0, int k_begin,
                                            int k_end, int smem) {
  extern __shared__ uint8_t smem_raw[];
  float* part = reinterpret_cast<float*>(smem_raw + smem);
  float* tiles = reinterpret_cast<float*>(smem_raw + smem + gemm::PART_BYTES);
  const bool works = threadIdx.x < REDO_THREADS;
  const int tx = threadIdx.x & 15, ty = (threadIdx.x >> 4) & 31;
  FmaSource<float, float, TILE, REDO_THREADS> fa, fb;
  float acc[4][8] = {};
  if (works) {
    fa.init(oa, b, m0, k_begin, k_end);
    fb.init(ob, b, n0, k_begin, k_end);
    fa.fetch();
    fb.fetch();
  }
  int buf = 0;
  for (int k0 = k_begin; k0 < k_end; k0 += FMA_K, buf ^= 1) {
    float* ta = tiles + buf * REDO_FLOATS;
    float* tb = ta + fma_tile<TILE>();
    if (works) {
      fa.store(ta);
      fb.store(tb);
      if (k0 + FMA_K < k_end) {
        fa.fetch();
        fb.fetch();
      }
    }
    __syncthreads();  // the other buffer has been read by all who are here
    if (works) fma_block<TILE, 2>(ta, tb, tx, ty, FMA_K, acc);
  }
  if (works) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 2; ++c)
        *reinterpret_cast<float4*>(part + (ty * 4 + i) * gemm::PART_LD + tx * 4 + 64 * c) =
            make_float4(acc[i][4 * c], acc[i][4 * c + 1], acc[i][4 * c + 2], acc[i][4 * c + 3]);
  }
}

template <int S, int W, bool PAIR, int ROWS>
__device__ __forceinline__ void store_out(const Params& p, const float* part, int rank, int warp, int b, int m0,
                                          int n0) {
  gemm::TileOut<S, W, PAIR, ROWS> out;
  out.prefetch(p, rank, warp, b, m0, n0);
  out.finish(p, part, rank, warp, b, m0, n0);
}

// FINE: an accumulator sums up half a K block (see matmul_general_execute).
template <typename T, bool FINE>
__global__ void __launch_bounds__(THREADS, 1)
    gemm_general_kernel(const Params p, const Operand oa, const Operand ob) {
  using Tr = Traits<T>;
  constexpr bool F32 = Tr::PIECES == 3;
  constexpr int STAGES = Tr::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  Barriers* bars = reinterpret_cast<Barriers*>(smem + STAGES * stage_bytes<T>());
  volatile int* abort_word = &bars->abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], LOADERS);
      mbar_init(&bars->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->acc_full[i], 1);
      mbar_init(&bars->acc_empty[i], 4);
    }
    bars->abort_word = 0;
    bars->outside = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(&bars->tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  grid_dep_wait();  // the set-up above overlaps the previous kernel's tail
  grid_dep_launch();

  const int rank = p.split_k > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  int b, tm, tn;
  gemm::tile_coords(p, static_cast<int>(blockIdx.x) / p.split_k, b, tm, tn);
  const int m0 = tm * TILE, n0 = tn * TILE;
  const int kb0 = static_cast<int>(static_cast<long long>(rank) * p.k_blocks / p.split_k);
  const int kb1 = static_cast<int>(static_cast<long long>(rank + 1) * p.k_blocks / p.split_k);
  const int blocks = kb1 - kb0;  // at least 1: the host never takes more slices than K blocks
  float* part = reinterpret_cast<float*>(smem);

  if (warp == 0) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(TILE, TILE, oa.mn_major, ob.mn_major);
      const uint32_t a_lbo = oa.mn_major ? 8192u : 16u, b_lbo = ob.mn_major ? 8192u : 16u;
      const uint32_t a_kstep = oa.mn_major ? 2048u : 32u, b_kstep = ob.mn_major ? 2048u : 32u;
      for (int it = 0; !FINE && it < blocks; ++it) {
        const int s = it % STAGES, group = it / p.sum_blocks, acc = group & 1;
        const bool first = it == group * p.sum_blocks, last = it + 1 == blocks || it + 1 == (group + 1) * p.sum_blocks;
        if ((first && !mbar_wait(&bars->acc_empty[acc], ((group >> 1) & 1) ^ 1, abort_word, 231)) ||
            !mbar_wait(&bars->full[s], (it / STAGES) & 1, abort_word, 232))
          break;
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + s * stage_bytes<T>()), sb = sa + Tr::PIECES * PIECE_BYTES;
        const uint32_t d = tmem_base + acc * TILE;
        // pieces (of A, of B), the smallest products first: l.h h.l m.m m.h h.m h.h
        constexpr int terms = F32 ? 6 : 1;
        constexpr int pa[6] = {F32 ? 2 : 0, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
        for (int t = 0; t < terms; ++t)
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_ss(d, smem_desc_sw128(sa + pa[t] * PIECE_BYTES + k * a_kstep, a_lbo, 1024),
                    smem_desc_sw128(sb + pb[t] * PIECE_BYTES + k * b_kstep, b_lbo, 1024), idesc,
                    (!first || (t | k) != 0) ? 1u : 0u);
        umma_commit(&bars->empty[s]);
        if (last) umma_commit(&bars->acc_full[acc]);
      }
      if (FINE) {
        bool ok = true;
        for (int it = 0; it < blocks && ok; ++it) {
          const int s = it % STAGES;
          if (!mbar_wait(&bars->full[s], (it / STAGES) & 1, abort_word, 233)) break;
          const uint32_t sa = smem_u32(smem + s * stage_bytes<T>()), sb = sa + PIECE_BYTES;
#pragma unroll
          for (int acc = 0; acc < 2; ++acc) {
            ok = mbar_wait(&bars->acc_empty[acc], (it & 1) ^ 1, abort_word, 234);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int k = 2 * acc; k < 2 * acc + 2; ++k)
              umma_ss(tmem_base + acc * TILE, smem_desc_sw128(sa + k * a_kstep, a_lbo, 1024),
                      smem_desc_sw128(sb + k * b_kstep, b_lbo, 1024), idesc, k & 1);
            umma_commit(&bars->acc_full[acc]);
          }
          if (ok) umma_commit(&bars->empty[s]);
        }
      }
    }
  } else if (warp <= LOADERS) {
    // ------------------------------------------------------------ loaders
    const int w = warp - 1;
    RowSource<T> ra, rb;
    ra.init(oa, b, m0, kb0 * BK, p.K, w, lane);
    rb.init(ob, b, n0, kb0 * BK, p.K, w, lane);
    typename PairOf<T>::type va[ROWS], vb[ROWS];
    bool exact = true;
    ra.load(va, lane);
    rb.load(vb, lane);
    for (int it = 0; it < blocks; ++it) {
      const int s = it % STAGES;
      if (!mbar_wait(&bars->empty[s], ((it / STAGES) & 1) ^ 1, abort_word, 131)) break;
      const uint32_t sa = smem_u32(smem + s * stage_bytes<T>()) + w * ROWS * 128;
      exact = store_rows(sa, lane, va) && exact;
      if (it + 1 < blocks) ra.load(va, lane);
      exact = store_rows(sa + Tr::PIECES * PIECE_BYTES, lane, vb) && exact;
      if (it + 1 < blocks) rb.load(vb, lane);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->full[s]);
    }
    if (!exact) bars->outside = 1;
  }
  if (warp > LOADERS) {
    // ------------------------------------------------------------ running sums: thread = row
    // They live in tensor memory beside the two accumulators of the K blocks: 128 columns per thread
    // in registers would leave the loader warps too few.
    const int quad = warp & 3;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const int groups = FINE ? 2 * blocks : (blocks + p.sum_blocks - 1) / p.sum_blocks;
    float zero = 0.f;  // NaN once a sum that is not finite has been met
    for (int g = 0; g < groups; ++g) {
      const int acc = g & 1;
      if (!mbar_wait(&bars->acc_full[acc], (g >> 1) & 1, abort_word, 331)) break;
      tc_fence_after();
      const bool last = g + 1 == groups;
#pragma unroll
      for (int c = 0; c < TILE; c += 32) {
        uint32_t r[32], t[32];
        tmem_ld32(t_row + acc * TILE + c, r);
        if (g > 0) {
          tmem_ld32(t_row + 2 * TILE + c, t);
          tmem_wait_ld(r, t);
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(t[j]) + __uint_as_float(r[j]));
        } else {
          tmem_wait_ld(r);
        }
        if (last) {
          // Every product is done and every stage read: the partial tile takes their place.
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            v[j] = __uint_as_float(r[j]);
            if (F32) zero = fmaf(v[j], 0.f, zero);
          }
          gemm::store_partial(part, quad * 32 + lane, c, v);
        } else {
          tmem_st32(t_row + 2 * TILE + c, r);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_empty[acc]);
    }
    if (zero != 0.f) bars->outside = 1;
  }
  __syncwarp();
  if (F32) {
    __syncthreads();
    if (bars->outside != 0)
      partial_by_fma(oa, ob, b, m0, n0, kb0 * BK, min(kb1 * BK, p.K),
                     static_cast<int>(smem - smem_raw));
  }
  if (p.split_k > 1) cluster_sync_all();
  else __syncthreads();
  if (warp >= 1) {
    switch (p.split_k) {
      case 1: store_out<1, WARPS - 1, false, 1>(p, part, rank, warp - 1, b, m0, n0); break;
      case 2: store_out<2, WARPS - 1, false, 1>(p, part, rank, warp - 1, b, m0, n0); break;
      case 4: store_out<4, WARPS - 1, false, 1>(p, part, rank, warp - 1, b, m0, n0); break;
      default: store_out<8, WARPS - 1, false, 1>(p, part, rank, warp - 1, b, m0, n0); break;
    }
  }
  __syncwarp();
  if (p.split_k > 1) cluster_sync_all();  // the other slices have read this CTA's partial
  else __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (threadIdx.x == 0 && *abort_word != 0) atomicExch(p.status, *abort_word);
}

// ------------------------------------------------------------ operands laid out first
// The loaders above bring an operand's row in once for every tile that uses it, two elements a lane, and split
// f32 values as often.  With scratch lent by the caller each operand is read once instead: lay_out_kernel
// writes it as bf16 pieces with rows on the 16-byte grid (an aligned bf16 operand stays where it is),
// and gemm_pieces_kernel loads the pieces by TMA.  Same pieces, same products, same sums.
struct Layout {
  const void* src;  // element (o, i) of a batch at src + batch * s_batch + o * s_outer + i * s_inner
  long long s_batch, s_outer, s_inner;
  __nv_bfloat16* dst;  // [piece][batch][outer][pitch]
  long long piece;     // elements per piece
  int outer, inner, pitch;
  int mn_major;  // 1: `inner` runs along M or N
  int mn_tiles, k_blocks;
  int* outside;  // f32: [batch][mn tile][k block], 1 where a value is not the sum of its pieces
};

// One CTA per 128 (M or N) x 64 (K) block: 128 row segments of 64 elements, a lane two neighbours.  Bound by launch
// and latency.
constexpr int LAY_THREADS = 256, LAY_ROWS = 128 / (LAY_THREADS / 32);
template <typename T>
__global__ void __launch_bounds__(LAY_THREADS) lay_out_kernel(const Layout la, const Layout lb, int blocks_a) {
  grid_dep_wait();
  grid_dep_launch();
  const bool second = static_cast<int>(blockIdx.x) >= blocks_a;
  const Layout l = second ? lb : la;
  int r = static_cast<int>(blockIdx.x) - (second ? blocks_a : 0);
  const int kb = r % l.k_blocks;
  r /= l.k_blocks;
  const int tile = r % l.mn_tiles, b = r / l.mn_tiles;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int seg = warp * LAY_ROWS;  // this warp's first row segment
  const int o0 = l.mn_major ? kb * BK + (seg & 63) : tile * TILE + seg;
  const int i0 = (l.mn_major ? tile * TILE + (seg & 64) : kb * BK) + 2 * lane;
  const T* src = static_cast<const T*>(l.src) + b * l.s_batch + o0 * l.s_outer + i0 * l.s_inner;
  __nv_bfloat16* dst = l.dst + (static_cast<long long>(b) * l.outer + o0) * l.pitch + i0;
  const int rows = l.outer - o0, first = i0 < l.inner ? rows : 0, second_e = i0 + 1 < l.inner ? rows : 0;
  typename PairOf<T>::type v[LAY_ROWS];
#pragma unroll
  for (int i = 0; i < LAY_ROWS; ++i, src += l.s_outer) {
    v[i].x = load_one_if(src, first - i);
    v[i].y = load_one_if(src + l.s_inner, second_e - i);
  }
  bool exact = true;
#pragma unroll
  for (int i = 0; i < LAY_ROWS; ++i, dst += l.pitch) {
    if (i >= first) break;
    if constexpr (Traits<T>::PIECES == 1) {
      *reinterpret_cast<uint32_t*>(dst) = v[i].x | (v[i].y << 16);
    } else {
      uint32_t h, m, lo;
      exact = split_pair(__uint_as_float(v[i].x), __uint_as_float(v[i].y), h, m, lo) && exact;
      *reinterpret_cast<uint32_t*>(dst) = h;
      *reinterpret_cast<uint32_t*>(dst + l.piece) = m;
      *reinterpret_cast<uint32_t*>(dst + 2 * l.piece) = lo;
    }
  }
  if (Traits<T>::PIECES > 1) {
    const int any = __syncthreads_or(!exact);
    if (threadIdx.x == 0) l.outside[(static_cast<long long>(b) * l.mn_tiles + tile) * l.k_blocks + kb] = any != 0;
  }
}

// One CTA takes a 128 x 128 tile (M128 N128), a pair of CTAs 256 x 128 (cta_group::2, M256 N128: each its own 128 rows of
// A and half of B's 128 columns).  Products whose operands both come from shared memory run at 107 clk per M128
// N128 K16 in one CTA and at 64 in a pair; one CTA is for up to 128 rows.  A K block arrives in slots, a piece of A and
// the same piece of B each, the last pieces first: they are released first.  bf16: two CTAs share an SM where there
// are more than one per SM; the running sums live in registers, so the two accumulators take half of the tensor memory.
template <typename T>
struct PieceTraits;
template <>
struct PieceTraits<float> {
  static constexpr int SUM_WARPS = 16;
};
template <>
struct PieceTraits<__nv_bfloat16> {
  static constexpr int SUM_WARPS = 8;
};
constexpr int slot_bytes(bool pair) { return PIECE_BYTES + (pair ? PIECE_BYTES / 2 : PIECE_BYTES); }
constexpr int shared_slots(bool pair) { return pair ? 4 : 3; }  // 96 KiB
constexpr int alone_slots(bool pair) { return pair ? 9 : 6; }
constexpr int MAX_SLOTS = 9;
struct PieceBarriers {
  uint64_t full[MAX_SLOTS];
  uint64_t empty[MAX_SLOTS];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_word;
  int outside;
};
static_assert(sizeof(PieceBarriers) <= 256, "barriers fit behind the slots");
constexpr size_t piece_smem_bytes(int slots, bool pair) { return 1024 + slots * slot_bytes(pair) + 256; }
static_assert(gemm::PART_BYTES <= shared_slots(true) * slot_bytes(true), "the partial tile takes the slots' place");
static_assert(gemm::PART_BYTES + 2 * REDO_FLOATS * sizeof(float) <= alone_slots(false) * slot_bytes(false) &&
                  gemm::PART_BYTES + 2 * REDO_FLOATS * sizeof(float) <= alone_slots(true) * slot_bytes(true),
              "the FMA tiles fit behind it");
template <typename T>
constexpr int piece_threads() { return (2 + PieceTraits<T>::SUM_WARPS) * 32; }

// warp 0 loads, warp 1 issues the products (of a pair: the first CTA's), the others add the accumulators up; all store.
template <typename T, int SLOTS, bool PAIR>
__global__ void __launch_bounds__(piece_threads<T>(), SLOTS == shared_slots(PAIR) ? 2 : 1)
    gemm_pieces_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                       const Params p, const Operand oa, const Operand ob, const int* __restrict__ outside_a,
                       const int* __restrict__ outside_b) {
  constexpr int PIECES = Traits<T>::PIECES, SUM_WARPS = PieceTraits<T>::SUM_WARPS;
  constexpr bool F32 = PIECES == 3;
  constexpr int COLS = TILE * 4 / SUM_WARPS, W = SUM_WARPS + 2, CTAS = PAIR ? 2 : 1, SLOT = slot_bytes(PAIR);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  PieceBarriers* bars = reinterpret_cast<PieceBarriers*>(smem + SLOTS * SLOT);
  volatile int* abort_word = &bars->abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool clustered = PAIR || p.split_k > 1;
  const int ctarank = clustered ? static_cast<int>(cluster_ctarank()) : 0;
  const int half = PAIR ? ctarank & 1 : 0, rank = ctarank / CTAS;  // CTA of the pair, K slice

  if (threadIdx.x == 0) {
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->acc_full[i], 1);
      mbar_init(&bars->acc_empty[i], CTAS * SUM_WARPS);  // (of a pair: the first CTA's is used)
    }
    bars->abort_word = 0;
    bars->outside = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(&bars->tmem_base, 2 * TILE);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(&bars->tmem_base, 2 * TILE);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // both CTAs' barriers exist before anything signals across the pair
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  grid_dep_wait();
  grid_dep_launch();

  int b, tm, tn;
  gemm::tile_coords(p, static_cast<int>(blockIdx.x) / (p.split_k * CTAS), b, tm, tn);
  const int m0 = tm * TILE * CTAS + half * TILE, n0 = tn * TILE;
  const int kb0 = static_cast<int>(static_cast<long long>(rank) * p.k_blocks / p.split_k);
  const int kb1 = static_cast<int>(static_cast<long long>(rank + 1) * p.k_blocks / p.split_k);
  const int blocks = kb1 - kb0;  // at least 1: the host never takes more slices than K blocks
  float* part = reinterpret_cast<float*>(smem);
  // a barrier of the pair's first CTA, of its second
  auto in_first = [&](uint64_t* bar) { return mapa_shared(smem_u32(bar), ctarank & ~1); };
  auto in_second = [&](uint64_t* bar) { return mapa_shared(smem_u32(bar), ctarank | 1); };

  if (warp == 0) {
    if (elect_one()) {
      uint32_t n = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1 && ok; ++kb)
        for (int piece = PIECES - 1; piece >= 0; --piece, ++n) {
          const uint32_t s = n % SLOTS;
          ok = mbar_wait(&bars->empty[s], ((n / SLOTS) & 1) ^ 1, abort_word, 151);
          if (!ok) break;
          uint8_t* sa = smem + s * SLOT;
          uint8_t* sb = sa + PIECE_BYTES;
          const int k0 = kb * BK;
          if constexpr (PAIR) {
            // the bytes of both CTAs land on the first one's barrier
            if (half == 0) mbar_arrive_expect_tx(&bars->full[s], 2 * SLOT);
            const uint32_t full = in_first(&bars->full[s]);
            if (p.a_mn) {
              tma_load_4d_pair(sa, &tmap_a, full, m0, k0, b, piece);
              tma_load_4d_pair(sa + 8192, &tmap_a, full, m0 + 64, k0, b, piece);
            } else {
              tma_load_4d_pair(sa, &tmap_a, full, k0, m0, b, piece);
            }
            if (p.b_mn) tma_load_4d_pair(sb, &tmap_b, full, n0 + half * 64, k0, b, piece);
            else tma_load_4d_pair(sb, &tmap_b, full, k0, n0 + half * 64, b, piece);
          } else {
            mbar_arrive_expect_tx(&bars->full[s], SLOT);
            if (p.a_mn) {
              tma_load_4d(sa, &tmap_a, &bars->full[s], m0, k0, b, piece);
              tma_load_4d(sa + 8192, &tmap_a, &bars->full[s], m0 + 64, k0, b, piece);
            } else {
              tma_load_4d(sa, &tmap_a, &bars->full[s], k0, m0, b, piece);
            }
            if (p.b_mn) {
              tma_load_4d(sb, &tmap_b, &bars->full[s], n0, k0, b, piece);
              tma_load_4d(sb + 8192, &tmap_b, &bars->full[s], n0 + 64, k0, b, piece);
            } else {
              tma_load_4d(sb, &tmap_b, &bars->full[s], k0, n0, b, piece);
            }
          }
        }
    }
  } else if (warp == 1) {
    if (half == 0 && elect_one()) {
      const uint32_t idesc = make_idesc_bf16(TILE * CTAS, TILE, p.a_mn, p.b_mn);
      const uint32_t a_lbo = p.a_mn ? 8192u : 16u, b_lbo = p.b_mn ? 8192u : 16u;
      const uint32_t a_kstep = p.a_mn ? 2048u : 32u, b_kstep = p.b_mn ? 2048u : 32u;
      const uint32_t base = smem_u32(smem);
      auto commit = [&](uint64_t* bar) {
        if (PAIR) {
          umma_commit_pair(in_first(bar));
          umma_commit_pair(in_second(bar));
        } else {
          umma_commit(bar);
        }
      };
      uint32_t n = 0;  // slots of a K block: n (the last pieces), n + 1, ...
      bool ok = true;
      for (int it = 0; it < blocks && ok; ++it, n += PIECES) {
        const int group = it / p.sum_blocks, acc = group & 1;
        const bool first = it == group * p.sum_blocks, last = it + 1 == blocks || it + 1 == (group + 1) * p.sum_blocks;
        if (first) ok = mbar_wait(&bars->acc_empty[acc], ((group >> 1) & 1) ^ 1, abort_word, 251);
        uint32_t at[PIECES];  // by piece
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
          const uint32_t s = (n + i) % SLOTS;
          at[PIECES - 1 - i] = base + s * SLOT;
          ok = ok && mbar_wait(&bars->full[s], ((n + i) / SLOTS) & 1, abort_word, 252);
        }
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem_base + acc * TILE;
        auto product = [&](int pa, int pb, bool fresh) {
          const uint32_t sa = at[pa], sb = at[pb] + PIECE_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t da = smem_desc_sw128(sa + k * a_kstep, a_lbo, 1024), db = smem_desc_sw128(sb + k * b_kstep, b_lbo, 1024);
            if (PAIR) umma_ss_pair(d, da, db, idesc, fresh && k == 0 ? 0u : 1u);
            else umma_ss(d, da, db, idesc, fresh && k == 0 ? 0u : 1u);
          }
        };
        auto release = [&](int piece) { commit(&bars->empty[(n + PIECES - 1 - piece) % SLOTS]); };
        if constexpr (F32) {  // the smallest products first
          product(2, 0, first);
          product(0, 2, false);
          release(2);
          product(1, 1, false);
          product(1, 0, false);
          product(0, 1, false);
          release(1);
          product(0, 0, false);
          release(0);
        } else {
          product(0, 0, first);
          release(0);
        }
        if (last) commit(&bars->acc_full[acc]);
      }
    }
  } else {
    const int quad = warp & 3, col0 = ((warp - 2) >> 2) * COLS;
    if (F32 && m0 < p.M) {
      int any = 0;
      const long long fa = (static_cast<long long>(b) * ((p.M + TILE - 1) / TILE) + m0 / TILE) * p.k_blocks;
      const long long fb = (static_cast<long long>(b) * p.num_n_tiles + tn) * p.k_blocks;
      for (int i = kb0 + static_cast<int>(threadIdx.x) - 64; i < kb1; i += SUM_WARPS * 32)
        any |= outside_a[fa + i] | outside_b[fb + i];
      if (any) bars->outside = 1;
    }
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + col0;
    const int groups = (blocks + p.sum_blocks - 1) / p.sum_blocks;
    float sum[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
    bool ok = true;
    for (int g = 0; g < groups; ++g) {
      const int acc = g & 1;
      ok = mbar_wait(&bars->acc_full[acc], (g >> 1) & 1, abort_word, 351);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < COLS; c += 16) {
        uint32_t r[16];
        tmem_ld16(t_row + acc * TILE + c, r);
        tmem_wait_ld(r);
#pragma unroll
        for (int j = 0; j < 16; ++j) sum[c + j] = g == 0 ? __uint_as_float(r[j]) : sum[c + j] + __uint_as_float(r[j]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(in_first(&bars->acc_empty[acc]));
        else mbar_arrive(&bars->acc_empty[acc]);
      }
    }
    // The last accumulator is complete: every slot has been read, the partial tile takes their place.
    if (ok) gemm::store_partial(part, quad * 32 + lane, col0, sum);
    if (F32) {
      float zero = 0.f;  // NaN once a sum that is not finite has been met
#pragma unroll
      for (int j = 0; j < COLS; ++j) zero = fmaf(sum[j], 0.f, zero);
      if (zero != 0.f) bars->outside = 1;
    }
  }
  __syncwarp();
  if (*abort_word != 0) {
    // Loads that may still be in flight land before shared memory is used again or released.
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  if (F32) {
    __syncthreads();
    if (bars->outside != 0)
      partial_by_fma(oa, ob, b, m0, n0, kb0 * BK, min(kb1 * BK, p.K), static_cast<int>(smem - smem_raw));
  }
  if (clustered) cluster_sync_all();
  else __syncthreads();
  if (m0 < p.M) {
    switch (p.split_k) {
      case 1: store_out<1, W, PAIR, 4>(p, part, rank, warp, b, m0, n0); break;
      case 2: store_out<2, W, PAIR, 4>(p, part, rank, warp, b, m0, n0); break;
      case 4: store_out<4, W, PAIR, 4>(p, part, rank, warp, b, m0, n0); break;
      default: store_out<PAIR ? 4 : 8, W, PAIR, 4>(p, part, rank, warp, b, m0, n0); break;
    }
  }
  __syncwarp();
  if (clustered) cluster_sync_all();  // the other slices have read this CTA's partial; the pair is done
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, 2 * TILE);
    else tmem_dealloc(tmem_base, 2 * TILE);
  }
  if (threadIdx.x == 0 && *abort_word != 0) atomicExch(p.status, *abort_word);
}

// The same in f64.
template <int N, int C>
__device__ __forceinline__ void fma_block(const double* ta, const double* tb, int tx, int ty, int left,
                                          double (&acc)[4][4 * C]) {
  static_assert(C == 1, "");
#pragma unroll
  for (int kk = 0; kk < FMA_K; ++kk) {
    if (kk % 4 == 0 && kk >= left) break;
    const double2* a2 = reinterpret_cast<const double2*>(ta + kk * (N + 4) + ty * 4);
    const double2* b2 = reinterpret_cast<const double2*>(tb + kk * (N + 4) + tx * 4);
    const double ar[4] = {a2[0].x, a2[0].y, a2[1].x, a2[1].y}, br[4] = {b2[0].x, b2[0].y, b2[1].x, b2[1].y};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fma(ar[i], br[j], acc[i][j]);
  }
}

// Products of a short K, one CTA per 64 x 64 tile: 4 x 4 sums a thread, stored as they stand.  Bound by launch,
// first loads and the store: no tensor memory, no staging of pieces, several CTAs per SM.  f32 products are
// summed in f64, where they are exact: the result carries one rounding (2.5e-8, 2-norm, against f64), where a
// chain of f32 FMAs has 4.0e-8 at K = 4 and 7.3e-8 at 16 and the pieces 4.7e-8 and 4.8e-8.  Products of bf16
// are exact in f32 and a chain of f32 adds has less error than the truncating tensor core (2.2e-8 against 2.5e-8
// at 16).
template <typename T> struct FmaSum { using type = float; };
template <> struct FmaSum<float> { using type = double; };
constexpr int FMA_TILE = 64, FMA_THREADS = 256, FMA_FLOATS = 2 * fma_tile<FMA_TILE>();
template <typename T>
__global__ void __launch_bounds__(FMA_THREADS) gemm_fma_kernel(const Params p, const Operand oa, const Operand ob) {
  using S = typename FmaSum<T>::type;
  __shared__ __align__(16) S tiles[2 * FMA_FLOATS];
  grid_dep_wait();
  grid_dep_launch();
  int b, tm, tn;
  gemm::tile_coords(p, static_cast<int>(blockIdx.x), b, tm, tn);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int row0 = tm * FMA_TILE + ty * 4, col = tn * FMA_TILE + tx * 4;
  FmaSource<T, S, FMA_TILE, FMA_THREADS> fa, fb;
  S acc[4][4] = {};
  fa.init(oa, b, tm * FMA_TILE, 0, p.K);
  fb.init(ob, b, tn * FMA_TILE, 0, p.K);
  fa.fetch();
  fb.fetch();
  // C is read ahead of the products: its latency, row after row, is longer than they are.
  float c[4][4] = {};
  if (p.c_mode != 0) {
    const bool vec = p.c_vec && col + 4 <= p.N;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (row0 + i >= p.M) continue;
      const long long at = b * p.c_batch + (row0 + i) * p.ldc + col;
      const float* cf = static_cast<const float*>(p.c) + at;
      const __nv_bfloat16* ch = static_cast<const __nv_bfloat16*>(p.c) + at;
      if (vec && p.c_mode == 2) {
        const float4 q = *reinterpret_cast<const float4*>(cf);
        c[i][0] = q.x; c[i][1] = q.y; c[i][2] = q.z; c[i][3] = q.w;
      } else if (vec) {
        const uint2 q = *reinterpret_cast<const uint2*>(ch);
        c[i][0] = bf16_lo(q.x); c[i][1] = bf16_hi(q.x); c[i][2] = bf16_lo(q.y); c[i][3] = bf16_hi(q.y);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (col + j < p.N) c[i][j] = p.c_mode == 2 ? cf[j] : __bfloat162float(ch[j]);
      }
    }
  }
  int buf = 0;
  for (int k0 = 0; k0 < p.K; k0 += FMA_K, buf ^= 1) {
    S* ta = tiles + buf * FMA_FLOATS;
    S* tb = ta + fma_tile<FMA_TILE>();
    fa.store(ta);
    fb.store(tb);
    if (k0 + FMA_K < p.K) {
      fa.fetch();
      fb.fetch();
    }
    __syncthreads();  // the other buffer has been read by all who are here
    fma_block<FMA_TILE, 1>(ta, tb, tx, ty, p.K - k0, acc);
  }
  const bool vec = p.d_vec && col + 4 <= p.N;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (row0 + i >= p.M) continue;
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = p.c_mode != 0 ? p.alpha * static_cast<float>(acc[i][j]) + p.beta * c[i][j] : p.alpha * static_cast<float>(acc[i][j]);
    const long long at = b * p.d_batch + (row0 + i) * p.ldd + col;
    float* df = static_cast<float*>(p.d) + at;
    __nv_bfloat16* dh = static_cast<__nv_bfloat16*>(p.d) + at;
    if (vec && p.out_f32) {
      *reinterpret_cast<float4*>(df) = make_float4(v[0], v[1], v[2], v[3]);
    } else if (vec) {
      *reinterpret_cast<uint2*>(dh) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (col + j < p.N) {
          if (p.out_f32) df[j] = v[j];
          else dh[j] = __float2bfloat16_rn(v[j]);
        }
    }
  }
}

// Whether the FMAs are done before the tensor-core kernel is: it takes 7.7 to 9 us (bf16 5.6 to 7.5) before K counts,
// the FMAs 2.7 and, per 16 of K and tile of an SM, 1.3 (bf16 0.7).  In microseconds, tensor cores -> FMAs: f32
// 1500 x 4 x 1027 10.1 -> 7.1, 2048 x 16 x 2048 19.2 -> 15.6, 4096 x 1 x 4096 64 -> 31, 64 x 48 x 64 8.0 -> 7.6; the
// other way at 64 x 64 x 8192, 8.7 against 9.3, and 2048 x 24 x 2048, 19.2 against 25.5.  bf16 1500 x 17 x 1027
// 8.0 -> 7.0, 4096 x 9 x 4097 54.6 -> 32.2, 300 x 49 x 301 7.6 -> 6.5; the other way at 2048 x 25 x 2049, 14.8
// against 16.7, and 1024 x 33 x 1025, 7.6 against 8.9.
static bool short_k(const Params& p, bool f32) {
  const int steps = (p.K + FMA_K - 1) / FMA_K;
  const long long tiles = static_cast<long long>(p.batch) * ((p.M + FMA_TILE - 1) / FMA_TILE) * ((p.N + FMA_TILE - 1) / FMA_TILE);
  const long long waves = (tiles + sm_count() - 1) / sm_count();
  return steps == 1 || steps * waves <= (f32 ? 3 : 4) || (!f32 && steps == 2 && (waves <= 4 || p.out_f32));
}
template <typename T>
static int32_t launch_fma(Params& p, const Operand& oa, const Operand& ob, cudaStream_t stream) {
  p.num_m_tiles = (p.M + FMA_TILE - 1) / FMA_TILE;
  p.num_n_tiles = (p.N + FMA_TILE - 1) / FMA_TILE;
  p.num_tiles = p.batch * p.num_m_tiles * p.num_n_tiles;
  CDL_CUDA(launch_pdl(gemm_fma_kernel<T>, dim3(static_cast<unsigned>(p.num_tiles)), dim3(FMA_THREADS), 0, stream, p, oa, ob));
  return CDL_OK;
}

// K slices per tile: the number whose waves of resident CTAs end first.  A CTA's time is its K blocks
// and a part that does not shrink (set-up, first loads, the exchange of the partial sums, stores).
// f32 300 x 2048 x 130 with 1, 2, 4, 8 slices: 69, 39, 24, 17 us; 1024 x 2048 x 1536 74, 81, 76, 121 us.
static int choose_splits(long long tiles, int k_blocks, int slots, double fixed) {
  int best = 1;
  double best_cost = 1e30;
  for (int s = 1; s <= gemm::MAX_SPLITS && s <= k_blocks; s *= 2) {
    const long long waves = (tiles * s + slots - 1) / slots;
    const double cost = static_cast<double>(waves) * (static_cast<double>((k_blocks + s - 1) / s) + fixed);
    if (cost < best_cost * 0.97) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}

// The two tensor-core paths in microseconds, fitted to 200 products (M 16 .. 4100, K 64 .. 4099, odd and even rows, forward and
// weight-gradient layouts) timed on both and with every K slicing: a wave's cost is a CTA's set-up and stores, its K
// blocks and the exchange of the slices' sums.  The root mean square of what the fits miss is 8 to 16 %.
// Waves are counted in clusters: with one CTA per SM 74 clusters of two fit on 148 SMs, 33 of four and 14 of
// eight (an SM of a group that cannot take a whole one stays empty).
static long long cluster_slots(int ctas) {
  const long long sms = sm_count();
  return std::max(1LL, ctas == 1 ? sms : ctas == 2 ? sms / 2 : ctas == 4 ? sms * 33 / 148 : sms * 14 / 148);
}
static double general_us(bool f32, long long batch, long long M, long long N, int k_blocks, int odd_operands) {
  const long long tiles = batch * ((M + TILE - 1) / TILE) * ((N + TILE - 1) / TILE);
  const int s = choose_splits(tiles, k_blocks, sm_count(), f32 ? 4.0 : 6.0);
  const long long waves = (tiles + cluster_slots(s) - 1) / cluster_slots(s);
  const double blocks = (k_blocks + s - 1) / s;
  // (the loaders bring in only the rows and columns that exist)
  const double fill = static_cast<double>(std::min<long long>(M, TILE) * std::min<long long>(N, TILE)) / (TILE * TILE);
  return f32 ? 2.5 + waves * (5.4 + (s > 1 ? 1.2 : 0.0) + (s > 2 ? 3.4 : 0.0) + blocks * (0.40 + 1.45 * fill + 0.18 * odd_operands))
             : 1.7 + waves * (5.5 + (s > 1 ? 0.7 : 0.0) + (s > 2 ? 3.1 : 0.0) + blocks * (0.95 * fill + 0.12 * odd_operands));
}
static double pieces_us(bool f32, bool pair, long long tiles, int k_blocks, int s, double laid_elements) {
  const int ctas = s * (pair ? 2 : 1);
  const long long slots = cluster_slots(ctas);
  const double waves = (tiles + slots - 1) / slots, blocks = waves * ((k_blocks + s - 1) / s);
  const double lay = laid_elements * 1e-6, split = s > 1, four = s > 1 && ctas >= 4, eight = ctas >= 8;
  if (f32) return 2.4 + 1.81 * lay + blocks * (pair ? 0.81 : 1.08) + waves * (8.5 - 0.2 * split + 1.2 * four + 1.7 * eight);
  // two CTAs fit on an SM: they share the tensor core, not the set-up
  const long long two = tiles * ctas > sm_count() ? 2 * slots : slots;
  const double sets = (tiles + two - 1) / two;
  return 1.3 + 0.87 * lay + blocks * (pair ? 0.29 : 0.19) + sets * (8.2 - 1.1 * split + 1.2 * four + 0.3 * eight);
}
static int choose_piece_splits(bool f32, bool pair, long long tiles, int k_blocks) {
  int best = 1;
  for (int s = 2; s * (pair ? 2 : 1) <= gemm::MAX_SPLITS && s <= k_blocks; s *= 2)
    if (pieces_us(f32, pair, tiles, k_blocks, s, 0) < pieces_us(f32, pair, tiles, k_blocks, best, 0)) best = s;
  return best;
}

template <typename T, bool FINE>
static int32_t launch(Params& p, const Operand& oa, const Operand& ob, double fixed, cudaStream_t stream) {
  using Tr = Traits<T>;
  static std::once_flag once[64];
  int dev = 0;
  CDL_CUDA(cudaGetDevice(&dev));
  cudaError_t err = cudaSuccess;
  std::call_once(once[dev & 63], [&] {
    err = cudaFuncSetAttribute(gemm_general_kernel<T, FINE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(smem_bytes<T>()));
  });
  if (err != cudaSuccess) return fail(CDL_ERR_CUDA, "cudaFuncSetAttribute failed: %s", cudaGetErrorString(err));
  p.split_k = choose_splits(p.num_tiles, p.k_blocks, sm_count(), fixed);
  CDL_CUDA(launch_pdl_cluster(gemm_general_kernel<T, FINE>, dim3(static_cast<unsigned>(p.num_tiles) * p.split_k),
                              dim3(THREADS), smem_bytes<T>(), p.split_k, stream, p, oa, ob));
  return CDL_OK;
}

// What gemm_pieces_kernel needs in scratch, in this order: the pieces of A, of B (f32 always, bf16 where TMA cannot read
// the operand where it is), and for f32 the two lists of blocks with values that have no pieces.
struct PiecePlan {
  bool lay_a, lay_b;
  int pitch_a, pitch_b;
  long long piece_a, piece_b;  // elements of one piece
  size_t off_b, off_flags_a, off_flags_b, bytes;
};
static bool tma_can_read(const Operand& o, long long batch, int outer, int inner) {
  const long long s_in = o.mn_major ? o.s_mn : o.s_k, s_out = o.mn_major ? o.s_k : o.s_mn;
  return (inner == 1 || s_in == 1) && (outer == 1 || (s_out % 8 == 0 && s_out >= inner)) &&
         (batch == 1 || (o.s_batch > 0 && o.s_batch % 8 == 0)) && reinterpret_cast<uintptr_t>(o.ptr) % 16 == 0;
}
static PiecePlan plan_pieces(const Operand& oa, const Operand& ob, long long batch, int K, bool f32) {
  PiecePlan q{};
  auto up = [](long long a, long long b) { return (a + b - 1) / b * b; };
  const int pieces = f32 ? 3 : 1;
  size_t at = 0;
  for (int i = 0; i < 2; ++i) {
    const Operand& o = i ? ob : oa;
    const int outer = o.mn_major ? K : o.mn, inner = o.mn_major ? o.mn : K;
    const bool lay = f32 || !tma_can_read(o, batch, outer, inner);
    const long long pitch = up(inner, 8), piece = batch * outer * pitch;
    (i ? q.lay_b : q.lay_a) = lay;
    (i ? q.pitch_b : q.pitch_a) = static_cast<int>(pitch);
    (i ? q.piece_b : q.piece_a) = piece;
    if (i) q.off_b = at;
    if (lay) at += up(2 * pieces * piece, 256);
  }
  if (f32) {
    const long long kb = (K + BK - 1) / BK;
    q.off_flags_a = at;
    at += up(4 * batch * ((oa.mn + TILE - 1) / TILE) * kb, 256);
    q.off_flags_b = at;
    at += up(4 * batch * ((ob.mn + TILE - 1) / TILE) * kb, 256);
  }
  q.bytes = at;
  return q;
}

template <typename T, int SLOTS, bool PAIR>
static int32_t launch_pieces_kernel(const Params& p, const CUtensorMap& ta, const CUtensorMap& tb, const Operand& oa,
                                    const Operand& ob, const int* fa, const int* fb, cudaStream_t stream) {
  static std::once_flag once[64];
  int dev = 0;
  CDL_CUDA(cudaGetDevice(&dev));
  cudaError_t err = cudaSuccess;
  std::call_once(once[dev & 63], [&] {
    err = cudaFuncSetAttribute(gemm_pieces_kernel<T, SLOTS, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(piece_smem_bytes(SLOTS, PAIR)));
  });
  if (err != cudaSuccess) return fail(CDL_ERR_CUDA, "cudaFuncSetAttribute failed: %s", cudaGetErrorString(err));
  const int cluster = p.split_k * (PAIR ? 2 : 1);
  CDL_CUDA(launch_pdl_cluster(gemm_pieces_kernel<T, SLOTS, PAIR>, dim3(static_cast<unsigned>(p.num_tiles) * cluster),
                              dim3(piece_threads<T>()), piece_smem_bytes(SLOTS, PAIR), cluster, stream, ta, tb, p, oa, ob,
                              fa, fb));
  return CDL_OK;
}

template <typename T>
static int32_t launch_pieces(Params& p, const Operand& oa, const Operand& ob, const PiecePlan& q, char* scratch,
                             cudaStream_t stream) {
  constexpr bool F32 = Traits<T>::PIECES == 3;
  const bool pair = p.M > TILE;
  CUtensorMap maps[2];
  Layout lay[2] = {};
  int blocks[2] = {0, 0};
  for (int i = 0; i < 2; ++i) {
    const Operand& o = i ? ob : oa;
    const int outer = o.mn_major ? p.K : o.mn, inner = o.mn_major ? o.mn : p.K;
    const bool laid = i ? q.lay_b : q.lay_a;
    const long long s_in = o.mn_major ? o.s_mn : o.s_k, s_out = o.mn_major ? o.s_k : o.s_mn;
    const int pitch = i ? q.pitch_b : q.pitch_a;
    const long long piece = i ? q.piece_b : q.piece_a;
    const void* base = laid ? scratch + (i ? q.off_b : 0) : o.ptr;
    const long long ld = laid ? pitch : outer > 1 ? s_out : pitch, sb = laid || p.batch == 1 ? outer * ld : o.s_batch;
    const uint64_t dims[4] = {static_cast<uint64_t>(inner), static_cast<uint64_t>(outer), static_cast<uint64_t>(p.batch),
                              F32 ? 3u : 1u};
    const uint64_t strides[4] = {0, 2 * static_cast<uint64_t>(ld), 2 * static_cast<uint64_t>(sb),
                                 2 * static_cast<uint64_t>(laid ? piece : sb * p.batch)};
    const uint32_t box[4] = {64, static_cast<uint32_t>(o.mn_major || (i == 1 && pair) ? 64 : TILE), 1, 1};
    CDL_CHECK(encode_tmap(&maps[i], base, CDL_BF16, 4, dims, strides, box, true));
    if (laid) {
      Layout& l = lay[i];
      l = {o.ptr, o.s_batch, s_out, s_in, static_cast<__nv_bfloat16*>(const_cast<void*>(base)), piece, outer, inner, pitch,
           o.mn_major, (o.mn + TILE - 1) / TILE, p.k_blocks,
           reinterpret_cast<int*>(scratch + (i ? q.off_flags_b : q.off_flags_a))};
      blocks[i] = p.batch * l.mn_tiles * l.k_blocks;
    }
  }
  p.a_mn = oa.mn_major;
  p.b_mn = ob.mn_major;
  if (blocks[0] + blocks[1] > 0)
    CDL_CUDA(launch_pdl(lay_out_kernel<T>, dim3(static_cast<unsigned>(blocks[0] + blocks[1])), dim3(LAY_THREADS), 0,
                        stream, lay[0], lay[1], blocks[0]));
  const int* fa = reinterpret_cast<const int*>(scratch + q.off_flags_a);
  const int* fb = reinterpret_cast<const int*>(scratch + q.off_flags_b);
  auto run = [&](auto is_pair) {
    constexpr bool PAIR = decltype(is_pair)::value;
    constexpr int CTAS = PAIR ? 2 : 1;
    p.num_m_tiles = (p.M + TILE * CTAS - 1) / (TILE * CTAS);
    p.num_tiles = p.batch * p.num_m_tiles * p.num_n_tiles;
    p.split_k = choose_piece_splits(F32, PAIR, p.num_tiles, p.k_blocks);
    if (!F32 && static_cast<long long>(p.num_tiles) * p.split_k * CTAS > sm_count())
      return launch_pieces_kernel<__nv_bfloat16, shared_slots(PAIR), PAIR>(p, maps[0], maps[1], oa, ob, fa, fb, stream);
    return launch_pieces_kernel<T, alone_slots(PAIR), PAIR>(p, maps[0], maps[1], oa, ob, fa, fb, stream);
  };
  return pair ? run(std::true_type{}) : run(std::false_type{});
}

// Whether the operands are laid out first: where that is estimated to be faster by a tenth, about what the estimates
// miss, and the other kernel takes long enough to hide the host's part: asking for the scratch, allocating it, a second
// launch and two tensor maps cost an eager caller 7 us on top of the 11 of a call (three products of 529 x 2049 x 451, none
// above 22 us: 51 us, all laid out 55).  General kernel -> laid out first, us; f32: 16 x 1027 x 2051 29.9 -> 21.1,
// 512 x 2051 x 1027 62 -> 32, 2047 x 2047 x 2047 152 -> 92; the other way 2049 x 64 x 2049 19.8 and 30.5,
// 512 x 1027 x 2051 29.0 and 30.4, 16 x 515 x 515 13.0 and 13.5.  bf16: 64 x 2049 x 2049 33.9 -> 15.2, 2047 x 2047 x 4095
// 167 -> 53; the other way 1500 x 300 x 900 11.6 and 11.7, 250 x 129 x 131 9.7 and 9.9.  Of 90 random shapes (M 8 .. 8192, K and
// N 64 .. 4096) those that it takes run f32 1.3 and bf16 1.8 times as fast on average.
static bool worth_laying_out(const Operand& oa, const Operand& ob, const PiecePlan& plan, long long batch, long long K, bool f32,
                             bool fine) {
  const long long M = oa.mn, N = ob.mn, kb = (K + BK - 1) / BK;
  const long long blocks = batch * ((M + TILE - 1) / TILE + (N + TILE - 1) / TILE) * kb;
  if (fine || blocks > INT32_MAX) return false;
  const bool pair = M > TILE;
  const long long m_tile = pair ? 2 * TILE : TILE, tiles = batch * ((M + m_tile - 1) / m_tile) * ((N + TILE - 1) / TILE);
  const int s = choose_piece_splits(f32, pair, tiles, static_cast<int>(kb));
  const double laid = (plan.lay_a ? 1.0 * M : 0.0) + (plan.lay_b ? 1.0 * N : 0.0);
  const double other = general_us(f32, batch, M, N, static_cast<int>(kb), !oa.pairs + !ob.pairs);
  return other > 18.0 && pieces_us(f32, pair, tiles, static_cast<int>(kb), s, laid * K * batch) < 0.9 * other;
}

}  // namespace gemm_general

static gemm_general::Operand general_operand(const cdl_tensor* t, int mn_dim, int k_dim) {
  gemm_general::Operand o{};
  o.ptr = t->ptr;
  o.mn = static_cast<int>(t->shape[mn_dim]);
  o.s_batch = t->rank == 3 ? t->stride[0] : 0;
  // an extent of 1 has no meaningful stride
  o.s_mn = t->shape[mn_dim] > 1 ? t->stride[mn_dim] : 0;
  o.s_k = t->shape[k_dim] > 1 ? t->stride[k_dim] : 0;
  o.mn_major = o.s_k != 1 && o.s_mn == 1;
  const long long inner = o.mn_major ? o.s_mn : o.s_k, outer = o.mn_major ? o.s_k : o.s_mn;
  o.pairs = inner == 1 && outer % 2 == 0 && o.s_batch % 2 == 0 &&
            reinterpret_cast<uintptr_t>(t->ptr) % (2 * dtype_size(t->dtype)) == 0;
  return o;
}

size_t matmul_general_scratch_bytes(const cdl_tensor* a, const cdl_tensor* b, const cdl_tensor* d) {
  using namespace gemm_general;
  const int r = a->rank;
  const long long batch = r == 3 ? a->shape[0] : 1;
  const long long M = a->shape[r - 2], K = a->shape[r - 1], N = b->shape[r - 1];
  const bool f32 = a->dtype == CDL_F32;
  if (batch <= 0 || M <= 0 || N <= 0 || K <= 0 || batch > 65535 || M > INT32_MAX || N > INT32_MAX || K > INT32_MAX)
    return 0;
  Params p{};
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.K = static_cast<int>(K);
  p.batch = static_cast<int>(batch);
  p.out_f32 = d->dtype == CDL_F32;
  if (short_k(p, f32)) return 0;
  const Operand oa = general_operand(a, r - 2, r - 1), ob = general_operand(b, r - 1, r - 2);
  const PiecePlan plan = plan_pieces(oa, ob, batch, p.K, f32);
  return worth_laying_out(oa, ob, plan, batch, K, f32, !f32 && p.out_f32 && K <= 100) ? plan.bytes : 0;
}

// Operands as validated by matmul_execute_epi (ranks, shapes, dtypes of one kind, contiguous last
// dimension of C and D); nothing here depends on alignment.
int32_t matmul_general_execute(const cdl_tensor* a, const cdl_tensor* b, const cdl_tensor* c,
                               const cdl_tensor* d, float alpha, float beta, void* scratch, size_t scratch_bytes,
                               cudaStream_t stream) {
  using namespace gemm_general;
  const int r = a->rank;
  const long long batch = r == 3 ? a->shape[0] : 1;
  const long long M = a->shape[r - 2], K = a->shape[r - 1], N = b->shape[r - 1];
  if (M > 65535LL * 64)
    return fail(CDL_ERR_UNSUPPORTED, "matmul (general path): more than %d rows", 65535 * 64);
  const Operand oa = general_operand(a, r - 2, r - 1), ob = general_operand(b, r - 1, r - 2);
  Params p{};
  p.M = static_cast<int>(M);
  p.N = static_cast<int>(N);
  p.K = static_cast<int>(K);
  p.batch = static_cast<int>(batch);
  p.num_m_tiles = static_cast<int>((M + TILE - 1) / TILE);
  p.num_n_tiles = static_cast<int>((N + TILE - 1) / TILE);
  const long long tiles = batch * p.num_m_tiles * p.num_n_tiles;
  if (tiles > INT32_MAX / gemm::MAX_SPLITS) return fail(CDL_ERR_UNSUPPORTED, "matmul: too many tiles");
  p.num_tiles = static_cast<int>(tiles);
  p.k_blocks = static_cast<int>((K + BK - 1) / BK);
  p.raster_w = gemm::RASTER_W;
  p.d = d->ptr;
  p.ldd = M > 1 ? d->stride[r - 2] : N;
  p.d_batch = r == 3 ? d->stride[0] : 0;
  p.out_f32 = d->dtype == CDL_F32 ? 1 : 0;
  auto vec_ok = [](const void* ptr, long long ld, long long bstride, size_t es) {
    return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && (ld * es) % 16 == 0 && (bstride * es) % 16 == 0;
  };
  p.d_vec = vec_ok(p.d, p.ldd, p.d_batch, dtype_size(d->dtype));
  if (c != nullptr && beta != 0.0f) {
    p.c = c->ptr;
    p.ldc = M > 1 ? c->stride[r - 2] : N;
    p.c_batch = r == 3 ? c->stride[0] : 0;
    p.c_mode = c->dtype == CDL_F32 ? 2 : 1;
    p.c_vec = vec_ok(p.c, p.ldc, p.c_batch, dtype_size(c->dtype));
    p.beta = beta;
  }
  p.alpha = alpha;
  p.status = device_status_ptr();
  if (!p.status) return fail(CDL_ERR_CUDA, "cannot resolve the device status word");
  // A tensor-core accumulator truncates: the sum of n steps of 16 bf16 products lies about 1.6e-8 n below its value
  // (2-norm, against f64: 3.8e-8 after two steps, 6.5e-8 after four, 4.7e-7 after 32), where a chain of K f32
  // additions has 7.3e-9 sqrt(K).  So much of K goes into one accumulator that its error stays below the
  // chain's; accumulators are added with round-to-nearest.  f32 results: half a K block up to K = 100 (4.7e-8 at
  // K = 64, chain 5.1e-8), else one (1.3e-7 at 2051, chain 3.9e-7).  bf16 results, rounded to 2^-9, take
  // 0.11 sqrt(K) blocks (2.4e-7 at 2051 before that rounding).
  const bool f32 = a->dtype == CDL_F32, out_f32 = d->dtype == CDL_F32, fine = !f32 && out_f32 && K <= 100;
  p.sum_blocks = f32 || out_f32 ? 1 : std::clamp(static_cast<int>(0.11 * sqrt(static_cast<double>(K))), 1, 8);
  ProfileScope ps(PROF_GEMM, 2.0 * batch * M * N * K, stream);
  if (short_k(p, f32)) return f32 ? launch_fma<float>(p, oa, ob, stream) : launch_fma<__nv_bfloat16>(p, oa, ob, stream);
  if (scratch != nullptr && reinterpret_cast<uintptr_t>(scratch) % 16 == 0) {
    const PiecePlan plan = plan_pieces(oa, ob, batch, p.K, f32);
    if (scratch_bytes >= plan.bytes && worth_laying_out(oa, ob, plan, batch, K, f32, fine))
      return f32 ? launch_pieces<float>(p, oa, ob, plan, static_cast<char*>(scratch), stream)
                 : launch_pieces<__nv_bfloat16>(p, oa, ob, plan, static_cast<char*>(scratch), stream);
  }
  if (f32) return launch<float, false>(p, oa, ob, 4.0, stream);
  return fine ? launch<__nv_bfloat16, true>(p, oa, ob, 6.0, stream)
              : launch<__nv_bfloat16, false>(p, oa, ob, 6.0, stream);
}

}  // namespace cdl
