// BF16 GEMM for problems that leave the 256 x 256 tiles of gemm.cu short of work: few rows (decoding,
// short sequences, small microbatches) or a small output.  Same operands and epilogues, 128 x 128
// tiles, and each tile's K range shared by a cluster of 1, 2, 4 or 8 CTAs whose partial sums meet in
// distributed shared memory (gemm_rows.cuh).
//
// What bounds these problems is the weights' way from HBM: a [2048, 5632] matrix is 23 MB, 3.5 us at
// the copy bandwidth, but only if every SM keeps loads in flight; 64 rows against it are 22 tiles of
// 128 x 256.  So the split is chosen for the number of SMs that load (choose_cluster_splits in gemm.cu),
// two CTAs can share an SM (or one has twice the operand stages), and K slices meet on chip: no scratch
// memory, no second launch, a fixed order of the sums.  The weight-gradient form adds each finished sum to D
// once, by a reduction at the L2; no other form uses atomics.
#include "gemm_rows.cuh"
#include "host.h"
#include "ops.h"
#include "ptx.cuh"

#include <mutex>

namespace cdl {
namespace gemm {
namespace {

constexpr int TILE_M = 128, TILE_N = CLUSTER_TILE_N, BK = 64;
constexpr int A_BYTES = TILE_M * BK * 2, B_BYTES = TILE_N * BK * 2;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
// Eight warps, all of which drain the accumulator and store; before that one lane of warp 0 issues the
// loads and one of warp 1 the MMAs.  Two CTAs per SM leave 128 registers a thread.
constexpr int WARPS = 8, THREADS = WARPS * 32;
constexpr int TMEM_COLS = 128;
// Operand stages: 3 where two CTAs share an SM, 6 where every CTA has an SM to itself; either way an SM
// keeps 192 KiB of loads in flight.
constexpr int SHARED_STAGES = 3, ALONE_STAGES = 6;
constexpr size_t smem_bytes(int stages) { return 1024 + stages * STAGE_BYTES + 128; }
static_assert(PART_BYTES <= SHARED_STAGES * STAGE_BYTES, "the partial tile takes the place of the operand stages");

struct Barriers {
  uint64_t full[ALONE_STAGES];
  uint64_t empty[ALONE_STAGES];
  uint64_t acc_full;
  uint32_t tmem_base;
  int abort_word;
};
static_assert(sizeof(Barriers) <= 128, "barriers fit behind the stages");

template <int S, int STAGES>
__global__ void __launch_bounds__(THREADS, STAGES == SHARED_STAGES ? 2 : 1)
    gemm_cluster_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                        const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  Barriers* bars = reinterpret_cast<Barriers*>(smem + STAGES * STAGE_BYTES);
  volatile int* abort_word = &bars->abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    mbar_init(&bars->acc_full, 1);
    bars->abort_word = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  // One (tile, K slice) per CTA; the slices of a tile are one cluster.
  const int rank = S > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  int b, tm, tn;
  tile_coords(p, static_cast<int>(blockIdx.x) / S, b, tm, tn);
  const int m0 = tm * TILE_M, n0 = tn * TILE_N;
  const int kb0 = static_cast<int>(static_cast<long long>(rank) * p.k_blocks / S);
  const int kb1 = static_cast<int>(static_cast<long long>(rank + 1) * p.k_blocks / S);
  // B is the weights: on their way from HBM to the L2 while the kernel ahead still runs (three products of 64 rows 43.9 ->
  // 42.5 us; in the CTA-pair kernel, whose CTAs find an SM only when that kernel ends, the same gave nothing).
  if (warp == 2 && tm == 0 && !p.atomic_out) {
    if (elect_one()) {
      for (int kb = kb0; kb < kb1 && kb < kb0 + STAGES; ++kb) {
        if (p.b_mn) {
#pragma unroll
          for (int i = 0; i < TILE_N / 64; ++i) tma_prefetch_3d(&tmap_b, n0 + i * 64, kb * BK, b);
        } else {
          tma_prefetch_3d(&tmap_b, kb * BK, n0, b);
        }
      }
    }
    __syncwarp();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  if (!p.early) grid_dep_wait();  // the set-up above overlaps the previous kernel's tail
  grid_dep_launch();

  float* part = reinterpret_cast<float*>(smem);
  TileOut<S, WARPS> tile_out;

  if (warp == 0) {
    if (elect_one()) {
      for (int kb = kb0; kb < kb1; ++kb) {
        const int it = kb - kb0, s = it % STAGES;
        if (!mbar_wait(&bars->empty[s], ((it / STAGES) & 1) ^ 1, abort_word, 121)) break;
        uint8_t* sa = smem + s * STAGE_BYTES;
        uint8_t* sb = sa + A_BYTES;
        mbar_arrive_expect_tx(&bars->full[s], STAGE_BYTES);
        const int k0 = kb * BK;
        if (p.a_mn) {
#pragma unroll
          for (int i = 0; i < TILE_M / 64; ++i)
            tma_load_3d(sa + i * 8192, &tmap_a, &bars->full[s], m0 + i * 64, k0, b);
        } else {
          tma_load_3d(sa, &tmap_a, &bars->full[s], k0, m0, b);
        }
        if (p.b_mn) {
#pragma unroll
          for (int i = 0; i < TILE_N / 64; ++i)
            tma_load_3d(sb + i * 8192, &tmap_b, &bars->full[s], n0 + i * 64, k0, b);
        } else {
          tma_load_3d(sb, &tmap_b, &bars->full[s], k0, n0, b);
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(TILE_M, TILE_N, p.a_mn, p.b_mn);
      const uint32_t a_lbo = p.a_mn ? 8192u : 16u, b_lbo = p.b_mn ? 8192u : 16u;
      const uint32_t a_kstep = p.a_mn ? 2048u : 32u, b_kstep = p.b_mn ? 2048u : 32u;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        const int it = kb - kb0, s = it % STAGES;
        if (!mbar_wait(&bars->full[s], (it / STAGES) & 1, abort_word, 221)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + s * STAGE_BYTES), sb = sa + A_BYTES;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          umma_ss(tmem_base, smem_desc_sw128(sa + k * a_kstep, a_lbo, 1024),
                  smem_desc_sw128(sb + k * b_kstep, b_lbo, 1024), idesc, (it | k) != 0 ? 1u : 0u);
        umma_commit(&bars->empty[s]);
      }
      if (ok) umma_commit(&bars->acc_full);
    }
  }
  __syncwarp();
  tile_out.prefetch(p, rank, warp, b, m0, n0);
  {
    // After this wait every product is done and the operand stages are free: the partial tile goes there.
    const bool ok = mbar_wait(&bars->acc_full, 0, abort_word, 321);
    tc_fence_after();
    const int row = (warp & 3) * 32 + lane, half = warp >> 2;
    if (ok && m0 + (warp & 3) * 32 < p.M) {
#pragma unroll
      for (int c = half * 64; c < half * 64 + 64; c += 16) {
        uint32_t r[16];
        tmem_ld16(tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + c, r);
        tmem_wait_ld(r);
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
        store_partial(part, row, c, v);
      }
    }
    tc_fence_before();
  }
  __syncwarp();
  if (*abort_word != 0) {
    // Loads that may still be in flight land before shared memory is used again or released.
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  if (S > 1) cluster_sync_all();
  else __syncthreads();
  tile_out.finish(p, part, rank, warp, b, m0, n0);
  __syncwarp();
  if (S > 1) cluster_sync_all();  // the other slices have read this CTA's partial
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (threadIdx.x == 0 && *abort_word != 0) atomicExch(p.status, *abort_word);
  if (p.early) grid_dep_wait();
}

// The unsplit weight-gradient form (D += A^T B, f32): many tiles with few K blocks each, so that launch,
// set-up, first loads and the store are most of a CTA's life.  One CTA per SM walks the tiles; loads and
// products of the next tile run under the store of this one (two accumulators, the partial tile in
// shared memory of its own).  Two tiles are a CTA's own, every further one is drawn from a counter, so a CTA
// that finds its SM late (another kernel, e.g. a collective, holds it) takes fewer tiles instead of holding a
// fixed share back to the end: 2048 x 6144 with K = 128 beside a kernel on 32 SMs 28.0 us, with fixed shares 32.5
// (alone 18.7 and 18.6; 8192 x 8192, K = 64, alone 106 and 112).  2048 x 5632 from HBM with K = 64, 256, 512: 22.7,
// 25.0, 30.7 us; as one short-lived CTA per tile 25.8, 28.9, 34.1 us.  What is left is the reductions: 92 MB of HBM traffic, 14 us.
constexpr int WALK_THREADS = 320;  // warp 0 TMA, warp 1 MMA, warps 2-9 drain and store
constexpr int WALK_TMEM_COLS = 256;
// The producer publishes the tile of step t in slot t % WALK_SLOTS, once the accumulator that step t uses is free.
// So no CTA holds more than two tiles that it has not begun to store, and the slot has been read by all warps.
// It also works out the coordinates: the two divisions would stand between a store warp's tiles (0.2 us each).
constexpr int WALK_SLOTS = 4, WALK_BARRIER_BYTES = 256;
constexpr size_t WALK_SMEM_BYTES = 1024 + SHARED_STAGES * STAGE_BYTES + PART_BYTES + WALK_BARRIER_BYTES;
struct WalkBarriers {
  uint64_t full[SHARED_STAGES];
  uint64_t empty[SHARED_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t tile_full[WALK_SLOTS];
  int4 tile_ring[WALK_SLOTS];  // batch (-1: no tile is left), first row, first column
  uint32_t tmem_base;
  int abort_word;
};
static_assert(sizeof(WalkBarriers) <= WALK_BARRIER_BYTES, "barriers fit behind the partial tile");
__device__ __forceinline__ void store_warps_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
// The same; true in all 256 threads if `flag` is in any.
__device__ __forceinline__ bool store_warps_any(bool flag) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(any)
      : "r"(static_cast<uint32_t>(flag))
      : "memory");
  return any != 0;
}

__global__ void __launch_bounds__(WALK_THREADS, 1)
    gemm_cluster_walk_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                             const Params p) {
  constexpr int STAGES = SHARED_STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  float* part = reinterpret_cast<float*>(smem + STAGES * STAGE_BYTES);
  WalkBarriers* bars = reinterpret_cast<WalkBarriers*>(smem + STAGES * STAGE_BYTES + PART_BYTES);
  volatile int* abort_word = &bars->abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->acc_full[i], 1);
      mbar_init(&bars->acc_empty[i], WARPS);
    }
    for (int i = 0; i < WALK_SLOTS; ++i) mbar_init(&bars->tile_full[i], 1);
    bars->abort_word = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, WALK_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  if (!p.early) grid_dep_wait();
  grid_dep_launch();

  if (warp == 0) {
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      // Every CTA draws after its second tile and each further one, until a draw runs past the last tile; the
      // launch's last draw, of num_tiles - ctas in all, puts the counter back to zero.  A draw is made as late as
      // the loads allow: a CTA that held three tiles ahead of its stores would finish after the others.
      const int ctas = static_cast<int>(gridDim.x);
      int tile = static_cast<int>(blockIdx.x);
      for (uint32_t t = 0; ok; ++t) {
        const bool done = tile >= p.num_tiles;
        int b = -1, m0 = 0, n0 = 0;
        if (!done) {
          int tm, tn;
          tile_coords(p, tile, b, tm, tn);
          m0 = tm * TILE_M;
          n0 = tn * TILE_N;
        }
        bars->tile_ring[t % WALK_SLOTS] = make_int4(b, m0, n0, 0);
        mbar_arrive(&bars->tile_full[t % WALK_SLOTS]);
        if (done) break;
        for (int kb = 0; kb < p.k_blocks; ++kb, ++it) {
          const uint32_t s = it % STAGES;
          if (!mbar_wait(&bars->empty[s], ((it / STAGES) & 1) ^ 1, abort_word, 141)) {
            ok = false;
            break;
          }
          uint8_t* sa = smem + s * STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          mbar_arrive_expect_tx(&bars->full[s], STAGE_BYTES);
          const int k0 = kb * BK;
          if (p.a_mn) {
#pragma unroll
            for (int i = 0; i < TILE_M / 64; ++i)
              tma_load_3d(sa + i * 8192, &tmap_a, &bars->full[s], m0 + i * 64, k0, b);
          } else {
            tma_load_3d(sa, &tmap_a, &bars->full[s], k0, m0, b);
          }
          if (p.b_mn) {
#pragma unroll
            for (int i = 0; i < TILE_N / 64; ++i)
              tma_load_3d(sb + i * 8192, &tmap_b, &bars->full[s], n0 + i * 64, k0, b);
          } else {
            tma_load_3d(sb, &tmap_b, &bars->full[s], k0, n0, b);
          }
        }
        if (!ok || !mbar_wait(&bars->acc_empty[(t + 1) & 1], (((t + 1) >> 1) & 1) ^ 1, abort_word, 142)) break;
        if (t == 0 || p.sched_counter == nullptr) {  // (without a counter: fixed shares)
          tile += ctas;
        } else {
          const unsigned drawn = atomicAdd(p.sched_counter, 1u);
          if (drawn + 1 == static_cast<unsigned>(p.num_tiles - ctas)) atomicExch(p.sched_counter, 0u);
          tile = 2 * ctas + static_cast<int>(drawn);
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(TILE_M, TILE_N, p.a_mn, p.b_mn);
      const uint32_t a_lbo = p.a_mn ? 8192u : 16u, b_lbo = p.b_mn ? 8192u : 16u;
      const uint32_t a_kstep = p.a_mn ? 2048u : 32u, b_kstep = p.b_mn ? 2048u : 32u;
      uint32_t it = 0;
      bool ok = true;
      for (uint32_t t = 0; ok; ++t) {
        if (!mbar_wait(&bars->tile_full[t % WALK_SLOTS], (t / WALK_SLOTS) & 1, abort_word, 243) ||
            bars->tile_ring[t % WALK_SLOTS].x < 0)
          break;
        const uint32_t acc = t & 1, d = tmem_base + acc * TILE_N;
        if (!mbar_wait(&bars->acc_empty[acc], ((t >> 1) & 1) ^ 1, abort_word, 241)) break;
        tc_fence_after();
        for (int kb = 0; kb < p.k_blocks; ++kb, ++it) {
          const uint32_t s = it % STAGES;
          if (!mbar_wait(&bars->full[s], (it / STAGES) & 1, abort_word, 242)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + s * STAGE_BYTES), sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_ss(d, smem_desc_sw128(sa + k * a_kstep, a_lbo, 1024), smem_desc_sw128(sb + k * b_kstep, b_lbo, 1024),
                    idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit(&bars->empty[s]);
        }
        if (ok) umma_commit(&bars->acc_full[acc]);
      }
    }
  } else {
    const int w = warp - 2, row = (warp & 3) * 32 + lane, half = w >> 2;
    for (uint32_t t = 0;; ++t) {
      bool ok = mbar_wait(&bars->tile_full[t % WALK_SLOTS], (t / WALK_SLOTS) & 1, abort_word, 342);
      const int4 tile = ok ? bars->tile_ring[t % WALK_SLOTS] : make_int4(-1, 0, 0, 0);
      const int b = tile.x, m0 = tile.y, n0 = tile.z;
      const uint32_t acc = t & 1;
      if (b >= 0) {
        ok = mbar_wait(&bars->acc_full[acc], (t >> 1) & 1, abort_word, 341);
        tc_fence_after();
        if (ok && m0 + (warp & 3) * 32 < p.M) {
#pragma unroll
          for (int c = half * 64; c < half * 64 + 64; c += 16) {
            uint32_t r[16];
            tmem_ld16(tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + acc * TILE_N + c, r);
            tmem_wait_ld(r);
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
            store_partial(part, row, c, v);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->acc_empty[acc]);
      }
      // The whole tile is in shared memory.  The end of the walk, or a wait that ran out, ends it for all eight
      // warps here: one that left alone would keep the others at the barrier.
      if (store_warps_any(!ok || b < 0)) break;
      TileOut<1, WARPS> tile_out;
      tile_out.finish(p, part, 0, w, b, m0, n0);
      __syncwarp();
      store_warps_sync();  // and has been read
    }
  }
  __syncwarp();
  if (*abort_word != 0) {
    // Loads that may still be in flight land before shared memory is released.
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, WALK_TMEM_COLS);
  }
  if (threadIdx.x == 0 && *abort_word != 0) atomicExch(p.status, *abort_word);
  if (p.early) grid_dep_wait();
}

template <int S, int STAGES>
int32_t launch(const CUtensorMap& tm_a, const CUtensorMap& tm_b, const Params& p, int dev, cudaStream_t stream) {
  static std::once_flag once[64];
  cudaError_t err = cudaSuccess;
  std::call_once(once[dev & 63], [&] {
    err = cudaFuncSetAttribute(gemm_cluster_kernel<S, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(smem_bytes(STAGES)));
  });
  if (err != cudaSuccess) return fail(CDL_ERR_CUDA, "cudaFuncSetAttribute failed: %s", cudaGetErrorString(err));
  CDL_CUDA(launch_pdl_cluster(gemm_cluster_kernel<S, STAGES>, dim3(static_cast<unsigned>(p.num_tiles) * S),
                              dim3(THREADS), smem_bytes(STAGES), S, stream, tm_a, tm_b, p));
  return CDL_OK;
}
template <int S>
int32_t launch(const CUtensorMap& tm_a, const CUtensorMap& tm_b, const Params& p, int dev, cudaStream_t stream) {
  return static_cast<long long>(p.num_tiles) * S <= sm_count() ? launch<S, ALONE_STAGES>(tm_a, tm_b, p, dev, stream)
                                                               : launch<S, SHARED_STAGES>(tm_a, tm_b, p, dev, stream);
}

}  // namespace

int32_t gemm_cluster_launch(const CUtensorMap& tm_a, const CUtensorMap& tm_b, const Params& p,
                            int early, cudaStream_t stream) {
  int dev = 0;
  CDL_CUDA(cudaGetDevice(&dev));
  // The walk pays where an SM gets two tiles or more.
  if (p.split_k == 1 && p.atomic_out && p.num_tiles >= 2 * sm_count()) {
    static std::once_flag once[64];
    cudaError_t err = cudaSuccess;
    std::call_once(once[dev & 63], [&] {
      err = cudaFuncSetAttribute(gemm_cluster_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(WALK_SMEM_BYTES));
    });
    if (err != cudaSuccess) return fail(CDL_ERR_CUDA, "cudaFuncSetAttribute failed: %s", cudaGetErrorString(err));
    Params walk = p;
    walk.sched_counter = sched_counter_for(gemm_counter_kind(early), dev, stream);  // launches of one stream that draw share a counter
    CDL_CUDA(launch_pdl(gemm_cluster_walk_kernel, dim3(static_cast<unsigned>(sm_count())), dim3(WALK_THREADS),
                        WALK_SMEM_BYTES, stream, tm_a, tm_b, walk));
    return CDL_OK;
  }
  switch (p.split_k) {
    case 1: return launch<1>(tm_a, tm_b, p, dev, stream);
    case 2: return launch<2>(tm_a, tm_b, p, dev, stream);
    case 4: return launch<4>(tm_a, tm_b, p, dev, stream);
    default: return launch<8>(tm_a, tm_b, p, dev, stream);
  }
}

}  // namespace gemm
}  // namespace cdl
