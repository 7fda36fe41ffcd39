// General NormFwd for what the vectorised kernels of rmsnorm.cu do not take: f32 inputs or
// outputs, f32 scale / bias, a column count that is not a multiple of 8 or exceeds 8192, strided or
// unaligned rows.  In the reference these shapes run on its Tile IR fallback (NormFwd with
// NormOutput::Plain, crates/cleandl/src/execgraph/ops/norm/mod.rs:223-261; the case list of
// fallback_configurations, crates/cleandl/tests/norm.rs:414-470: every combination of f32 / bf16
// x, output, scale and bias for both norm types, and rows of 20000 columns).
//
//   RmsNorm:   y = x * rsqrt(mean x^2 + eps) * scale + bias
//   LayerNorm: y = (x - mean x) * rsqrt(mean (x - mean x)^2 + eps) * scale + bias
// in f32.  Two kernels: rows with contiguous columns (norm_rows_kernel: the row is read from HBM once
// and stays in registers) and any other layout (norm_general_kernel: one warp per row, scalar accesses,
// the row read two or three times, from cache after the first).
#include "host.h"
#include "ops.h"
#include "ptx.cuh"

namespace cdl {
namespace norm_general {

struct Vec {
  const void* ptr;  // nullable
  long long stride;
  int f32;
  int vec;  // 1 = contiguous and aligned for the accesses of norm_rows_kernel
};
struct Params {
  const void* x;
  long long x_row, x_col;
  int x_f32;
  void* y;
  long long y_row, y_col;
  int y_f32;
  Vec scale, bias;
  float* mean;  // nullable
  long long mean_stride;
  float* r_inv;  // nullable
  long long r_inv_stride;
  int rows, cols;
  float eps;
  int layer;
};

__device__ __forceinline__ float load(const void* p, long long i, int f32) {
  return f32 ? static_cast<const float*>(p)[i]
             : __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void __launch_bounds__(256) norm_general_kernel(const Params p) {
  const int lane = threadIdx.x & 31;
  const long long warp = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const long long stride = static_cast<long long>(gridDim.x) * 8;
  const float inv_cols = 1.0f / static_cast<float>(p.cols);
  for (long long row = warp; row < p.rows; row += stride) {
    const long long xb = row * p.x_row;
    float mean = 0.f;
    if (p.layer) {
      float s = 0.f;
      for (int c = lane; c < p.cols; c += 32) s += load(p.x, xb + c * p.x_col, p.x_f32);
      mean = warp_sum(s) * inv_cols;
    }
    float ss = 0.f;
    for (int c = lane; c < p.cols; c += 32) {
      const float d = load(p.x, xb + c * p.x_col, p.x_f32) - mean;
      ss = fmaf(d, d, ss);
    }
    const float r = rsqrtf(warp_sum(ss) * inv_cols + p.eps);
    if (lane == 0) {
      if (p.mean != nullptr) p.mean[row * p.mean_stride] = mean;
      if (p.r_inv != nullptr) p.r_inv[row * p.r_inv_stride] = r;
    }
    const long long yb = row * p.y_row;
    for (int c = lane; c < p.cols; c += 32) {
      float v = (load(p.x, xb + c * p.x_col, p.x_f32) - mean) * r;
      if (p.scale.ptr != nullptr) v *= load(p.scale.ptr, c * p.scale.stride, p.scale.f32);
      if (p.bias.ptr != nullptr) v += load(p.bias.ptr, c * p.bias.stride, p.bias.f32);
      const long long yi = yb + c * p.y_col;
      if (p.y_f32) static_cast<float*>(p.y)[yi] = v;
      else static_cast<__nv_bfloat16*>(p.y)[yi] = __float2bfloat16_rn(v);
    }
  }
}

// Rows with contiguous columns, up to 32 * WARPS * E of them: WARPS warps share a row, a thread holds E
// values of it in registers, V consecutive columns per access.
//
// Bound by HBM: x is read once and y written once.  V is the widest access that every row's start
// allows (four f32 where rows are on the 16-byte grid, two or one where they are not: a [8192, 2050]
// f32 row starts on the 8-byte grid), so a warp's access still covers whole 64- or 128-byte lines.
// Wide rows take four warps (single columns up to 16) so that a thread's share stays at 20 or 32 values up to
// 4096 columns: 12 or 9 rows are then in flight per SM, where one warp per row would need over 64 registers a
// thread for the row alone.  From there to 8192 a share of 64 leaves 5.
// LayerNorm of f32 [8192, 2050] to f32 (134 MB): 27 us, 5.0 TB/s; norm_general_kernel, which reads the row
// three times with scalar accesses, 125 us.
template <int V>
__device__ __forceinline__ void load_cols(const float* q, float (&v)[V]) {
  if (V == 4) {
    const float4 w = *reinterpret_cast<const float4*>(q);
    v[0] = w.x; v[1 % V] = w.y; v[2 % V] = w.z; v[3 % V] = w.w;
  } else if (V == 2) {
    const float2 w = *reinterpret_cast<const float2*>(q);
    v[0] = w.x; v[1 % V] = w.y;
  } else {
    v[0] = *q;
  }
}
template <int V>
__device__ __forceinline__ void load_cols(const __nv_bfloat16* q, float (&v)[V]) {
  if (V == 4) {
    const uint2 w = *reinterpret_cast<const uint2*>(q);
    v[0] = bf16_lo(w.x); v[1 % V] = bf16_hi(w.x); v[2 % V] = bf16_lo(w.y); v[3 % V] = bf16_hi(w.y);
  } else if (V == 2) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(q);
    v[0] = bf16_lo(w); v[1 % V] = bf16_hi(w);
  } else {
    v[0] = __bfloat162float(*q);
  }
}
template <int V>
__device__ __forceinline__ void store_cols(float* q, const float (&v)[V]) {
  if (V == 4) *reinterpret_cast<float4*>(q) = make_float4(v[0], v[1 % V], v[2 % V], v[3 % V]);
  else if (V == 2) *reinterpret_cast<float2*>(q) = make_float2(v[0], v[1 % V]);
  else *q = v[0];
}
template <int V>
__device__ __forceinline__ void store_cols(__nv_bfloat16* q, const float (&v)[V]) {
  if (V == 4) *reinterpret_cast<uint2*>(q) = make_uint2(pack_bf16x2(v[0], v[1 % V]), pack_bf16x2(v[2 % V], v[3 % V]));
  else if (V == 2) *reinterpret_cast<uint32_t*>(q) = pack_bf16x2(v[0], v[1 % V]);
  else *q = __float2bfloat16_rn(v[0]);
}
template <int V>
__device__ __forceinline__ void load_vec(const Vec& s, int col, float (&v)[V]) {
  if (s.vec) {
    if (s.f32) load_cols<V>(static_cast<const float*>(s.ptr) + col, v);
    else load_cols<V>(static_cast<const __nv_bfloat16*>(s.ptr) + col, v);
  } else {
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] = load(s.ptr, (col + j) * s.stride, s.f32);
  }
}
template <int V, int N, int T, typename Y>
__device__ __forceinline__ void write_row(const Params& p, const float (&v)[N][V], float mean, float r, int c0, Y* y) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int col = c0 + i * T * V;
    if (col < p.cols) {
      float g[V], o[V];
#pragma unroll
      for (int j = 0; j < V; ++j) o[j] = (v[i][j] - mean) * r;
      if (p.scale.ptr != nullptr) {
        load_vec<V>(p.scale, col, g);
#pragma unroll
        for (int j = 0; j < V; ++j) o[j] *= g[j];
      }
      if (p.bias.ptr != nullptr) {
        load_vec<V>(p.bias, col, g);
#pragma unroll
        for (int j = 0; j < V; ++j) o[j] += g[j];
      }
      store_cols<V>(y + i * T * V, o);
    }
  }
}
// Sum over the WARPS warps that share a row; `slots` is a buffer of this call's own.
template <int WARPS>
__device__ __forceinline__ float row_sum(float v, float* slots) {
  v = warp_sum(v);
  if (WARPS == 1) return v;
  if ((threadIdx.x & 31) == 0) slots[threadIdx.x >> 5] = v;
  __syncthreads();
  v = 0.f;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) v += slots[w];
  return v;
}

template <int V, int E, int WARPS>
__global__ void __launch_bounds__(WARPS == 1 ? 256 : WARPS * 32) norm_rows_kernel(const Params p) {
  constexpr int N = E / V;              // accesses per thread
  constexpr int T = WARPS * 32;         // threads per row
  __shared__ float slots[2][WARPS];
  grid_dep_wait();
  grid_dep_launch();
  const int t = threadIdx.x % T;
  const long long row = WARPS == 1 ? static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5) : blockIdx.x;
  if (WARPS == 1 && row >= p.rows) return;  // (one row per CTA otherwise)
  // Per-thread bases, so that every access is a base and a constant offset.
  const int c0 = t * V;
  float v[N][V];
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < V; ++j) v[i][j] = 0.f;
  if (p.x_f32) {
    const float* x = static_cast<const float*>(p.x) + row * p.x_row + c0;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (c0 + i * T * V < p.cols) load_cols<V>(x + i * T * V, v[i]);
  } else {
    const __nv_bfloat16* x = static_cast<const __nv_bfloat16*>(p.x) + row * p.x_row + c0;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (c0 + i * T * V < p.cols) load_cols<V>(x + i * T * V, v[i]);
  }
  const float inv_cols = 1.0f / static_cast<float>(p.cols);
  float mean = 0.f;
  if (p.layer) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int j = 0; j < V; ++j) s += v[i][j];
    mean = row_sum<WARPS>(s, slots[0]) * inv_cols;
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (c0 + i * T * V < p.cols) {
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const float d = v[i][j] - mean;
        ss = fmaf(d, d, ss);
      }
    }
  const float r = rsqrtf(row_sum<WARPS>(ss, slots[1]) * inv_cols + p.eps);
  if (t == 0) {
    if (p.mean != nullptr) p.mean[row * p.mean_stride] = mean;
    if (p.r_inv != nullptr) p.r_inv[row * p.r_inv_stride] = r;
  }
  if (p.y_f32) write_row<V, N, T>(p, v, mean, r, c0, static_cast<float*>(p.y) + row * p.y_row + c0);
  else write_row<V, N, T>(p, v, mean, r, c0, static_cast<__nv_bfloat16*>(p.y) + row * p.y_row + c0);
}

// Columns of one access: the widest of 4, 2, 1 that x and y allow in every row.
static int access_width(const Params& p) {
  auto ok = [&](const void* ptr, long long row_stride, int f32, int v) {
    const long long bytes = v * (f32 ? 4 : 2);
    return reinterpret_cast<uintptr_t>(ptr) % bytes == 0 &&
           (p.rows == 1 || row_stride * (f32 ? 4 : 2) % bytes == 0);
  };
  for (int v = 4; v > 1; v /= 2)
    if (p.cols % v == 0 && ok(p.x, p.x_row, p.x_f32, v) && ok(p.y, p.y_row, p.y_f32, v)) return v;
  return 1;
}

// One row per CTA (E values a thread, WARPS warps), or one per warp.
template <int V, int E, int WARPS>
static cudaError_t launch_as(const Params& p, cudaStream_t stream) {
  const unsigned rows = static_cast<unsigned>(p.rows);
  return launch_pdl(norm_rows_kernel<V, E, WARPS>, dim3(WARPS == 1 ? (rows + 7) / 8 : rows),
                    dim3(WARPS == 1 ? 256 : WARPS * 32), 0, stream, p);
}
template <int V>
static cudaError_t launch_rows(const Params& p, cudaStream_t stream) {
  if (p.cols <= 256) return launch_as<V, 8, 1>(p, stream);
  if constexpr (V == 1) {
    // Single columns: an access moves 64 or 128 bytes, so instructions count, those beyond the row's end too.  A
    // thread takes few values and capacities lie closer.  LayerNorm of bf16, with the capacities below -> with
    // these: [40000, 257] 42.2 -> 23.7 us, [1024, 513] 9.4 -> 4.8, [8192, 1025] 26.7 -> 19.4, [8192, 4097] 152 -> 81;
    // norm_general_kernel takes 37.7, 8.6, 28.9 and 133.
    if (p.cols <= 384) return launch_as<1, 12, 1>(p, stream);
    if (p.cols <= 1024) return launch_as<1, 8, 4>(p, stream);
    if (p.cols <= 1536) return launch_as<1, 12, 4>(p, stream);
    if (p.cols <= 2560) return launch_as<1, 20, 4>(p, stream);
    if (p.cols <= 4096) return launch_as<1, 16, 8>(p, stream);
    if (p.cols <= 5120) return launch_as<1, 20, 8>(p, stream);
    return launch_as<1, 16, 16>(p, stream);
  } else {
    if (p.cols <= 1024) return launch_as<V, 32, 1>(p, stream);
    // 20 values leave room for 12 rows per SM, 32 for 9; f32 [8192, 2050] 27.1 us, with 32 values 32.8.
    if (p.cols <= 2560) return launch_as<V, 20, 4>(p, stream);
    if (p.cols <= 4096) return launch_as<V, 32, 4>(p, stream);
    return launch_as<V, 64, 4>(p, stream);
  }
}
constexpr int MAX_REGISTER_COLS = 8192;

static bool float_type(int32_t dt) { return dt == CDL_BF16 || dt == CDL_F32; }

}  // namespace norm_general

// layer = 0: RmsNorm (mean must be null), 1: LayerNorm.  Validates everything itself.
int32_t norm_general_execute(int layer, const cdl_tensor* x, const cdl_tensor* scale,
                             const cdl_tensor* bias, float eps, const cdl_tensor* y,
                             const cdl_tensor* mean, const cdl_tensor* r_inv, cudaStream_t stream) {
  using namespace norm_general;
  const char* op = layer ? "norm_fwd (layer norm)" : "norm_fwd";
  if (!x || !y) return fail(CDL_ERR_INVALID, "%s: x and y are required", op);
  if (x->rank != 2) return fail(CDL_ERR_INVALID, "%s: x must be a 2D tensor", op);
  const long long rows = x->shape[0], cols = x->shape[1];
  if (y->rank != 2 || y->shape[0] != rows || y->shape[1] != cols)
    return fail(CDL_ERR_INVALID, "%s: y must be a 2D tensor of shape [%lld, %lld]", op, rows, cols);
  if (!float_type(x->dtype) || !float_type(y->dtype))
    return fail(CDL_ERR_UNSUPPORTED, "%s: x and y must be f32 or bf16", op);
  for (const cdl_tensor* v : {scale, bias}) {
    if (!v) continue;
    if (v->rank != 1 || v->shape[0] != cols)
      return fail(CDL_ERR_INVALID, "%s: %s must have shape [%lld]", op, v == scale ? "scale" : "bias",
                  cols);
    if (!float_type(v->dtype))
      return fail(CDL_ERR_UNSUPPORTED, "%s: %s must be f32 or bf16", op, v == scale ? "scale" : "bias");
  }
  for (const cdl_tensor* v : {mean, r_inv}) {
    if (!v) continue;
    if (v->rank != 1 || v->shape[0] != rows || v->dtype != CDL_F32)
      return fail(CDL_ERR_INVALID, "%s: %s must be f32 [%lld]", op, v == mean ? "mean" : "r_inv", rows);
  }
  if (rows == 0 || cols == 0) return CDL_OK;
  if (rows > INT32_MAX || cols > INT32_MAX)
    return fail(CDL_ERR_UNSUPPORTED, "%s: shape [%lld, %lld] is too large", op, rows, cols);
  Params p{};
  p.x = x->ptr; p.x_row = x->stride[0]; p.x_col = x->stride[1]; p.x_f32 = x->dtype == CDL_F32;
  p.y = y->ptr; p.y_row = y->stride[0]; p.y_col = y->stride[1]; p.y_f32 = y->dtype == CDL_F32;
  if (scale) p.scale = Vec{scale->ptr, scale->stride[0], scale->dtype == CDL_F32, 0};
  if (bias) p.bias = Vec{bias->ptr, bias->stride[0], bias->dtype == CDL_F32, 0};
  if (mean) { p.mean = static_cast<float*>(mean->ptr); p.mean_stride = mean->stride[0]; }
  if (r_inv) { p.r_inv = static_cast<float*>(r_inv->ptr); p.r_inv_stride = r_inv->stride[0]; }
  p.rows = static_cast<int>(rows);
  p.cols = static_cast<int>(cols);
  p.eps = eps;
  p.layer = layer;
  const double elem = (p.x_f32 ? 4.0 : 2.0) + (p.y_f32 ? 4.0 : 2.0);
  ProfileScope ps(PROF_NORM_FWD, elem * rows * cols, stream);
  if ((p.x_col == 1 || cols == 1) && (p.y_col == 1 || cols == 1) && cols <= MAX_REGISTER_COLS) {
    const int v = access_width(p);
    for (Vec* s : {&p.scale, &p.bias})
      s->vec = s->stride == 1 && reinterpret_cast<uintptr_t>(s->ptr) % (v * (s->f32 ? 4 : 2)) == 0;
    CDL_CUDA(v == 4 ? launch_rows<4>(p, stream) : v == 2 ? launch_rows<2>(p, stream) : launch_rows<1>(p, stream));
    return CDL_OK;
  }
  const long long want = (rows + 7) / 8;
  const unsigned grid = static_cast<unsigned>(want < 16LL * sm_count() ? want : 16LL * sm_count());
  norm_general_kernel<<<grid, 256, 0, stream>>>(p);
  CDL_CUDA(cudaGetLastError());
  return CDL_OK;
}

}  // namespace cdl
