// Quantised dense linears: y_i = x W_i^T for up to three planar Q8_0 / Q4_K weights
// that share the input (the q, k and v projections), as one C call:
//   1. linear_rows_kernel: the input rows as fp16 (optionally RMS-normalised first),
//      in the column order(s) the weights' layouts read, plus the segment [0, rows];
//   2. one launch for all weights of a layout (regime by the row count);
//   3. where k was split, linear_finish_kernel: the k-split partial sums of all outputs added, rounded
//      to the output type and, for a block's last projection, added to the residual.
// Replaces, per linear, a cast, a column shuffle, a torch.tensor upload of the segment
// (a host synchronisation), a sum over partials and a cast.  One B200, q/k/v/output
// projections of 4096 rows, hidden 4096, Q8_0: the three bf16 -> fp16 casts of the
// shared input took 43 us each, step 1 takes 17 us once with the norm and 13 us without.
#include "kernels.h"

namespace b200moe {
namespace {

constexpr int LIN_MAX = 3;
constexpr int LR_THREADS = 256;
constexpr int LR_MAXV = 4;  // 8-element vectors per thread kept in registers between the passes

template <int DT>
__device__ __forceinline__ void lin_load8(const void* p, size_t i, float (&v)[8]) {
  if constexpr (DT == B200MOE_DT_F32) {
    const float4 a = *reinterpret_cast<const float4*>(static_cast<const float*>(p) + i);
    const float4 b = *reinterpret_cast<const float4*>(static_cast<const float*>(p) + i + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
    const uint4 raw = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p) + i);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if constexpr (DT == B200MOE_DT_BF16) {
        v[2 * j] = __uint_as_float(w[j] << 16);
        v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
      } else {
        const float2 f = __half22float2(u32_as_h2(w[j]));
        v[2 * j] = f.x; v[2 * j + 1] = f.y;
      }
    }
  }
}

struct LinRowsArgs {
  const void* x;
  const float* norm_w;  // NULL: no norm
  float eps;
  int K;
  int rows;
  __half* plain;        // columns in order, or NULL
  __half* perm;         // halves of every 16 bytes in the order 0,4,1,5,2,6,3,7, or NULL
  int32_t* seg;
};

__device__ __forceinline__ void lin_store8(const LinRowsArgs& a, size_t i, const float (&v)[8]) {
  // no saturation: an input beyond fp16 becomes an infinity, as in a plain cast
  auto pk = [](float lo, float hi) { return h2_as_u32(__floats2half2_rn(lo, hi)); };
  if (a.plain != nullptr)
    *reinterpret_cast<uint4*>(a.plain + i) = make_uint4(pk(v[0], v[1]), pk(v[2], v[3]), pk(v[4], v[5]), pk(v[6], v[7]));
  if (a.perm != nullptr)
    *reinterpret_cast<uint4*>(a.perm + i) = make_uint4(pk(v[0], v[4]), pk(v[1], v[5]), pk(v[2], v[6]), pk(v[3], v[7]));
}

// One CTA per row, 16-byte accesses.  HBM-bound: x read once (rows of up to 8192
// columns stay in registers between the norm's two passes), fp16 written once.
template <int DT>
__global__ void __launch_bounds__(LR_THREADS) linear_rows_kernel(const LinRowsArgs a) {
  __shared__ float s_red[LR_THREADS / 32];
  const int tid = threadIdx.x;
  const size_t base = static_cast<size_t>(blockIdx.x) * a.K;
  const int nvec = a.K / 8;
  grid_dep_wait();
  grid_dep_launch();
  if (blockIdx.x == 0 && tid < 2) a.seg[tid] = tid * a.rows;
  if (a.norm_w == nullptr) {
    for (int j = tid; j < nvec; j += LR_THREADS) {
      float v[8];
      lin_load8<DT>(a.x, base + 8 * j, v);
      lin_store8(a, base + 8 * j, v);
    }
    return;
  }
  float x[LR_MAXV][8];
  float ss = 0.f;
#pragma unroll
  for (int r = 0; r < LR_MAXV; ++r) {
    const int j = tid + r * LR_THREADS;
    if (j < nvec) {
      lin_load8<DT>(a.x, base + 8 * j, x[r]);
#pragma unroll
      for (int i = 0; i < 8; ++i) ss = fmaf(x[r][i], x[r][i], ss);
    }
  }
  for (int j = tid + LR_MAXV * LR_THREADS; j < nvec; j += LR_THREADS) {
    float v[8];
    lin_load8<DT>(a.x, base + 8 * j, v);
#pragma unroll
    for (int i = 0; i < 8; ++i) ss = fmaf(v[i], v[i], ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) s_red[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < LR_THREADS / 32; ++i) tot += s_red[i];
  const float rstd = 1.0f / sqrtf(tot / static_cast<float>(a.K) + a.eps);
#pragma unroll
  for (int r = 0; r < LR_MAXV; ++r) {
    const int j = tid + r * LR_THREADS;
    if (j < nvec) {
      float w[8];
      lin_load8<B200MOE_DT_F32>(a.norm_w, 8 * j, w);
#pragma unroll
      for (int i = 0; i < 8; ++i) x[r][i] = w[i] * (x[r][i] * rstd);
      lin_store8(a, base + 8 * j, x[r]);
    }
  }
  for (int j = tid + LR_MAXV * LR_THREADS; j < nvec; j += LR_THREADS) {
    float v[8], w[8];
    lin_load8<DT>(a.x, base + 8 * j, v);
    lin_load8<B200MOE_DT_F32>(a.norm_w, 8 * j, w);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = w[i] * (v[i] * rstd);
    lin_store8(a, base + 8 * j, v);
  }
}

struct LinFinishArgs {
  const float* part[LIN_MAX];   // [ks][rows * N]
  void* out[LIN_MAX];
  long long n[LIN_MAX];         // rows * N (a multiple of 4)
  int ks[LIN_MAX];
  long long vec_end[LIN_MAX];   // running count of 4-element vectors
  const void* residual;         // added to entry 0, or NULL; output dtype
  int count;
};

__device__ __forceinline__ float lin_round(float v, int dt) {
  if (dt == B200MOE_DT_BF16) return __bfloat162float(__float2bfloat16_rn(v));
  if (dt == B200MOE_DT_F16) return __half2float(__float2half_rn(v));
  return v;
}

// Four elements per thread; partials added in split order.
template <int DT>
__global__ void __launch_bounds__(256) linear_finish_kernel(const LinFinishArgs a) {
  const long long total = a.vec_end[a.count - 1];
  grid_dep_wait();
  grid_dep_launch();
  for (long long vi = blockIdx.x * 256ll + threadIdx.x; vi < total; vi += gridDim.x * 256ll) {
    int o = 0;
    while (vi >= a.vec_end[o]) ++o;
    const long long i = 4 * (vi - (o > 0 ? a.vec_end[o - 1] : 0));
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = 0; c < a.ks[o]; ++c) {
      const float4 p = __ldcs(reinterpret_cast<const float4*>(a.part[o] + c * a.n[o] + i));
      v[0] += p.x; v[1] += p.y; v[2] += p.z; v[3] += p.w;
    }
    if (a.residual != nullptr && o == 0) {
      // as `h + y` on tensors: y is rounded to its type, then the sum
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = lin_round(v[j], DT);
      if constexpr (DT == B200MOE_DT_F32) {
        const float4 r = *reinterpret_cast<const float4*>(static_cast<const float*>(a.residual) + i);
        v[0] += r.x; v[1] += r.y; v[2] += r.z; v[3] += r.w;
      } else {
        const uint2 raw = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(a.residual) + i);
        const uint32_t w[2] = {raw.x, raw.y};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if constexpr (DT == B200MOE_DT_BF16) {
            v[2 * j] += __uint_as_float(w[j] << 16);
            v[2 * j + 1] += __uint_as_float(w[j] & 0xffff0000u);
          } else {
            const float2 f = __half22float2(u32_as_h2(w[j]));
            v[2 * j] += f.x; v[2 * j + 1] += f.y;
          }
        }
      }
    }
    if constexpr (DT == B200MOE_DT_F32) {
      *reinterpret_cast<float4*>(static_cast<float*>(a.out[o]) + i) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
      uint32_t w[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if constexpr (DT == B200MOE_DT_BF16) {
          const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
          w[j] = *reinterpret_cast<const uint32_t*>(&b);
        } else {
          w[j] = h2_as_u32(__floats2half2_rn(v[2 * j], v[2 * j + 1]));
        }
      }
      *reinterpret_cast<uint2*>(static_cast<uint16_t*>(a.out[o]) + i) = make_uint2(w[0], w[1]);
    }
  }
}

inline size_t up1k(size_t v) { return (v + 1023) / 1024 * 1024; }

// Weights of one layout go into one launch, with one kernel choice and k split.
struct LinGroup {
  const b200moe_weight_t* w[LIN_MAX];
  int index[LIN_MAX];  // place in the caller's list
  int count, ks;
  bool tensor;
  bool direct;  // the product writes the finished outputs itself
};

LinGroup lin_group(const b200moe_weight_t* const* w, int count, int rows, int layout) {
  LinGroup g{};
  g.tensor = true;
  for (int i = 0; i < count; ++i) {
    if (w[i]->layout != layout) continue;
    g.w[g.count] = w[i];
    g.index[g.count++] = i;
    g.tensor = g.tensor && pick_regime(B200MOE_REGIME_AUTO, w[i], rows, true) == B200MOE_REGIME_TENSOR;
  }
  if (g.count > 0) g.ks = g.tensor ? tc_linear_ksplit(g.w, g.count, rows) : stream_linear_ksplit(g.w, g.count, rows);
  g.direct = g.tensor && g.ks == 1;
  return g;
}

constexpr int LIN_LAYOUTS[2] = {B200MOE_LAYOUT_Q8_0, B200MOE_LAYOUT_Q4_K};

struct LinWorkspace {
  int32_t* seg;
  __half* plain;
  __half* perm;
  float* part[LIN_MAX];
  int ks[LIN_MAX];  // 0: no partial sums
  size_t bytes;
};

// `x_ready`: the input is fp16 already and no norm is asked for: weights that read
// columns in order take it as it is.
LinWorkspace lin_carve(const b200moe_weight_t* const* w, int count, int rows, bool x_ready, void* base) {
  LinWorkspace o{};
  uint8_t* p = static_cast<uint8_t*>(base);
  size_t off = 0;
  auto take = [&](size_t n) {
    void* r = p ? p + off : nullptr;
    off += up1k(n);
    return r;
  };
  bool plain = false, perm = false;
  for (int i = 0; i < count; ++i)
    (b200moe_kperm(w[i]->layout, B200MOE_REGIME_AUTO, rows) ? perm : plain) = true;
  const size_t row_bytes = static_cast<size_t>(rows) * w[0]->cols * 2;
  o.seg = static_cast<int32_t*>(take(8));
  if (plain && !x_ready) o.plain = static_cast<__half*>(take(row_bytes));
  if (perm) o.perm = static_cast<__half*>(take(row_bytes));
  for (int layout : LIN_LAYOUTS) {
    const LinGroup g = lin_group(w, count, rows, layout);
    for (int i = 0; i < g.count; ++i) o.ks[g.index[i]] = g.direct ? 0 : g.ks;
  }
  for (int i = 0; i < count; ++i)
    if (o.ks[i] > 0) o.part[i] = static_cast<float*>(take(static_cast<size_t>(o.ks[i]) * rows * w[i]->rows * 4));
  o.bytes = off;
  return o;
}

bool lin_dtype(int dt) { return dt == B200MOE_DT_F32 || dt == B200MOE_DT_F16 || dt == B200MOE_DT_BF16; }

int lin_check(const b200moe_weight_t* const* w, int count, int rows) {
  B200_REQUIRE(w != nullptr && count >= 1 && count <= LIN_MAX, "linear: 1..%d weights", LIN_MAX);
  B200_REQUIRE(rows >= 0, "linear: negative row count");
  for (int i = 0; i < count; ++i) {
    B200_REQUIRE(w[i] != nullptr && w[i]->experts == 1, "linear: weight %d must be a stack of one matrix", i);
    B200_REQUIRE(w[i]->layout == B200MOE_LAYOUT_Q8_0 || w[i]->layout == B200MOE_LAYOUT_Q4_K,
                 "linear: weight %d layout %d unsupported", i, w[i]->layout);
    B200_REQUIRE(w[i]->cols == w[0]->cols && w[i]->cols > 0 && w[i]->cols % 256 == 0 && w[i]->rows > 0 &&
                     w[i]->rows % 128 == 0,
                 "linear: weight %d is %d x %d (rows a multiple of 128, cols of 256 and equal)", i, w[i]->rows,
                 w[i]->cols);
  }
  return B200MOE_OK;
}

}  // namespace
}  // namespace b200moe

using namespace b200moe;

extern "C" {

size_t b200moe_linear_workspace_bytes(const b200moe_weight_t* const* weights, int32_t count, int32_t rows,
                                      int x_dtype, int has_norm) {
  if (lin_check(weights, count, rows) != B200MOE_OK || rows == 0) return 0;
  return lin_carve(weights, count, rows, x_dtype == B200MOE_DT_F16 && !has_norm, nullptr).bytes;
}

int b200moe_linear(const void* x, int x_dtype, int32_t rows, const float* norm_weight, float eps,
                   const b200moe_weight_t* const* weights, int32_t count, void* const* outs, int out_dtype,
                   const void* residual, void* workspace, size_t workspace_bytes, void* stream) {
  if (int rc = lin_check(weights, count, rows)) return rc;
  if (rows == 0) return B200MOE_OK;
  B200_REQUIRE(x && outs && workspace, "linear: NULL buffer");
  B200_REQUIRE(lin_dtype(x_dtype) && lin_dtype(out_dtype), "linear: unknown dtype");
  B200_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(norm_weight) |
                 reinterpret_cast<uintptr_t>(residual)) & 15) == 0,
               "linear: x, norm weight and residual must be 16-byte aligned");
  for (int i = 0; i < count; ++i)
    B200_REQUIRE(outs[i] && (reinterpret_cast<uintptr_t>(outs[i]) & 15) == 0, "linear: output %d missing or misaligned", i);
  const bool x_ready = x_dtype == B200MOE_DT_F16 && norm_weight == nullptr;
  const LinWorkspace w = lin_carve(weights, count, rows, x_ready, workspace);
  if (w.bytes > workspace_bytes) {
    set_error("linear: workspace needs %zu bytes, got %zu", w.bytes, workspace_bytes);
    return B200MOE_ERR_WORKSPACE;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  LinRowsArgs ra{x, norm_weight, eps, weights[0]->cols, rows, w.plain, w.perm, w.seg};
  // (with nothing to convert one CTA still writes the segment)
  const unsigned row_ctas = (w.plain != nullptr || w.perm != nullptr) ? static_cast<unsigned>(rows) : 1u;
  if (x_dtype == B200MOE_DT_F32)
    B200_CHECK_CUDA(launch_dependent(linear_rows_kernel<B200MOE_DT_F32>, dim3(row_ctas), dim3(LR_THREADS), 0, st, ra));
  else if (x_dtype == B200MOE_DT_F16)
    B200_CHECK_CUDA(launch_dependent(linear_rows_kernel<B200MOE_DT_F16>, dim3(row_ctas), dim3(LR_THREADS), 0, st, ra));
  else
    B200_CHECK_CUDA(launch_dependent(linear_rows_kernel<B200MOE_DT_BF16>, dim3(row_ctas), dim3(LR_THREADS), 0, st, ra));
  LinFinishArgs fa{};
  long long run = 0;
  for (int layout : LIN_LAYOUTS) {
    const LinGroup g = lin_group(weights, count, rows, layout);
    if (g.count == 0) continue;
    const void* xs = b200moe_kperm(layout, B200MOE_REGIME_AUTO, rows) ? static_cast<const void*>(w.perm)
                     : x_ready                                        ? x
                                                                      : static_cast<const void*>(w.plain);
    float* parts[LIN_MAX] = {};
    void* dst[LIN_MAX] = {};
    for (int i = 0; i < g.count; ++i) {
      parts[i] = w.part[g.index[i]];
      dst[i] = outs[g.index[i]];
    }
    const void* res = g.index[0] == 0 ? residual : nullptr;
    if (int rc = g.tensor ? launch_tc_linear(xs, w.seg, rows, g.w, g.count, g.ks, parts, dst, out_dtype, res, st)
                          : launch_stream_linear(xs, w.seg, rows, g.w, g.count, g.ks, parts, st))
      return rc;
  }
  for (int i = 0; i < count; ++i) {
    if (w.ks[i] == 0) continue;
    const int o = fa.count++;
    fa.part[o] = w.part[i];
    fa.out[o] = outs[i];
    fa.ks[o] = w.ks[i];
    fa.n[o] = static_cast<long long>(rows) * weights[i]->rows;
    run += fa.n[o] / 4;
    fa.vec_end[o] = run;
    if (i == 0) fa.residual = residual;
  }
  if (fa.count == 0) return B200MOE_OK;
  const long long want = (run + 255) / 256, most = 16ll * sm_count();
  const unsigned ctas = static_cast<unsigned>(want < most ? want : most);
  if (out_dtype == B200MOE_DT_F32)
    B200_CHECK_CUDA(launch_dependent(linear_finish_kernel<B200MOE_DT_F32>, dim3(ctas), dim3(256), 0, st, fa));
  else if (out_dtype == B200MOE_DT_F16)
    B200_CHECK_CUDA(launch_dependent(linear_finish_kernel<B200MOE_DT_F16>, dim3(ctas), dim3(256), 0, st, fa));
  else
    B200_CHECK_CUDA(launch_dependent(linear_finish_kernel<B200MOE_DT_BF16>, dim3(ctas), dim3(256), 0, st, fa));
  return B200MOE_OK;
}

}  // extern "C"
