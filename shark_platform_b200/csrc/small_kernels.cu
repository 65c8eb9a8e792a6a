// Router, route plan, row permutation, combine, reference dequantisation and
// GGUF block unpacking.  All HBM-bound or latency-bound helpers around the two
// expert-GEMM kernels.
#include <atomic>

#include "common.cuh"
#include "kernels.h"

namespace b200moe {

// ------------------------------------------------------------------ router
// RMS norm in fp32, router logits from the fp32 normalised row, fp32 softmax, top-k by
// descending probability (ties: lowest expert id) and renormalised gates.  All router
// kernels compute a logit as rstd * sum((x * norm_w) * router_w) + bias, eight
// consecutive columns per lane, 256 per warp, warps added in order.
template <typename T>
__device__ __forceinline__ void load8(const T* p, float (&v)[8]);

template <>
__device__ __forceinline__ void load8<float>(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <>
__device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

constexpr int MAX_EXPERTS = 64;
constexpr int MAX_TOPK = 8;

// Softmax over the logits of one token held in shared memory, top-k and gate
// renormalisation by one warp (shared by the router kernels).
__device__ __forceinline__ void router_select(const float* logit, int lane, int E, int k,
                                              int32_t* experts_out, float* gates_out) {
  const float NEG = -INFINITY;
  float l0 = lane < E ? logit[lane] : NEG;
  float l1 = lane + 32 < E ? logit[lane + 32] : NEG;
  float mx = fmaxf(l0, l1);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float p0 = lane < E ? expf(l0 - mx) : 0.f;
  float p1 = lane + 32 < E ? expf(l1 - mx) : 0.f;
  float sum = p0 + p1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  p0 = lane < E ? p0 / sum : -1.f;
  p1 = lane + 32 < E ? p1 / sum : -1.f;
  float sel_p[MAX_TOPK];
  int sel_i[MAX_TOPK];
  float gsum = 0.f;
#pragma unroll
  for (int i = 0; i < MAX_TOPK; ++i) {
    if (i < k) {
      float bp = p0;
      int bi = lane;
      if (p1 > bp) { bp = p1; bi = lane + 32; }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float op = __shfl_xor_sync(0xffffffffu, bp, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (op > bp || (op == bp && oi < bi)) { bp = op; bi = oi; }
      }
      sel_p[i] = bp;
      sel_i[i] = bi;
      gsum += bp;
      if (bi == lane) p0 = -1.f;
      if (bi == lane + 32) p1 = -1.f;
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < MAX_TOPK; ++i) {
      if (i < k) {
        experts_out[i] = sel_i[i];
        gates_out[i] = sel_p[i] / gsum;
      }
    }
  }
}

// Sums of eight values over the warp: after each of the first three exchanges a lane
// keeps half of the values, so 9 shuffles do what eight butterflies do in 40, with the
// additions of a plain xor-16-8-4-2-1 butterfly.  Returns, on every lane, the sum of
// value 4*bit4 + 2*bit3 + bit2 of the lane number.
__device__ __forceinline__ float warp_sum8(const float (&a)[9], int lane) {
  float b[4], c[2];
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) b[i] = (h4 ? a[4 + i] : a[i]) + __shfl_xor_sync(0xffffffffu, h4 ? a[i] : a[4 + i], 16);
#pragma unroll
  for (int i = 0; i < 2; ++i) c[i] = (h3 ? b[2 + i] : b[i]) + __shfl_xor_sync(0xffffffffu, h3 ? b[i] : b[2 + i], 8);
  float v = (h2 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, h2 ? c[0] : c[1], 4);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v;
}
__device__ __forceinline__ int warp_sum8_index(int lane) { return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1); }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Many tokens: one CTA routes RT_TOKENS tokens at a time, warp w taking the column
// chunks w, w + 8, ... of 256.  Every router weight that is loaded serves four tokens,
// and the CTAs of an SM share the weights through L1; the kernel before this one (a
// warp per token, weights in shared memory, one 8-warp CTA per SM) waited for latency
// most of the time.  Writes the token's rstd and the CTA's expert counts for
// route_permute_kernel, or (xn_out) the normalised rows as fp16.
// One B200, us: 4096 tokens, hidden 4096, 8 experts 59 -> 35; 8192 tokens, hidden 6144
// 186 -> 78; 777 tokens 42 -> 14.
constexpr int RT_TOKENS = 4;
constexpr int RT_THREADS = 256;

template <typename T>
__global__ void __launch_bounds__(RT_THREADS, 2)
router_tokens_kernel(const T* __restrict__ h, int tokens, int d, int E, int k, float eps,
                     const float* __restrict__ norm_w, const float* __restrict__ rw,
                     const float* __restrict__ rb, __half* __restrict__ xn_out,
                     int32_t* __restrict__ experts_out, float* __restrict__ gates_out,
                     float* __restrict__ rstd_out, int32_t* __restrict__ hist) {
  constexpr int WARPS = RT_THREADS / 32;
  __shared__ float s_part[WARPS][RT_TOKENS][9];  // eight logit sums, sum of squares
  __shared__ float s_logit[RT_TOKENS][MAX_EXPERTS];
  __shared__ float s_rstd[RT_TOKENS];
  __shared__ int32_t s_sel[RT_TOKENS * MAX_TOPK];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int t0 = blockIdx.x * RT_TOKENS;
  const int nt = min(RT_TOKENS, tokens - t0);
  const T* rows = h + static_cast<size_t>(t0) * d;
  for (int e0 = 0; e0 < E; e0 += 8) {
    float acc[RT_TOKENS][9];
#pragma unroll
    for (int q = 0; q < RT_TOKENS; ++q)
#pragma unroll
      for (int e = 0; e < 9; ++e) acc[q][e] = 0.f;
    for (int j = warp * 256 + lane * 8; j < d; j += WARPS * 256) {
      float x[RT_TOKENS][8], w[8];
#pragma unroll
      for (int q = 0; q < RT_TOKENS; ++q)
        load8<T>(rows + static_cast<size_t>(q < nt ? q : 0) * d + j, x[q]);
      load8<float>(norm_w + j, w);
#pragma unroll
      for (int q = 0; q < RT_TOKENS; ++q)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          acc[q][8] = fmaf(x[q][i], x[q][i], acc[q][8]);
          x[q][i] *= w[i];
        }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if (e0 + e < E) {
          load8<float>(rw + static_cast<size_t>(e0 + e) * d + j, w);
#pragma unroll
          for (int q = 0; q < RT_TOKENS; ++q)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[q][e] = fmaf(x[q][i], w[i], acc[q][e]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < RT_TOKENS; ++q) {
      const float v = warp_sum8(acc[q], lane), ss = warp_sum(acc[q][8]);
      if ((lane & 3) == 0) s_part[warp][q][warp_sum8_index(lane)] = v;
      if (lane == 0) s_part[warp][q][8] = ss;
    }
    __syncthreads();
    if (tid < RT_TOKENS * 8) {
      const int q = tid >> 3, e = tid & 7;
      float tot = 0.f, v = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        tot += s_part[w][q][8];
        v += s_part[w][q][e];
      }
      const float rstd = 1.0f / sqrtf(tot / static_cast<float>(d) + eps);
      if (e0 + e < E) s_logit[q][e0 + e] = v * rstd + (rb ? rb[e0 + e] : 0.f);
      if (e == 0) s_rstd[q] = rstd;
    }
    __syncthreads();
  }
  if (warp < nt) {
    router_select(s_logit[warp], lane, E, k, s_sel + warp * k, gates_out + static_cast<size_t>(t0 + warp) * k);
    __syncwarp();
    if (lane < k) experts_out[static_cast<size_t>(t0 + warp) * k + lane] = s_sel[warp * k + lane];
    if (lane == 0 && rstd_out != nullptr) rstd_out[t0 + warp] = s_rstd[warp];
  }
  if (hist != nullptr) {
    __syncthreads();
    for (int e = tid; e < E; e += RT_THREADS) {
      int c = 0;
      for (int i = 0; i < nt * k; ++i) c += s_sel[i] == e;
      hist[static_cast<size_t>(blockIdx.x) * E + e] = c;
    }
  }
  if (xn_out != nullptr) {
    for (int q = 0; q < nt; ++q) {
      const float rstd = s_rstd[q];
      for (int j = tid * 8; j < d; j += RT_THREADS * 8) {
        float x[8], w[8];
        load8<T>(rows + static_cast<size_t>(q) * d + j, x);  // second pass: from L1 / L2
        load8<float>(norm_w + j, w);
        uint32_t packed[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          packed[i] = h2_as_u32(__halves2half2(to_half_sat(w[2 * i] * (x[2 * i] * rstd)),
                                               to_half_sat(w[2 * i + 1] * (x[2 * i + 1] * rstd))));
        *reinterpret_cast<uint4*>(xn_out + static_cast<size_t>(t0 + q) * d + j) =
            make_uint4(packed[0], packed[1], packed[2], packed[3]);
      }
    }
  }
}

// Route plan, norm and row permutation of a whole prefill call, after
// router_tokens_kernel: one CTA per RP_TOKENS tokens adds up the router CTAs' expert
// counts (all of them for the segment offsets, those before it for its own rank base),
// ranks its pairs (stable by pair index, as route_plan_kernel does) and writes each
// token's normalised row to its k sorted positions.  The row is read once and never
// stored unpermuted: plan and permutation took two launches and three passes over the
// fp16 rows.  One B200, us, plan + permutation -> this kernel: 4096 tokens, hidden 4096,
// top 2 11 + 17 -> 21; 8192 tokens, hidden 6144 20 + 56 -> 61.
constexpr int RP_TOKENS = 8;
constexpr int RP_THREADS = 256;
// the counts are read whole by every CTA: up to 64 KB of them
constexpr long long RP_MAX_COUNTS = 16384;

template <typename T>
__global__ void __launch_bounds__(RP_THREADS)
route_permute_kernel(const T* __restrict__ h, int tokens, int d, int E, int k,
                     const float* __restrict__ norm_w, const float* rstd, const int32_t* experts, const int32_t* hist,
                     int32_t* __restrict__ counts, int32_t* __restrict__ seg, int32_t* __restrict__ perm,
                     int32_t* __restrict__ inv, int kperm, uint4* __restrict__ xs) {
  __shared__ int s_total[MAX_EXPERTS], s_before[MAX_EXPERTS], s_seg[MAX_EXPERTS + 1];
  __shared__ int s_e[RP_TOKENS * MAX_TOPK], s_pos[RP_TOKENS * MAX_TOPK];
  static_assert(RP_TOKENS % RT_TOKENS == 0, "a CTA starts at a router CTA's first token");
  const int tid = threadIdx.x;
  const int t0 = blockIdx.x * RP_TOKENS;
  const int nt = min(RP_TOKENS, tokens - t0);
  const int np = nt * k;
  grid_dep_wait();
  grid_dep_launch();
  for (int e = tid; e < MAX_EXPERTS; e += RP_THREADS) s_total[e] = s_before[e] = 0;
  for (int i = tid; i < np; i += RP_THREADS) s_e[i] = experts[static_cast<size_t>(t0) * k + i];
  __syncthreads();
  // consecutive threads take consecutive (count row, expert) entries; where E divides
  // the CTA's stride a thread stays on its four experts and adds up in registers
  const int rows = (tokens + RT_TOKENS - 1) / RT_TOKENS, mine = t0 / RT_TOKENS;
  if (E % 4 == 0 && (4 * RP_THREADS) % E == 0) {
    const int4* h4 = reinterpret_cast<const int4*>(hist);
    int4 all = make_int4(0, 0, 0, 0), before = all;
#pragma unroll 8
    for (int i = tid; i < rows * E / 4; i += RP_THREADS) {
      const int4 c = h4[i];
      all.x += c.x; all.y += c.y; all.z += c.z; all.w += c.w;
      if (4 * i < mine * E) { before.x += c.x; before.y += c.y; before.z += c.z; before.w += c.w; }
    }
    const int e = (4 * tid) % E;
    // lanes E/4 apart hold the same experts
    for (int o = 16; o >= E / 4 && o > 0; o >>= 1) {
      all.x += __shfl_xor_sync(0xffffffffu, all.x, o); all.y += __shfl_xor_sync(0xffffffffu, all.y, o);
      all.z += __shfl_xor_sync(0xffffffffu, all.z, o); all.w += __shfl_xor_sync(0xffffffffu, all.w, o);
      before.x += __shfl_xor_sync(0xffffffffu, before.x, o); before.y += __shfl_xor_sync(0xffffffffu, before.y, o);
      before.z += __shfl_xor_sync(0xffffffffu, before.z, o); before.w += __shfl_xor_sync(0xffffffffu, before.w, o);
    }
    if ((tid & 31) < E / 4) {
      atomicAdd(&s_total[e], all.x); atomicAdd(&s_total[e + 1], all.y);
      atomicAdd(&s_total[e + 2], all.z); atomicAdd(&s_total[e + 3], all.w);
      atomicAdd(&s_before[e], before.x); atomicAdd(&s_before[e + 1], before.y);
      atomicAdd(&s_before[e + 2], before.z); atomicAdd(&s_before[e + 3], before.w);
    }
  } else {
    for (int i = tid; i < rows * E; i += RP_THREADS) {
      const int c = hist[i], e = i % E;
      if (c != 0) {
        atomicAdd(&s_total[e], c);
        if (i < mine * E) atomicAdd(&s_before[e], c);
      }
    }
  }
  __syncthreads();
  if (tid == 0) {
    int run = 0;
    for (int e = 0; e < E; ++e) {
      s_seg[e] = run;
      run += s_total[e];
    }
    s_seg[E] = run;
  }
  __syncthreads();
  if (blockIdx.x == 0)
    for (int e = tid; e <= E; e += RP_THREADS) {
      seg[e] = s_seg[e];
      if (e < E) counts[e] = s_total[e];
    }
  for (int i = tid; i < np; i += RP_THREADS) {
    const int e = s_e[i];
    int rank = 0;
    for (int j = 0; j < i; ++j) rank += s_e[j] == e;
    const int pos = s_seg[e] + s_before[e] + rank;
    const int p = t0 * k + i;
    s_pos[i] = pos;
    perm[pos] = p;
    inv[p] = pos;
  }
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31;
  const int nvec = d / 8;
  for (int q = warp; q < nt; q += RP_THREADS / 32) {
    const T* row = h + static_cast<size_t>(t0 + q) * d;
    const float r = rstd[t0 + q];
    // four vectors at a time: their loads are in flight together (nvec is a multiple of 32)
    for (int j0 = lane; j0 < nvec; j0 += 128) {
      float x[4][8];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j0 + 32 * u < nvec) load8<T>(row + (j0 + 32 * u) * 8, x[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = j0 + 32 * u;
        if (j >= nvec) break;
        float w[8];
        load8<float>(norm_w + j * 8, w);
        __half v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = to_half_sat(w[i] * (x[u][i] * r));
        uint4 o;
        if (kperm) {  // halves in the order 0,4,1,5,2,6,3,7 (see permute_rows_kernel)
          o.x = h2_as_u32(__halves2half2(v[0], v[4]));
          o.y = h2_as_u32(__halves2half2(v[1], v[5]));
          o.z = h2_as_u32(__halves2half2(v[2], v[6]));
          o.w = h2_as_u32(__halves2half2(v[3], v[7]));
        } else {
          o.x = h2_as_u32(__halves2half2(v[0], v[1]));
          o.y = h2_as_u32(__halves2half2(v[2], v[3]));
          o.z = h2_as_u32(__halves2half2(v[4], v[5]));
          o.w = h2_as_u32(__halves2half2(v[6], v[7]));
        }
        for (int s = 0; s < k; ++s) xs[static_cast<size_t>(s_pos[q * k + s]) * nvec + j] = o;
      }
    }
  }
}

// One CTA per token: used for small token counts (decode), where a warp per
// token leaves most of the GPU idle.  The row stays in registers between the
// two passes (hidden <= 8192).
constexpr int RB_THREADS = 512;
constexpr int RB_MAXV = 2;  // 8-element vectors per thread

// Router for the token of this CTA.  Leaves the normalised row in `x` (this
// thread's 8-element vectors tid + v*RB_THREADS); writes it as fp16 to xn_row
// unless that is null; warp 0 writes the token's experts and gates.
// One token is all latency, so there is one round of memory and one reduction: the
// row, the norm weights and the first eight experts' router weights are fetched
// together, and the logits are rstd * sum(x * norm_w * router_w), so that they need
// not wait for the norm's own sum.  `loaded` runs once that round is back.
template <typename T, typename F>
__device__ __forceinline__ void router_block_body(const T* __restrict__ row, int d, int E, int k,
                                                  float eps, const float* __restrict__ norm_w,
                                                  const float* __restrict__ rw,
                                                  const float* __restrict__ rb,
                                                  __half* __restrict__ xn_row,
                                                  int32_t* __restrict__ experts_row,
                                                  float* __restrict__ gates_row,
                                                  float (&x)[RB_MAXV][8], F&& loaded) {
  constexpr int WARPS = RB_THREADS / 32;
  __shared__ float s_part[WARPS][9];  // eight logit sums, sum of squares
  __shared__ float s_logit[MAX_EXPERTS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nvec = d / 8;
  float nw[RB_MAXV][8];
  float rstd = 0.f;
  for (int e0 = 0; e0 < E; e0 += 8) {
    float acc[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) acc[e] = 0.f;
#pragma unroll
    for (int v = 0; v < RB_MAXV; ++v) {
      const int j = tid + v * RB_THREADS;
      if (j < nvec) {
        if (e0 == 0) {
          load8<T>(row + j * 8, x[v]);
          load8<float>(norm_w + j * 8, nw[v]);
        }
        float r[8][8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (e0 + e < E) load8<float>(rw + static_cast<size_t>(e0 + e) * d + j * 8, r[e]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          acc[8] = fmaf(x[v][i], x[v][i], acc[8]);
          const float xw = x[v][i] * nw[v][i];
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (e0 + e < E) acc[e] = fmaf(xw, r[e][i], acc[e]);
        }
      }
    }
    {
      const float v = warp_sum8(acc, lane), ss = warp_sum(acc[8]);
      if ((lane & 3) == 0) s_part[warp][warp_sum8_index(lane)] = v;
      if (lane == 0) s_part[warp][8] = ss;
    }
    if (e0 == 0) loaded();
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) tot += s_part[w][8];
    rstd = 1.0f / sqrtf(tot / static_cast<float>(d) + eps);
    if (tid < 8 && e0 + tid < E) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) v += s_part[w][tid];
      s_logit[e0 + tid] = v * rstd + (rb ? rb[e0 + tid] : 0.f);
    }
    if (e0 + 8 < E) __syncthreads();  // s_part is rewritten
  }
#pragma unroll
  for (int v = 0; v < RB_MAXV; ++v) {
    const int j = tid + v * RB_THREADS;
    if (j < nvec) {
#pragma unroll
      for (int i = 0; i < 8; ++i) x[v][i] = nw[v][i] * (x[v][i] * rstd);
      if (xn_row != nullptr) {
        uint32_t packed[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          packed[i] = h2_as_u32(__halves2half2(to_half_sat(x[v][2 * i]), to_half_sat(x[v][2 * i + 1])));
        *reinterpret_cast<uint4*>(xn_row + j * 8) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
      }
    }
  }
  // the logits were written by threads of warp 0, which also selects
  if (warp == 0) {
    __syncwarp();
    router_select(s_logit, lane, E, k, experts_row, gates_row);
  }
}

template <typename T>
__global__ void __launch_bounds__(RB_THREADS)
router_block_kernel(const T* __restrict__ h, int d, int E, int k, float eps,
                    const float* __restrict__ norm_w, const float* __restrict__ rw,
                    const float* __restrict__ rb, __half* __restrict__ xn_out,
                    int32_t* __restrict__ experts_out, float* __restrict__ gates_out) {
  const size_t t = blockIdx.x;
  float x[RB_MAXV][8];
  router_block_body<T>(h + t * d, d, E, k, eps, norm_w, rw, rb, xn_out + t * d,
                       experts_out + t * k, gates_out + t * k, x, [] {});
}

// ------------------------------------------------- fused decode front end
// Router, route plan and row permutation in one cooperative launch, one CTA
// per token (tokens <= FRONT_MAX_TOKENS).  After its token's experts are known
// every CTA meets the others at a grid-wide barrier, ranks its own k pairs
// among all pairs (stable by pair index, as route_plan_kernel does) and stores
// the normalised row, still in registers, at its k sorted positions.  Outputs
// are bit-identical to router_block_kernel + route_plan_kernel +
// permute_rows_kernel; the fp16 copy of the normalised rows is not written.
constexpr int FRONT_MAX_TOKENS = 128;
constexpr int FRONT_MAX_PAIRS = FRONT_MAX_TOKENS * MAX_TOPK;
constexpr int FRONT_PAIRS_PER_THREAD = FRONT_MAX_PAIRS / RB_THREADS;
constexpr int FRONT_SYNC_SLOTS = 32;

// {arrived, departed} per slot; zero between launches (the last CTA to leave
// the barrier resets its slot).  The host hands slots out in rotation, so up to
// FRONT_SYNC_SLOTS launches may be in flight on one device.
__device__ unsigned g_front_sync[FRONT_SYNC_SLOTS][2];

// Bounded grid-wide meeting point for a cooperative launch of `n` CTAs.
// Returns false if the others did not arrive within ~2^31 clock ticks (the
// status word then carries DEV_ERR_WAIT_TIMEOUT and the slot is left for the
// host to clear).
__device__ __forceinline__ bool front_grid_meet(unsigned* sync, unsigned n, int32_t* status) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&sync[0], 1u);
    const long long t0 = clock64();
    int ok = 1;
    while (*reinterpret_cast<volatile unsigned*>(&sync[0]) < n) {
      if (clock64() - t0 > (1ll << 31)) {
        atomicOr(status, DEV_ERR_WAIT_TIMEOUT);
        ok = 0;
        break;
      }
    }
    __threadfence();
    if (ok && atomicAdd(&sync[1], 1u) == n - 1) {
      // everyone has seen arrived == n: nobody reads the slot again
      *reinterpret_cast<volatile unsigned*>(&sync[0]) = 0;
      *reinterpret_cast<volatile unsigned*>(&sync[1]) = 0;
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

template <typename T>
__global__ void __launch_bounds__(RB_THREADS)
front_fused_kernel(const T* __restrict__ h, int d, int E, int k, float eps,
                   const float* __restrict__ norm_w, const float* __restrict__ rw,
                   const float* __restrict__ rb, int32_t* experts_out, float* __restrict__ gates_out,
                   int32_t* __restrict__ counts, int32_t* __restrict__ seg,
                   int32_t* __restrict__ perm, int32_t* __restrict__ inv, int kperm,
                   uint4* __restrict__ xs, unsigned* sync, int32_t* status) {
  __shared__ int s_total[MAX_EXPERTS];
  __shared__ int s_seg[MAX_EXPERTS + 1];
  __shared__ int s_rank[MAX_TOPK];
  const int tid = threadIdx.x;
  const int t = blockIdx.x, tokens = gridDim.x, pairs = tokens * k;
  float x[RB_MAXV][8];
  router_block_body<T>(h + static_cast<size_t>(t) * d, d, E, k, eps, norm_w, rw, rb, nullptr,
                       experts_out + static_cast<size_t>(t) * k, gates_out + static_cast<size_t>(t) * k, x,
                       // gate/up may start once this kernel's own loads are back: its prefetches
                       // then run beside the selection and the barrier, not against the loads
                       [] { grid_dep_launch(); });
  if (tid < MAX_EXPERTS) s_total[tid] = 0;
  if (tid < MAX_TOPK) s_rank[tid] = 0;
  if (!front_grid_meet(sync, static_cast<unsigned>(tokens), status)) return;

  // every CTA sees all pairs; mine are p0 .. p0+k-1
  const int p0 = t * k;
  int mine[MAX_TOPK];
#pragma unroll
  for (int i = 0; i < MAX_TOPK; ++i) mine[i] = i < k ? __ldcg(experts_out + p0 + i) : -1;
  int before[MAX_TOPK];
#pragma unroll
  for (int i = 0; i < MAX_TOPK; ++i) before[i] = 0;
#pragma unroll
  for (int r = 0; r < FRONT_PAIRS_PER_THREAD; ++r) {
    const int q = tid + r * RB_THREADS;
    if (q < pairs) {
      const int e = __ldcg(experts_out + q);
      if (e >= 0 && e < E) atomicAdd(&s_total[e], 1);
#pragma unroll
      for (int i = 0; i < MAX_TOPK; ++i)
        if (i < k && q < p0 + i && e == mine[i]) ++before[i];
    }
  }
#pragma unroll
  for (int i = 0; i < MAX_TOPK; ++i) {
    if (i < k) {
      int c = before[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
      if ((tid & 31) == 0 && c != 0) atomicAdd(&s_rank[i], c);
    }
  }
  __syncthreads();
  if (tid == 0) {
    int run = 0;
    for (int e = 0; e < E; ++e) {
      s_seg[e] = run;
      run += s_total[e];
    }
    s_seg[E] = run;
  }
  __syncthreads();
  if (t == 0 && tid <= E) {
    seg[tid] = s_seg[tid];
    if (tid < E) counts[tid] = s_total[tid];
  }
  int pos[MAX_TOPK];
#pragma unroll
  for (int i = 0; i < MAX_TOPK; ++i) {
    pos[i] = i < k ? s_seg[mine[i]] + s_rank[i] : 0;
    if (i < k && tid == i) {
      perm[pos[i]] = p0 + i;
      inv[p0 + i] = pos[i];
    }
  }
  // the row goes from registers to its k sorted positions
  const int nvec = d / 8;
#pragma unroll
  for (int v = 0; v < RB_MAXV; ++v) {
    const int j = tid + v * RB_THREADS;
    if (j < nvec) {
      uint4 o;
      if (kperm) {  // halves in the order 0,4,1,5,2,6,3,7 (see permute_rows_kernel)
        o.x = h2_as_u32(__halves2half2(to_half_sat(x[v][0]), to_half_sat(x[v][4])));
        o.y = h2_as_u32(__halves2half2(to_half_sat(x[v][1]), to_half_sat(x[v][5])));
        o.z = h2_as_u32(__halves2half2(to_half_sat(x[v][2]), to_half_sat(x[v][6])));
        o.w = h2_as_u32(__halves2half2(to_half_sat(x[v][3]), to_half_sat(x[v][7])));
      } else {
        o.x = h2_as_u32(__halves2half2(to_half_sat(x[v][0]), to_half_sat(x[v][1])));
        o.y = h2_as_u32(__halves2half2(to_half_sat(x[v][2]), to_half_sat(x[v][3])));
        o.z = h2_as_u32(__halves2half2(to_half_sat(x[v][4]), to_half_sat(x[v][5])));
        o.w = h2_as_u32(__halves2half2(to_half_sat(x[v][6]), to_half_sat(x[v][7])));
      }
#pragma unroll
      for (int i = 0; i < MAX_TOPK; ++i) {
        if (i < k) xs[static_cast<size_t>(pos[i]) * nvec + j] = o;
      }
    }
  }
}

// Address of g_front_sync on the current device (cached per device).
static unsigned* front_sync_base() {
  static unsigned* ptrs[16] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) {
    set_error("front: no usable current device");
    return nullptr;
  }
  if (ptrs[dev] == nullptr) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_front_sync);
    if (e != cudaSuccess) {
      cuda_fail(e, "cudaGetSymbolAddress(g_front_sync)");
      return nullptr;
    }
    ptrs[dev] = static_cast<unsigned*>(p);
  }
  return ptrs[dev];
}

bool front_fused_supported(int tokens, const b200moe_layer_t* L) {
  return tokens >= 1 && tokens <= FRONT_MAX_TOKENS && L->hidden <= 8 * RB_THREADS * RB_MAXV &&
         L->hidden % 256 == 0 && L->top_k >= 1 && L->top_k <= MAX_TOPK && L->experts <= MAX_EXPERTS;
}

int launch_front_fused(const void* h, int h_dtype, int tokens, const b200moe_layer_t* L,
                       int32_t* experts, float* gates, int32_t* counts, int32_t* seg,
                       int32_t* perm, int32_t* inv, int kperm, void* xs, int32_t* status,
                       cudaStream_t st) {
  B200_REQUIRE(front_fused_supported(tokens, L), "front: unsupported shape (tokens %d, hidden %d)",
               tokens, L->hidden);
  B200_REQUIRE(L->top_k <= L->experts, "front: top_k (%d) exceeds experts (%d)", L->top_k, L->experts);
  B200_REQUIRE(h_dtype == B200MOE_DT_F32 || h_dtype == B200MOE_DT_BF16,
               "front: activations must be fp32 or bf16");
  static std::atomic<unsigned> next_slot{0};
  unsigned* base = front_sync_base();
  if (base == nullptr) return B200MOE_ERR_CUDA;
  unsigned* sync = base + 2 * (next_slot.fetch_add(1) % FRONT_SYNC_SLOTS);
  int d = L->hidden, E = L->experts, k = L->top_k;
  float eps = L->rms_epsilon;
  const float* norm_w = L->ffn_norm_weight;
  const float* rw = L->router_weight;
  const float* rb = L->router_bias;
  uint4* xs4 = static_cast<uint4*>(xs);
  void* args[] = {&h, &d, &E, &k, &eps, &norm_w, &rw, &rb, &experts, &gates, &counts, &seg,
                  &perm, &inv, &kperm, &xs4, &sync, &status};
  const void* fn = h_dtype == B200MOE_DT_F32
                       ? reinterpret_cast<const void*>(&front_fused_kernel<float>)
                       : reinterpret_cast<const void*>(&front_fused_kernel<__nv_bfloat16>);
  // One CTA meets only itself at the grid barrier: an ordinary launch is enough
  // (and a few microseconds cheaper than a cooperative one) for a single token.
  if (tokens == 1)
    B200_CHECK_CUDA(cudaLaunchKernel(fn, dim3(1), dim3(RB_THREADS), args, 0, st));
  else
    B200_CHECK_CUDA(cudaLaunchCooperativeKernel(fn, dim3(tokens), dim3(RB_THREADS), args, 0, st));
  return B200MOE_OK;
}

int clear_front_sync(cudaStream_t st) {
  unsigned* base = front_sync_base();
  if (base == nullptr) return B200MOE_ERR_CUDA;
  B200_CHECK_CUDA(cudaMemsetAsync(base, 0, sizeof(unsigned) * 2 * FRONT_SYNC_SLOTS, st));
  return B200MOE_OK;
}

// One CTA per token (router_block_kernel) instead of four tokens per CTA.
static bool router_per_token(int tokens, int hidden) { return tokens <= 512 && hidden <= 8 * RB_THREADS * RB_MAXV; }

int launch_router(const void* h, int h_dtype, int tokens, const b200moe_layer_t* L, void* xn,
                  int32_t* experts, float* gates, cudaStream_t st) {
  B200_REQUIRE(L->hidden % 256 == 0, "router: hidden (%d) must be a multiple of 256", L->hidden);
  B200_REQUIRE(L->experts >= 1 && L->experts <= MAX_EXPERTS, "router: experts (%d) must be 1..64",
               L->experts);
  B200_REQUIRE(L->top_k >= 1 && L->top_k <= MAX_TOPK && L->top_k <= L->experts,
               "router: top_k (%d) must be 1..min(8, experts)", L->top_k);
  if (tokens == 0) return B200MOE_OK;
  B200_REQUIRE(h_dtype == B200MOE_DT_F32 || h_dtype == B200MOE_DT_BF16,
               "router: activations must be fp32 or bf16");
  if (router_per_token(tokens, L->hidden)) {
    if (h_dtype == B200MOE_DT_F32)
      router_block_kernel<float><<<tokens, RB_THREADS, 0, st>>>(
          static_cast<const float*>(h), L->hidden, L->experts, L->top_k, L->rms_epsilon,
          L->ffn_norm_weight, L->router_weight, L->router_bias, static_cast<__half*>(xn), experts,
          gates);
    else
      router_block_kernel<__nv_bfloat16><<<tokens, RB_THREADS, 0, st>>>(
          static_cast<const __nv_bfloat16*>(h), L->hidden, L->experts, L->top_k, L->rms_epsilon,
          L->ffn_norm_weight, L->router_weight, L->router_bias, static_cast<__half*>(xn), experts,
          gates);
    B200_CHECK_CUDA(cudaGetLastError());
    return B200MOE_OK;
  }
  const dim3 grid((tokens + RT_TOKENS - 1) / RT_TOKENS), block(RT_THREADS);
  if (h_dtype == B200MOE_DT_F32)
    router_tokens_kernel<float><<<grid, block, 0, st>>>(
        static_cast<const float*>(h), tokens, L->hidden, L->experts, L->top_k, L->rms_epsilon,
        L->ffn_norm_weight, L->router_weight, L->router_bias, static_cast<__half*>(xn), experts, gates, nullptr,
        nullptr);
  else
    router_tokens_kernel<__nv_bfloat16><<<grid, block, 0, st>>>(
        static_cast<const __nv_bfloat16*>(h), tokens, L->hidden, L->experts, L->top_k, L->rms_epsilon,
        L->ffn_norm_weight, L->router_weight, L->router_bias, static_cast<__half*>(xn), experts, gates, nullptr,
        nullptr);
  B200_CHECK_CUDA(cudaGetLastError());
  return B200MOE_OK;
}

// Above the fused front's token count, while the count rows stay small enough to be
// read whole by every CTA of the second kernel, and where router_tokens_kernel has CTAs
// enough: a quarter of the tokens, each with four rows and all router weights to read, are
// slower than one CTA per token until the SMs fill, the later the longer the rows and the
// more experts there are.  Whole call with a small ffn, one B200, us, three kernels (router,
// plan, permutation) / two: hidden 4096, 8 experts, 129 / 256 / 320 / 448 tokens 47.7 / 54.4,
// 56.5 / 59.8, 61.7 / 62.0, 68.5 / 66.5; hidden 6144 256 / 512 tokens 73.7 / 83.7, 104.7 / 104.0;
// hidden 2048, 64 experts, top 8, 129 / 256 / 320 tokens 80.7 / 106, 103.5 / 112, 121 / 115;
// hidden 1024, 8 experts, 160 / 512 tokens 31.0 / 30.4, 46.4 / 40.5.
bool front_prefill_supported(int tokens, const b200moe_layer_t* L) {
  if (router_per_token(tokens, L->hidden) &&
      tokens < static_cast<long long>(L->hidden) * (64 + L->experts) / 832)
    return false;
  return tokens > FRONT_MAX_TOKENS && L->hidden % 256 == 0 && L->experts >= 1 && L->experts <= MAX_EXPERTS &&
         L->top_k >= 1 && L->top_k <= MAX_TOPK && L->top_k <= L->experts &&
         static_cast<long long>((tokens + RT_TOKENS - 1) / RT_TOKENS) * L->experts <= RP_MAX_COUNTS;
}

// Router, plan and permutation of a prefill call in two launches.  `scratch` holds
// tokens floats and the count rows; the caller's fp16 row buffer (tokens * hidden * 2
// bytes, not written on this path) is large enough.
int launch_front_prefill(const void* h, int h_dtype, int tokens, const b200moe_layer_t* L, int32_t* experts,
                         float* gates, int32_t* counts, int32_t* seg, int32_t* perm, int32_t* inv, int kperm,
                         void* xs, void* scratch, cudaStream_t st) {
  B200_REQUIRE(front_prefill_supported(tokens, L), "front: unsupported shape (tokens %d, hidden %d, experts %d)",
               tokens, L->hidden, L->experts);
  B200_REQUIRE(h_dtype == B200MOE_DT_F32 || h_dtype == B200MOE_DT_BF16, "front: activations must be fp32 or bf16");
  float* rstd = static_cast<float*>(scratch);
  int32_t* hist = reinterpret_cast<int32_t*>(rstd + (tokens + 3) / 4 * 4);  // read 16 bytes at a time
  const dim3 rgrid((tokens + RT_TOKENS - 1) / RT_TOKENS), pgrid((tokens + RP_TOKENS - 1) / RP_TOKENS);
#define B200_FRONT(T)                                                                                              \
  router_tokens_kernel<T><<<rgrid, RT_THREADS, 0, st>>>(                                                           \
      static_cast<const T*>(h), tokens, L->hidden, L->experts, L->top_k, L->rms_epsilon, L->ffn_norm_weight,       \
      L->router_weight, L->router_bias, nullptr, experts, gates, rstd, hist);                                      \
  B200_CHECK_CUDA(cudaGetLastError());                                                                             \
  B200_CHECK_CUDA(launch_dependent(route_permute_kernel<T>, pgrid, dim3(RP_THREADS), 0, st,                        \
                                   static_cast<const T*>(h), tokens, L->hidden, L->experts, L->top_k,              \
                                   L->ffn_norm_weight, rstd, experts, hist, counts, seg, perm, inv, kperm,         \
                                   static_cast<uint4*>(xs)));
  if (h_dtype == B200MOE_DT_F32) {
    B200_FRONT(float)
  } else {
    B200_FRONT(__nv_bfloat16)
  }
#undef B200_FRONT
  return B200MOE_OK;
}

// -------------------------------------------------------------- route plan
// Stable counting sort of (token, slot) pairs by expert in one CTA: a shared
// histogram gives the segment offsets, then each 1024-pair chunk ranks its
// pairs with warp match/ballot masks and a per-expert scan over the 32 warps.
constexpr int PLAN_THREADS = 1024;

__global__ void __launch_bounds__(PLAN_THREADS)
route_plan_kernel(const int32_t* __restrict__ experts, int pairs, int e_begin, int E,
                  int32_t* __restrict__ counts, int32_t* __restrict__ seg,
                  int32_t* __restrict__ perm, int32_t* __restrict__ inv) {
  __shared__ int s_total[MAX_EXPERTS];
  __shared__ int s_run[MAX_EXPERTS];
  __shared__ int s_warp[32][MAX_EXPERTS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < MAX_EXPERTS) s_total[tid] = 0;
  __syncthreads();
  for (int p = tid; p < pairs; p += PLAN_THREADS) {
    const int le = experts[p] - e_begin;
    if (le >= 0 && le < E) atomicAdd(&s_total[le], 1);
  }
  __syncthreads();
  if (tid == 0) {
    int run = 0;
    for (int e = 0; e < E; ++e) {
      seg[e] = run;
      counts[e] = s_total[e];
      s_run[e] = run;
      run += s_total[e];
    }
    seg[E] = run;
  }
  __syncthreads();
  for (int base = 0; base < pairs; base += PLAN_THREADS) {
    const int p = base + tid;
    int le = -1;
    if (p < pairs) {
      le = experts[p] - e_begin;
      if (le < 0 || le >= E) le = -1;
    }
    for (int e = lane; e < E; e += 32) s_warp[warp][e] = 0;
    __syncwarp();
    const unsigned peers = __match_any_sync(0xffffffffu, le);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    if (le >= 0 && rank == 0) s_warp[warp][le] = __popc(peers);
    __syncthreads();
    if (tid < E) {
      int run = s_run[tid];
      for (int w = 0; w < 32; ++w) {
        const int c = s_warp[w][tid];
        s_warp[w][tid] = run;
        run += c;
      }
      s_run[tid] = run;
    }
    __syncthreads();
    if (p < pairs) {
      if (le >= 0) {
        const int pos = s_warp[warp][le] + rank;
        perm[pos] = p;
        inv[p] = pos;
      } else {
        inv[p] = -1;
      }
    }
    __syncthreads();
  }
}

int launch_route_plan(const int32_t* experts, int pairs, int e_begin, int E, int32_t* counts,
                      int32_t* seg, int32_t* perm, int32_t* inv, cudaStream_t st) {
  B200_REQUIRE(E >= 1 && E <= MAX_EXPERTS, "route_plan: local experts (%d) must be 1..64", E);
  B200_REQUIRE(pairs >= 0, "route_plan: negative pair count");
  route_plan_kernel<<<1, PLAN_THREADS, 0, st>>>(experts, pairs, e_begin, E, counts, seg, perm, inv);
  B200_CHECK_CUDA(cudaGetLastError());
  return B200MOE_OK;
}

// ------------------------------------------------------------ permute rows
// xs[pos,:] = xn[perm[pos]/k,:].  With kperm the eight halves of every 16-byte
// group are written in the order 0,4,1,5,2,6,3,7 — the order in which the Q4_K
// kernels pull nibble pairs out of a 32-bit word.
__global__ void __launch_bounds__(128)
permute_rows_kernel(const uint4* __restrict__ xn, const int32_t* __restrict__ perm,
                    const int32_t* __restrict__ seg, int E, int k, int vec_per_row, int kperm,
                    uint4* __restrict__ xs) {
  const int pos = blockIdx.x;
  if (pos >= seg[E]) return;
  const int tok = perm[pos] / k;
  const uint4* src = xn + static_cast<size_t>(tok) * vec_per_row;
  uint4* dst = xs + static_cast<size_t>(pos) * vec_per_row;
  for (int j = threadIdx.x; j < vec_per_row; j += blockDim.x) {
    uint4 v = src[j];
    if (kperm) {
      uint4 o;
      o.x = __byte_perm(v.x, v.z, 0x5410);  // (h0, h4)
      o.y = __byte_perm(v.x, v.z, 0x7632);  // (h1, h5)
      o.z = __byte_perm(v.y, v.w, 0x5410);  // (h2, h6)
      o.w = __byte_perm(v.y, v.w, 0x7632);  // (h3, h7)
      v = o;
    }
    dst[j] = v;
  }
}

int launch_permute_rows(const void* xn, const int32_t* perm, const int32_t* seg, int E, int pairs,
                        int k, int d, int kperm, void* xs, cudaStream_t st) {
  B200_REQUIRE(d % 8 == 0, "permute_rows: hidden must be a multiple of 8");
  if (pairs == 0) return B200MOE_OK;
  permute_rows_kernel<<<pairs, 128, 0, st>>>(static_cast<const uint4*>(xn), perm, seg, E, k,
                                             d / 8, kperm, static_cast<uint4*>(xs));
  B200_CHECK_CUDA(cudaGetLastError());
  return B200MOE_OK;
}

// --------------------------------------------------- exchange plan (EP)
// Rows arrive from `world` source ranks, each rank's rows ordered by local
// expert: arrival order is (source, expert) blocks, the kernels want (expert,
// source) blocks.  counts[s*el + e] = rows from source s for local expert e.
// One CTA computes the segment offsets and both permutations.
__global__ void __launch_bounds__(1024)
exchange_plan_kernel(const int32_t* __restrict__ counts, int world, int el,
                     int32_t* __restrict__ seg, int32_t* __restrict__ perm,
                     int32_t* __restrict__ inv) {
  __shared__ int s_arr[MAX_EXPERTS * MAX_EXPERTS];  // arrival offset of block (s, e)
  __shared__ int s_srt[MAX_EXPERTS * MAX_EXPERTS];  // sorted offset of block (s, e)
  const int nb = world * el;
  if (threadIdx.x == 0) {
    int run = 0;
    for (int b = 0; b < nb; ++b) { s_arr[b] = run; run += counts[b]; }
    run = 0;
    for (int e = 0; e < el; ++e) {
      seg[e] = run;
      for (int s = 0; s < world; ++s) { s_srt[s * el + e] = run; run += counts[s * el + e]; }
    }
    seg[el] = run;
  }
  __syncthreads();
  for (int b = 0; b < nb; ++b) {
    const int c = counts[b], a0 = s_arr[b], p0 = s_srt[b];
    for (int i = threadIdx.x; i < c; i += blockDim.x) {
      perm[p0 + i] = a0 + i;
      inv[a0 + i] = p0 + i;
    }
  }
}

int launch_exchange_plan(const int32_t* counts, int world, int el, int32_t* seg, int32_t* perm,
                         int32_t* inv, cudaStream_t st) {
  B200_REQUIRE(world >= 1 && el >= 1 && world * el <= MAX_EXPERTS * MAX_EXPERTS && el <= MAX_EXPERTS,
               "exchange_plan: %d ranks x %d local experts out of range", world, el);
  exchange_plan_kernel<<<1, 1024, 0, st>>>(counts, world, el, seg, perm, inv);
  B200_CHECK_CUDA(cudaGetLastError());
  return B200MOE_OK;
}

// out[i,:] = rows[idx[i] / div,:] for i < n; rows of `vec_per_row` 16-byte vectors.
__global__ void __launch_bounds__(128)
gather_rows_kernel(const uint4* __restrict__ rows, const int32_t* __restrict__ idx, int div,
                   int vec_per_row, uint4* __restrict__ out) {
  const int i = blockIdx.x;
  const uint4* src = rows + static_cast<size_t>(idx[i] / div) * vec_per_row;
  uint4* dst = out + static_cast<size_t>(i) * vec_per_row;
  for (int j = threadIdx.x; j < vec_per_row; j += blockDim.x) dst[j] = src[j];
}

int launch_gather_rows(const void* rows, const int32_t* idx, int n, int div, int row_bytes,
                       void* out, cudaStream_t st) {
  B200_REQUIRE(row_bytes % 16 == 0 && div >= 1, "gather_rows: rows must be multiples of 16 bytes");
  if (n == 0) return B200MOE_OK;
  gather_rows_kernel<<<n, 128, 0, st>>>(static_cast<const uint4*>(rows), idx, div, row_bytes / 16,
                                        static_cast<uint4*>(out));
  B200_CHECK_CUDA(cudaGetLastError());
  return B200MOE_OK;
}

// ----------------------------------------------------------------- combine
// One CTA per token: sum over slots (in slot order) of gate * (sum of the
// k-split partials of the pair's down-projection row), optional output RMS
// norm, residual add.
template <typename T>
__device__ __forceinline__ float load1(const T* p);
template <>
__device__ __forceinline__ float load1<float>(const float* p) { return *p; }
template <>
__device__ __forceinline__ float load1<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}
template <typename T>
__device__ __forceinline__ void store1(T* p, float v);
template <>
__device__ __forceinline__ void store1<float>(float* p, float v) { *p = v; }
template <>
__device__ __forceinline__ void store1<__nv_bfloat16>(__nv_bfloat16* p, float v) {
  *p = __float2bfloat16_rn(v);
}

constexpr int COMBINE_THREADS = 256;

// four consecutive elements at once (16-byte / 8-byte accesses)
template <typename T>
__device__ __forceinline__ void load4(const T* p, float (&v)[4]);
template <>
__device__ __forceinline__ void load4<float>(const float* p, float (&v)[4]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
template <>
__device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[4]) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  v[0] = __uint_as_float(raw.x << 16);
  v[1] = __uint_as_float(raw.x & 0xffff0000u);
  v[2] = __uint_as_float(raw.y << 16);
  v[3] = __uint_as_float(raw.y & 0xffff0000u);
}
template <typename T>
__device__ __forceinline__ void store4(T* p, const float (&v)[4]);
template <>
__device__ __forceinline__ void store4<float>(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
template <>
__device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, const float (&v)[4]) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]);
  const __nv_bfloat162 hi = __floats2bfloat162_rn(v[2], v[3]);
  uint2 raw;
  raw.x = *reinterpret_cast<const uint32_t*>(&lo);
  raw.y = *reinterpret_cast<const uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = raw;
}

// gate-weighted sum over the token's slots for four columns; per element the
// same operations in the same order as a scalar loop over slots and partials
template <typename TD>
__device__ __forceinline__ void combine4(const TD* dpart, int ksplit, size_t part_stride,
                                         const int (&pos)[MAX_TOPK], const float (&gate)[MAX_TOPK],
                                         int k, int d, int j, float (&acc)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] = 0.f;
#pragma unroll
  for (int s = 0; s < MAX_TOPK; ++s) {
    if (s < k && pos[s] >= 0) {
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      for (int c = 0; c < ksplit; ++c) {
        float p4[4];
        load4<TD>(dpart + c * part_stride + static_cast<size_t>(pos[s]) * d + j, p4);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] += p4[i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] += gate[s] * v[i];
    }
  }
}

template <typename TD, typename TH, typename TY>
__global__ void __launch_bounds__(COMBINE_THREADS)
combine_kernel(const TD* dpart, int ksplit, size_t part_stride, const int32_t* inv, const float* gates,
               const TH* __restrict__ h, int d, int k, const float* __restrict__ out_norm_w,
               float eps, int add_residual, TY* __restrict__ y) {
  extern __shared__ float s_row[];
  __shared__ float s_red[COMBINE_THREADS / 32];
  const size_t t = blockIdx.x;
  int pos[MAX_TOPK];
  float gate[MAX_TOPK];
  grid_dep_wait();
#pragma unroll
  for (int s = 0; s < MAX_TOPK; ++s) {
    pos[s] = s < k ? inv[t * k + s] : -1;
    gate[s] = s < k ? gates[t * k + s] : 0.f;
  }
  if (gridDim.y > 1) {
    // no output norm: column slices are independent, one slice per blockIdx.y
    const int per = ((d / 4 + gridDim.y - 1) / gridDim.y) * 4;
    const int j0 = blockIdx.y * per, j1 = min(d, j0 + per);
    for (int j = j0 + threadIdx.x * 4; j < j1; j += COMBINE_THREADS * 4) {
      float acc[4];
      combine4<TD>(dpart, ksplit, part_stride, pos, gate, k, d, j, acc);
      if (add_residual) {
        float r[4];
        load4<TH>(h + t * d + j, r);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] += r[i];
      }
      store4<TY>(y + t * d + j, acc);
    }
    return;
  }
  float ss = 0.f;
  for (int j = threadIdx.x * 4; j < d; j += COMBINE_THREADS * 4) {
    float acc[4];
    combine4<TD>(dpart, ksplit, part_stride, pos, gate, k, d, j, acc);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s_row[j + i] = acc[i];
      ss = fmaf(acc[i], acc[i], ss);
    }
  }
  float scale = 1.f;
  if (out_norm_w != nullptr && add_residual) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
    for (int w = 0; w < COMBINE_THREADS / 32; ++w) tot += s_red[w];
    scale = 1.0f / sqrtf(tot / static_cast<float>(d) + eps);
  }
  // every thread re-reads only the columns it wrote itself
  for (int j = threadIdx.x * 4; j < d; j += COMBINE_THREADS * 4) {
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = s_row[j + i];
    if (add_residual) {
      float r[4];
      load4<TH>(h + t * d + j, r);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (out_norm_w != nullptr) v[i] = out_norm_w[j + i] * (v[i] * scale);
        v[i] += r[i];
      }
    }
    store4<TY>(y + t * d + j, v);
  }
}

int launch_combine(const void* dpart, int d_dtype, int ksplit, int pairs, const int32_t* inv,
                   const float* gates, const void* h, int h_dtype, int tokens,
                   const b200moe_layer_t* L, int add_residual, void* y, int y_dtype,
                   cudaStream_t st) {
  if (tokens == 0) return B200MOE_OK;
  const int d = L->hidden, k = L->top_k;
  const size_t smem = static_cast<size_t>(d) * sizeof(float);
  B200_REQUIRE(smem <= 48 * 1024, "combine: hidden (%d) too large", d);
  B200_REQUIRE(d % 4 == 0 && k >= 1 && k <= MAX_TOPK, "combine: hidden must be a multiple of 4, top_k 1..8");
  const size_t stride = static_cast<size_t>(pairs) * d;
  const bool need_row = L->layer_output_norm_weight != nullptr && add_residual;
  int slices = 1;
  if (!need_row && tokens < 1024) slices = max(1, min(d / COMBINE_THREADS, 2048 / tokens));
  dim3 grid(tokens, slices), block(COMBINE_THREADS);
#define LAUNCH(TD, TH, TY)                                                                     \
  B200_CHECK_CUDA(launch_dependent(combine_kernel<TD, TH, TY>, grid, block, smem, st,             \
                                   static_cast<const TD*>(dpart), ksplit, stride, inv, gates,     \
                                   static_cast<const TH*>(h), d, k, L->layer_output_norm_weight,  \
                                   L->rms_epsilon, add_residual, static_cast<TY*>(y)))
  const bool dbf = d_dtype == B200MOE_DT_BF16;
  B200_REQUIRE(dbf || d_dtype == B200MOE_DT_F32, "combine: partial rows must be fp32 or bf16");
  if (h_dtype == B200MOE_DT_F32 && y_dtype == B200MOE_DT_F32) {
    if (dbf) LAUNCH(__nv_bfloat16, float, float); else LAUNCH(float, float, float);
  } else if (h_dtype == B200MOE_DT_BF16 && y_dtype == B200MOE_DT_BF16) {
    if (dbf) LAUNCH(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16); else LAUNCH(float, __nv_bfloat16, __nv_bfloat16);
  } else if (h_dtype == B200MOE_DT_BF16 && y_dtype == B200MOE_DT_F32) {
    if (dbf) LAUNCH(__nv_bfloat16, __nv_bfloat16, float); else LAUNCH(float, __nv_bfloat16, float);
  } else {
    B200_REQUIRE(false, "combine: unsupported dtype pair (%d, %d)", h_dtype, y_dtype);
  }
#undef LAUNCH
  B200_CHECK_CUDA(cudaGetLastError());
  return B200MOE_OK;
}

// ----------------------------------------------------- reference dequantise
template <typename TO>
__global__ void dequant_q8_kernel(const int8_t* __restrict__ qs, const __half* __restrict__ d,
                                  size_t n, TO* __restrict__ out) {
  const size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const __half scale = d[i >> 5];
  if constexpr (sizeof(TO) == 2) {
    out[i] = __hmul(scale, __int2half_rn(qs[i]));
  } else {
    out[i] = __half2float(scale) * static_cast<float>(qs[i]);
  }
}

template <typename TO>
__global__ void dequant_q4k_kernel(const uint8_t* __restrict__ qs, const __half2* __restrict__ sub,
                                   size_t n, TO* __restrict__ out) {
  const size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const uint8_t b = qs[i >> 1];
  const int q = (i & 1) ? (b >> 4) : (b & 0xF);
  const __half2 sm = sub[i >> 5];
  // the _rn forms are never contracted into an fma: the reference rounds after
  // the product and again after the subtraction
  const __half w = __hsub_rn(__hmul_rn(__low2half(sm), __int2half_rn(q)), __high2half(sm));
  if constexpr (sizeof(TO) == 2) {
    out[i] = w;
  } else {
    out[i] = __half2float(w);
  }
}

template <typename TO>
__global__ void dequant_f16_kernel(const __half* __restrict__ w, size_t n, TO* __restrict__ out) {
  const size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  if constexpr (sizeof(TO) == 2) {
    out[i] = w[i];
  } else {
    out[i] = __half2float(w[i]);
  }
}

int launch_dequant(const b200moe_weight_t* w, int out_dtype, void* out, cudaStream_t st) {
  B200_REQUIRE(out_dtype == B200MOE_DT_F16 || out_dtype == B200MOE_DT_F32,
               "dequant: out_dtype must be fp16 or fp32");
  const size_t n = static_cast<size_t>(w->experts) * w->rows * w->cols;
  if (n == 0) return B200MOE_OK;
  const int threads = 256;
  const unsigned blocks = static_cast<unsigned>((n + threads - 1) / threads);
  const bool f16 = out_dtype == B200MOE_DT_F16;
  switch (w->layout) {
    case B200MOE_LAYOUT_Q8_0:
      B200_REQUIRE(w->cols % 32 == 0, "dequant: Q8_0 needs cols %% 32 == 0");
      if (f16)
        dequant_q8_kernel<__half><<<blocks, threads, 0, st>>>(
            static_cast<const int8_t*>(w->qs), static_cast<const __half*>(w->d), n,
            static_cast<__half*>(out));
      else
        dequant_q8_kernel<float><<<blocks, threads, 0, st>>>(
            static_cast<const int8_t*>(w->qs), static_cast<const __half*>(w->d), n,
            static_cast<float*>(out));
      break;
    case B200MOE_LAYOUT_Q4_K:
      B200_REQUIRE(w->cols % 256 == 0, "dequant: Q4_K needs cols %% 256 == 0");
      if (f16)
        dequant_q4k_kernel<__half><<<blocks, threads, 0, st>>>(
            static_cast<const uint8_t*>(w->qs), static_cast<const __half2*>(w->sub), n,
            static_cast<__half*>(out));
      else
        dequant_q4k_kernel<float><<<blocks, threads, 0, st>>>(
            static_cast<const uint8_t*>(w->qs), static_cast<const __half2*>(w->sub), n,
            static_cast<float*>(out));
      break;
    case B200MOE_LAYOUT_F16:
      if (f16)
        dequant_f16_kernel<__half><<<blocks, threads, 0, st>>>(static_cast<const __half*>(w->qs),
                                                               n, static_cast<__half*>(out));
      else
        dequant_f16_kernel<float><<<blocks, threads, 0, st>>>(static_cast<const __half*>(w->qs),
                                                              n, static_cast<float*>(out));
      break;
    default:
      B200_REQUIRE(false, "dequant: unknown layout %d", w->layout);
  }
  B200_CHECK_CUDA(cudaGetLastError());
  return B200MOE_OK;
}

// ------------------------------------------------- Q8_0 scale transposition
// d [rows, K/32] -> [K/256][rows][8]: the eight scales one row needs for a
// 256-k stage become 16 contiguous bytes and consecutive rows are adjacent, so
// a stage's scale tile is one contiguous run (one bulk copy instead of one
// 16-byte TMA request per row).
__global__ void q8_scales_tile_kernel(const uint4* __restrict__ d, long long rows, int groups,
                                      uint4* __restrict__ out) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i >= rows * groups) return;
  const long long r = i / groups;
  const int g = static_cast<int>(i % groups);
  out[static_cast<long long>(g) * rows + r] = d[i];
}

int launch_q8_prepare(const void* d, long long rows, int cols, void* out, cudaStream_t st) {
  B200_REQUIRE(cols % 256 == 0, "q8_prepare: cols (%d) must be a multiple of 256", cols);
  const int groups = cols / 256;
  const long long n = rows * groups;
  if (n == 0) return B200MOE_OK;
  q8_scales_tile_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(
      static_cast<const uint4*>(d), rows, groups, static_cast<uint4*>(out));
  B200_CHECK_CUDA(cudaGetLastError());
  return B200MOE_OK;
}

// --------------------------------------------------------- Q4_K scale fold
// One thread per super-block: the eight 6-bit sub-scales / sub-mins
// (low nibble plane | 2-bit high plane << 4) times d / dmin, each product
// rounded once to fp16.
__global__ void q4k_prepare_kernel(const __half* __restrict__ d, const __half* __restrict__ dmin,
                                   const uint8_t* __restrict__ sh, const uint8_t* __restrict__ sl,
                                   const uint8_t* __restrict__ mh, const uint8_t* __restrict__ ml,
                                   long long blocks, __half2* __restrict__ sub) {
  const long long b = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (b >= blocks) return;
  const __half dd = d[b], dm = dmin[b];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int sc = ((sl[b * 4 + (i >> 1)] >> ((i & 1) * 4)) & 0xF) |
                   (((sh[b * 2 + (i >> 2)] >> ((i & 3) * 2)) & 3) << 4);
    const int mn = ((ml[b * 4 + (i >> 1)] >> ((i & 1) * 4)) & 0xF) |
                   (((mh[b * 2 + (i >> 2)] >> ((i & 3) * 2)) & 3) << 4);
    sub[b * 8 + i] = __halves2half2(__hmul(dd, __int2half_rn(sc)), __hmul(dm, __int2half_rn(mn)));
  }
}

int launch_q4k_prepare(const void* d, const void* dmin, const uint8_t* sh, const uint8_t* sl,
                       const uint8_t* mh, const uint8_t* ml, long long blocks, void* sub,
                       cudaStream_t st) {
  if (blocks == 0) return B200MOE_OK;
  const int threads = 256;
  q4k_prepare_kernel<<<static_cast<unsigned>((blocks + threads - 1) / threads), threads, 0, st>>>(
      static_cast<const __half*>(d), static_cast<const __half*>(dmin), sh, sl, mh, ml, blocks,
      static_cast<__half2*>(sub));
  B200_CHECK_CUDA(cudaGetLastError());
  return B200MOE_OK;
}

// ------------------------------------------------------------- GGUF unpack
// Q8_0 file block: fp16 scale + 32 int8.  One thread per quant.
__global__ void gguf_q8_kernel(const uint8_t* __restrict__ raw, long long blocks,
                               uint16_t* __restrict__ d, int8_t* __restrict__ qs) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i >= blocks * 32) return;
  const long long b = i >> 5;
  const int j = static_cast<int>(i & 31);
  const uint8_t* blk = raw + b * 34;
  qs[i] = static_cast<int8_t>(blk[2 + j]);
  if (j == 0) d[b] = static_cast<uint16_t>(blk[0]) | (static_cast<uint16_t>(blk[1]) << 8);
}

// Q4_K file super-block (144 B): d, dmin, 12 bytes of 6-bit fields, 128 bytes
// of nibbles.  One thread per super-block writes the planar planes.
__global__ void gguf_q4k_kernel(const uint8_t* __restrict__ raw, long long blocks,
                                uint16_t* __restrict__ d, uint16_t* __restrict__ dmin,
                                uint8_t* __restrict__ sh, uint8_t* __restrict__ sl,
                                uint8_t* __restrict__ mh, uint8_t* __restrict__ ml,
                                uint8_t* __restrict__ qs) {
  const long long b = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (b >= blocks) return;
  const uint8_t* blk = raw + b * 144;
  d[b] = static_cast<uint16_t>(blk[0]) | (static_cast<uint16_t>(blk[1]) << 8);
  dmin[b] = static_cast<uint16_t>(blk[2]) | (static_cast<uint16_t>(blk[3]) << 8);
  const uint8_t* s = blk + 4;
  uint8_t sc[8], mn[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    sc[i] = s[i] & 63;
    mn[i] = s[i + 4] & 63;
    sc[i + 4] = (s[i + 8] & 0xF) | ((s[i] >> 6) << 4);
    mn[i + 4] = (s[i + 8] >> 4) | ((s[i + 4] >> 6) << 4);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    sl[b * 4 + j] = (sc[2 * j] & 0xF) | ((sc[2 * j + 1] & 0xF) << 4);
    ml[b * 4 + j] = (mn[2 * j] & 0xF) | ((mn[2 * j + 1] & 0xF) << 4);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    sh[b * 2 + j] = (sc[4 * j] >> 4) | ((sc[4 * j + 1] >> 4) << 2) | ((sc[4 * j + 2] >> 4) << 4) |
                    ((sc[4 * j + 3] >> 4) << 6);
    mh[b * 2 + j] = (mn[4 * j] >> 4) | ((mn[4 * j + 1] >> 4) << 2) | ((mn[4 * j + 2] >> 4) << 4) |
                    ((mn[4 * j + 3] >> 4) << 6);
  }
  const uint8_t* q = blk + 16;
  uint8_t* o = qs + b * 128;
  for (int g = 0; g < 4; ++g) {
    for (int i = 0; i < 16; ++i) {
      const uint8_t a = q[32 * g + 2 * i], c = q[32 * g + 2 * i + 1];
      o[(2 * g) * 16 + i] = (a & 0xF) | ((c & 0xF) << 4);
      o[(2 * g + 1) * 16 + i] = (a >> 4) | ((c >> 4) << 4);
    }
  }
}

int launch_gguf_q8(const uint8_t* raw, long long blocks, void* d, int8_t* qs, cudaStream_t st) {
  if (blocks == 0) return B200MOE_OK;
  const long long n = blocks * 32;
  gguf_q8_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(
      raw, blocks, static_cast<uint16_t*>(d), qs);
  B200_CHECK_CUDA(cudaGetLastError());
  return B200MOE_OK;
}

int launch_gguf_q4k(const uint8_t* raw, long long blocks, void* d, void* dmin, uint8_t* sh,
                    uint8_t* sl, uint8_t* mh, uint8_t* ml, uint8_t* qs, cudaStream_t st) {
  if (blocks == 0) return B200MOE_OK;
  gguf_q4k_kernel<<<static_cast<unsigned>((blocks + 127) / 128), 128, 0, st>>>(
      raw, blocks, static_cast<uint16_t*>(d), static_cast<uint16_t*>(dmin), sh, sl, mh, ml, qs);
  B200_CHECK_CUDA(cudaGetLastError());
  return B200MOE_OK;
}

}  // namespace b200moe
