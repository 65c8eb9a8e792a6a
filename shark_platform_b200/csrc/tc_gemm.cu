// Tensor-core grouped expert GEMM for the prefill regime (many tokens per
// expert): tcgen05.mma with fp32 accumulators in tensor memory.
//
// Orientation is "swap-AB" with the A operand in tensor memory: a tile of 128
// weight rows is M, up to 192 tokens of one expert are N.  Weights never touch
// shared memory in dequantised form: warps read the TMA-staged quantised bytes
// (one thread per weight row), dequantise to fp16 in registers and write the
// row into tensor memory with tcgen05.st, where it is the A operand of the next
// MMAs.  The token rows (fp16, K-major, 128-byte swizzle) are the B operand, read
// from shared memory through a matrix descriptor.  Shared memory therefore only
// carries quantised bytes and token tiles.
//
// A CTA holds two row sets per tile, each with its own accumulator:
// gate rows + up rows of the same 128 columns (SiLU/GELU-gated product in the
// epilogue), or 256 consecutive rows of the down matrix.
//
// Three independent shared-memory rings, because their slots live for very
// different times:
//   weights  2, 4 or 5 slots x (2 sets x 128 rows x 128 k) int8, 128-byte swizzle;
//            a slot is free again as soon as the dequant warps have read it
//   tokens   2 or 3 slots x (64, 128 or 192 rows x 128 k) fp16; a slot is held until
//            the MMAs that read it have completed
//   scales   2 slots x (2 sets x 128 rows x 8) fp16 = 256 k
//
// Warp roles (608 threads, one CTA per SM, persistent over tiles):
//   warps 0-7   group 0: dequantise the even 64-k stages (warps 0-3 set 0,
//               warps 4-7 set 1; warp w owns TMEM lanes 32(w%4)..+31), epilogue
//   warps 8-15  group 1: the same for the odd stages, so that one group's
//               tensor-memory store latency hides behind the other's arithmetic
//               (the 64- and 128-token variants hand over two stages at a time:
//               group g takes every second 128-k weight slot whole)
//   warp  16    TMA producer for weights and scales
//   warp  17    TMA producer for token tiles
//   warp  18    TMEM allocation; issues the MMAs of row set 0 and commits
//   warp  19    issues the MMAs of row set 1
// The MMAs are issued by an elected lane (elect.sync) of a converged warp.  Issued
// under `if (lane == 0)` instead, an MMA costs its thread ~70 clocks and the loop
// took 1055 clocks per 64-k stage where the tensor pipe needs 704: the compiler
// cannot know that one lane is active and guards the instruction's uniform
// operands.  Measured, one B200, us per launch, gate/up + down: 4096 tokens Q8_0
// 1618 + 873 -> 1500 + 804, 2048 tokens Q4_K 942 + 482 -> 840 + 428, 128 tokens Q8_0
// 250 + 129 -> 209 + 110.
// Each row set has its own A-slot barriers, so the two sets are independent
// pipelines that share only the token tiles.
//
// Tensor-memory columns (512 allocated): accumulators at 0 and 192 (192 fp32
// columns each), two A staging slots of 2 x 32 columns at 384..511.
//
// All mbarrier waits are bounded; on expiry the CTA raises its abort flag, every
// role falls out of its loops, its copies and MMAs in flight are waited for (bounded,
// mbar_drain), the CTA frees its tensor memory and returns.
#include <math.h>

#include "common.cuh"

namespace b200moe {
namespace {

constexpr int TC_DQ_WARPS = 16;
constexpr int TC_WARP_WPROD = TC_DQ_WARPS;
constexpr int TC_WARP_XPROD = TC_DQ_WARPS + 1;
constexpr int TC_WARP_MMA = TC_DQ_WARPS + 2;   // issues the MMAs of row set 0 (and owns the TMEM allocation)
constexpr int TC_WARP_MMA1 = TC_DQ_WARPS + 3;  // issues the MMAs of row set 1
constexpr int TC_THREADS = (TC_DQ_WARPS + 4) * 32;
constexpr int TC_KT = 64;            // k per stage (one token slot, one A slot)
constexpr int TC_ROWS = 128;         // weight rows per set
constexpr int TC_NTOK = 192;         // largest token tile / accumulator width
constexpr int TC_MAX_E = 64;
constexpr int TC_WSET = TC_ROWS * 128;          // bytes of one set in a weight slot (128 k)
constexpr int TC_WSLOT = 2 * TC_WSET;
constexpr int TC_SGROUP = 4;                    // stages covered by one scale tile (256 k)
constexpr int TC_SSLOTS = 2;
constexpr int TC_SSET = TC_ROWS * 32;           // per row and group: 8 fp16 scales (Q8_0, 16 B used) or 8 half2 scale/min pairs (Q4_K)
constexpr int TC_SSLOT = 2 * TC_SSET;

// Geometry for token tiles of at most NMAX rows.  The two accumulators take
// 2 x NMAX tensor-memory columns; what is left of the 512 holds A staging slots
// of 64 columns, so narrow tiles get a deeper A ring (the MMA lane and the
// dequant warps then rarely wait for each other) and, because their token slots
// are small, a deeper weight ring (more bytes in flight per SM, which is what a
// weight-streaming tile needs).
template <int NMAX>
struct TcCfg {
  static_assert(NMAX == 64 || NMAX == 128 || NMAX == 192, "token tile widths: 64, 128, 192");
  static constexpr int ASLOTS = (512 - 2 * NMAX) / 64;  // 6, 4, 2 stages of 64 k
  // stages per hand-over from the dequant warps to the issuers: two where the ring
  // holds more than two, which halves the waits, votes, fences and arrivals per
  // weight on both sides
  static constexpr int HK = NMAX <= 128 ? 2 : 1;
  static constexpr int HSLOTS = ASLOTS / HK;            // 3, 2, 2
  static constexpr int WSLOTS = NMAX == 192 ? 2 : NMAX == 128 ? 4 : 5;
  // With HK = 2 a group waits on every second weight fill only.  An even ring keeps each
  // slot with one group.  In an odd one the slots change groups, and a wait by parity
  // also passes when the other group's fill of the slot, WSLOTS fills ago, has not landed
  // yet.  What then vouches for that fill is the group's last hand-over, two fills ago: it
  // needed the MMAs of the hand-over HSLOTS before it.  (Three slots with two hand-over
  // slots broke this rule: stale weights, arrivals on a used-up phase.)
  // What 128-token tiles could take instead: one-stage hand-overs with three weight and
  // three token slots.  One B200, Q8_0, gate/up + down, us, 4 + 2 slots as here / that:
  // 200 tokens 237 + 115 / 244 + 126, 320 tokens 267 + 135 / 261 + 131, 387 tokens
  // 296 + 140 / 278 + 136; q, k and v of 41 to 96 rows 16.5 .. 21.2 / 17.9 .. 21.7.
  static_assert(HK == 1 || WSLOTS % 2 == 0 || HSLOTS + 2 <= WSLOTS, "a group could pass a slot that is still being filled");
  // a token slot holds two 64-k stages (two swizzled sub-tiles of NMAX rows x 128 B):
  // one wait and one release per 128 k on the issuing lanes, whose instruction
  // stream is the kernel's critical path
  static constexpr int XSLOTS = NMAX == 128 ? 2 : 3;
  static constexpr int XSUB = NMAX * TC_KT * 2;
  static constexpr int XSLOT = 2 * XSUB;
  static constexpr int OFF_X = WSLOTS * TC_WSLOT;
  static constexpr int OFF_S = OFF_X + XSLOTS * XSLOT;
  static constexpr int OFF_BAR = OFF_S + TC_SSLOTS * TC_SSLOT;
  static constexpr int SMEM = 1024 + OFF_BAR + 512;
  static constexpr uint32_t COL_ACC0 = 0, COL_ACC1 = NMAX, COL_A = 2 * NMAX;
  static_assert(XSLOT % 1024 == 0 && TC_WSLOT % 1024 == 0, "slot alignment for the swizzle");
  static_assert(SMEM <= 232448, "shared memory budget");
  static_assert(2 * (WSLOTS + XSLOTS + TC_SSLOTS + 2 * HSLOTS) + 4 <= 64, "barrier area");
};

struct TcArgs {
  const int32_t* seg;
  int E, N, K;
  int row_tile;    // weight rows per set (96, 112 or 128): tc_row_tile
  int ntiles;      // row tiles per expert (N / row_tile for gate+up, N / 256 for down)
  int tok_tile;    // upper bound on tokens per tile (multiple of 16, <= 192)
  int ksplit;      // k partitions per tile (down only); partial kc goes to out + kc*P*N
  int P;
  int act;
  int out_kperm;   // gate/up only: interleave output columns for a Q4_K down matrix
  int prefetch;    // PREFETCH_*
  void* out;
  int32_t* status;
  // scales transposed to [K/256][rows][8] (one contiguous run per row tile and
  // 256-k group) or NULL = fetch them from `d` as 16-byte TMA rows
  const uint8_t* st0;
  const uint8_t* st1;
  long long total_rows;
  // NMAT == 3: up to three matrices over the same rows [seg[0], seg[1]), matrix e in
  // the place of expert e (E of them) with its own row count, output and scales
  int mtiles[3];
  int mrows[3];
  float* mout[3];
  const uint8_t* mst[3];
  // with an unsplit k the finished values go out at once: mdst[e] of type mdtype, the
  // residual (of that type) added to matrix 0; else mout[e] gets fp32 partial sums
  void* mdst[3];
  int mdtype;
  const void* residual;
};

__device__ __forceinline__ float tc_load_residual(const void* p, int dt, size_t i) {
  if (dt == B200MOE_DT_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
  if (dt == B200MOE_DT_F16) return __half2float(static_cast<const __half*>(p)[i]);
  return static_cast<const float*>(p)[i];
}
// y rounded to its type and, with a residual, the sum rounded again (`h + y` on tensors).
__device__ __forceinline__ void tc_store_linear(void* dst, int dt, bool add, float residual, size_t i, float v) {
  if (dt == B200MOE_DT_BF16) {
    __nv_bfloat16 r = __float2bfloat16_rn(v);
    if (add) r = __float2bfloat16_rn(residual + __bfloat162float(r));
    static_cast<__nv_bfloat16*>(dst)[i] = r;
  } else if (dt == B200MOE_DT_F16) {
    __half r = __float2half_rn(v);
    if (add) r = __float2half_rn(residual + __half2float(r));
    static_cast<__half*>(dst)[i] = r;
  } else {
    static_cast<float*>(dst)[i] = add ? residual + v : v;
  }
}

__device__ __forceinline__ void tc_bulk_load(uint32_t dst, const void* src, uint32_t bytes,
                                             uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// ---- tcgen05 wrappers ------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst),
               "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem descriptor], the four K=16 MMAs of a 64-k stage in one
// statement: A at a_tmem + 8 j columns, B descriptors differing in the start-address field only (32 bytes = 2 units
// per K step; the upper descriptor word is constant).  The first one overwrites
// the accumulator when `accumulate` is 0.
__device__ __forceinline__ void tc_mma_ts_x4(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_desc_lo,
                                             uint32_t b_desc_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, t;\n\t.reg .b64 d0, d1, d2, d3;\n\t.reg .b32 l1, l2, l3, a1, a2, a3;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.ne.b32 t, %4, 0;\n\t"
      "add.u32 l1, %2, 2;\n\tadd.u32 l2, %2, 4;\n\tadd.u32 l3, %2, 6;\n\t"
      "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
      "mov.b64 d0, {%2, %3};\n\tmov.b64 d1, {l1, %3};\n\tmov.b64 d2, {l2, %3};\n\tmov.b64 d3, {l3, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d0, %4, p;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], d1, %4, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], d2, %4, t;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], d3, %4, t;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_desc_lo), "r"(b_desc_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
      "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
      "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]),
      "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]),
      "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, rows of
// 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3FFFFu) >> 4);          // start address
  d |= static_cast<uint64_t>(1024u >> 4) << 32;                // stride byte offset
  d |= static_cast<uint64_t>(1) << 46;                         // descriptor version (sm_100)
  d |= static_cast<uint64_t>(2) << 61;                         // SWIZZLE_128B
  return d;
}

// Instruction descriptor: fp16 x fp16 -> fp32, both operands K-major.
__device__ __forceinline__ uint32_t make_idesc(int m, int n) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// L2 prefetch of the first weight stages of this CTA's first tile, before the results
// of the earlier kernels may be read.  With PREFETCH_SEGMENTS the segment offsets are
// those of a kernel that had completed before the one just ahead of us started; they
// are read past L1 and, should they be stale all the same, only steer the prefetch to
// other rows of the same matrix.  The first TC_PREFETCH_K columns of the tile's k part: what
// the weight ring holds and a few slots more, about what HBM delivers while the previous
// kernel drains.
constexpr int TC_PREFETCH_K = 1536;
template <int LAYOUT, int NMAT>
__device__ __forceinline__ void tc_prefetch(const CUtensorMap& tm_w0, const CUtensorMap& tm_w1, const TcArgs& args) {
  constexpr bool Q4 = LAYOUT == B200MOE_LAYOUT_Q4_K;
  int tile = blockIdx.x, e = 0, kc = 0;
  if (args.prefetch == PREFETCH_ALL_EXPERTS) {
    e = tile / (args.ntiles * args.ksplit);
    if (e >= args.E) return;
    tile -= e * args.ntiles * args.ksplit;
  } else {
    int a = __ldcg(args.seg);
    for (;; ++e) {
      if (e >= args.E) return;
      const int b = __ldcg(args.seg + e + 1);
      const int mt = b > a ? (b - a + args.tok_tile - 1) / args.tok_tile : 0;
      const int items = mt * args.ntiles * args.ksplit;
      if (tile < items) { tile /= mt; break; }
      tile -= items;
      a = b;
    }
  }
  kc = tile % args.ksplit;
  const int nt = tile / args.ksplit;
  if (nt < 0 || nt >= args.ntiles) return;
  const int k_part = args.K / args.ksplit;
  const int grow0 = e * args.N + nt * (NMAT == 2 ? args.row_tile : 2 * TC_ROWS);
  for (int k = 0; k < TC_PREFETCH_K && k < k_part; k += 128) {
    const int x = (kc * k_part + k) / (Q4 ? 2 : 1);
    tma_prefetch_2d(&tm_w0, x, grow0);
    if constexpr (NMAT == 2) tma_prefetch_2d(&tm_w1, x, grow0);
    else tma_prefetch_2d(&tm_w0, x, grow0 + TC_ROWS);
  }
}

template <int LAYOUT, int NMAT, int NMAX>
__global__ void __launch_bounds__(TC_THREADS, 1)
tc_gemm_kernel(const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_w1,
               const __grid_constant__ CUtensorMap tm_s0, const __grid_constant__ CUtensorMap tm_s1,
               const __grid_constant__ CUtensorMap tm_x16, const __grid_constant__ CUtensorMap tm_x32,
               const __grid_constant__ CUtensorMap tm_x64, const __grid_constant__ CUtensorMap tm_x96,
               const __grid_constant__ CUtensorMap tm_x128, const __grid_constant__ CUtensorMap tm_x192,
               const __grid_constant__ CUtensorMap tm_w2, const __grid_constant__ CUtensorMap tm_s2,
               const TcArgs args) {
  constexpr bool MULTI = NMAT == 3;  // q, k and v projections in one launch; tiles as in the down product
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_seg[TC_MAX_E + 1];
  __shared__ int s_prefix[TC_MAX_E + 1];
  __shared__ int s_abort;
  __shared__ uint32_t s_tmem;

  using G = TcCfg<NMAX>;
  constexpr int TC_WSLOTS = G::WSLOTS, TC_XSLOTS = G::XSLOTS, TC_XSLOT = G::XSLOT, TC_XSUB = G::XSUB, HK = G::HK, HSLOTS = G::HSLOTS;
  constexpr uint32_t TC_COL_ACC0 = G::COL_ACC0, TC_COL_ACC1 = G::COL_ACC1, TC_COL_A = G::COL_A;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t x_base = smem_base + G::OFF_X;
  const uint32_t scale_base = smem_base + G::OFF_S;
  const uint32_t bar_base = smem_base + G::OFF_BAR;
  int nb = 0;
  auto take = [&](int n) { const uint32_t b = bar_base + 8u * nb; nb += n; return b; };
  const uint32_t wfull = take(TC_WSLOTS), wempty = take(TC_WSLOTS);
  const uint32_t xfull = take(TC_XSLOTS), xempty = take(TC_XSLOTS);
  const uint32_t sfull = take(TC_SSLOTS), sempty = take(TC_SSLOTS);
  const uint32_t a_ready = take(2 * HSLOTS), a_free = take(2 * HSLOTS);  // [slot][row set]
  const uint32_t acc_full_bar = take(1), acc_empty_bar = take(1);
  const uint32_t mma_done = take(2);  // [row set]

  // the shuffle tells the compiler that the warp index is warp-uniform
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < TC_WSLOTS; ++s) {
      mbar_init(wfull + 8u * s, 1);
      mbar_init(wempty + 8u * s, HK == 2 ? TC_DQ_WARPS / 2 : TC_DQ_WARPS);  // the warps that read the slot
    }
    for (int s = 0; s < TC_XSLOTS; ++s) {
      mbar_init(xfull + 8u * s, 1);
      mbar_init(xempty + 8u * s, 2);  // both issuers commit
    }
    for (int s = 0; s < TC_SSLOTS; ++s) {
      mbar_init(sfull + 8u * s, 1);
      mbar_init(sempty + 8u * s, TC_DQ_WARPS);
    }
    for (int s = 0; s < 2 * HSLOTS; ++s) {
      mbar_init(a_ready + 8u * s, TC_DQ_WARPS / 4);  // one arrival per warp of the group and row set that fills it
      mbar_init(a_free + 8u * s, 1);
    }
    mbar_init(acc_full_bar, 2);  // both issuers commit
    mbar_init(acc_empty_bar, TC_DQ_WARPS);  // one arrival per dequant warp
    mbar_init(mma_done, 1);
    mbar_init(mma_done + 8u, 1);
    fence_mbar_init();
  }
  if (warp == TC_WARP_MMA) {
    tmem_alloc(smem_u32(&s_tmem), 512);
    tmem_relinquish();
  }
  if (NMAT != 3 && args.prefetch != PREFETCH_NONE && warp == TC_WARP_WPROD && lane == 0) tc_prefetch<LAYOUT, NMAT>(tm_w0, tm_w1, args);
  // from here on the results of earlier kernels are read
  grid_dep_wait();
  grid_dep_launch();
  if (tid == 0) {
    int run = 0;
    for (int e = 0; e < args.E; ++e) {
      const int a = args.seg[MULTI ? 0 : e], b = args.seg[MULTI ? 1 : e + 1];
      s_seg[e] = a;
      s_prefix[e] = run;
      run += ((b - a + args.tok_tile - 1) / args.tok_tile) * (MULTI ? args.mtiles[MULTI ? e : 0] : args.ntiles) * args.ksplit;
    }
    s_seg[args.E] = args.seg[MULTI ? 1 : args.E];
    s_prefix[args.E] = run;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const int total_tiles = s_prefix[args.E];
  volatile int* abort_flag = &s_abort;
  const int stages_per_tile = args.K / TC_KT / args.ksplit;  // a multiple of 4
  constexpr bool Q4 = LAYOUT == B200MOE_LAYOUT_Q4_K;
  const uint32_t set_rows = static_cast<uint32_t>(args.row_tile);
  const uint32_t WSET_BYTES = set_rows * (Q4 ? 64 : 128);  // one set, 128 k
  const uint32_t SSET_BYTES = set_rows * (Q4 ? 32 : 16);   // one set, 256 k

  // tile -> (expert, row tile | k partition << 16 | matrix << 24, first token row, token rows, MMA N)
  auto decode = [&](int tile, int& e, int& nt, int& row0, int& rows, int& ncols) {
    e = 0;
    while (tile >= s_prefix[e + 1]) ++e;
    const int local = tile - s_prefix[e];
    const int seg0 = s_seg[e], seg1 = s_seg[MULTI ? args.E : e + 1];
    const int m = seg1 - seg0;
    const int mtiles = (m + args.tok_tile - 1) / args.tok_tile;
    const int mt = local % mtiles;
    const int rest = local / mtiles;
    nt = (rest / args.ksplit) | ((rest % args.ksplit) << 16);
    if constexpr (MULTI) nt |= e << 24;
    const int per = ((m + mtiles - 1) / mtiles + 15) & ~15;  // balanced, multiple of 16
    row0 = seg0 + mt * per;
    rows = min(per, seg1 - row0);
    if (rows < 0) rows = 0;
    ncols = (max(rows, 1) + 15) & ~15;
  };

  if (warp == TC_WARP_WPROD) {
    // ------------------------------------------- TMA producer: weights + scales
    if (lane == 0) {
      uint32_t n = 0;  // global stage counter; weight slots advance every 2, scale slots every 4
      uint32_t gn = 0;  // scale slots filled
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        int e, nt, row0, rows, ncols;
        decode(tile, e, nt, row0, rows, ncols);
        const int kbase = ((nt >> 16) & 0xff) * stages_per_tile * TC_KT;
        nt &= 0xffff;
        const CUtensorMap* const mw0 = MULTI && e == 1 ? &tm_w1 : MULTI && e == 2 ? &tm_w2 : &tm_w0;
        const CUtensorMap* const ms0 = MULTI && e == 1 ? &tm_s1 : MULTI && e == 2 ? &tm_s2 : &tm_s0;
        const CUtensorMap* const mw1 = NMAT == 2 ? &tm_w1 : mw0;
        const CUtensorMap* const ms1 = NMAT == 2 ? &tm_s1 : ms0;
        const uint8_t* const st0 = MULTI ? args.mst[MULTI ? e : 0] : args.st0;
        const uint8_t* const st1 = NMAT == 2 ? args.st1 : st0;
        const long long total_rows = MULTI ? args.mrows[MULTI ? e : 0] : args.total_rows;
        const int grow0 = (MULTI ? 0 : e * args.N) + nt * (NMAT == 2 ? args.row_tile : 2 * TC_ROWS);
        const int grow1 = NMAT == 2 ? grow0 : grow0 + TC_ROWS;
        for (int st = 0; st < stages_per_tile; st += 2, n += 2) {
          const int k0 = kbase + st * TC_KT;
          if (st % TC_SGROUP == 0) {
            const int ss = gn % TC_SSLOTS;
            if (!mbar_wait(sempty + 8u * ss, ((gn / TC_SSLOTS) & 1u) ^ 1u, abort_flag, args.status)) { ok = false; break; }
            fence_proxy_async_smem();
            ++gn;
            const uint32_t sdst = scale_base + ss * TC_SSLOT;
            const uint32_t sb = sfull + 8u * ss;
            mbar_expect_tx(sb, 2 * SSET_BYTES);
            if constexpr (Q4) {
              tma_load_2d(sdst, ms0, (k0 / 32) * 4, grow0, sb);
              tma_load_2d(sdst + TC_SSET, ms1, (k0 / 32) * 4, grow1, sb);
            } else if (st0 != nullptr) {
              const long long goff = static_cast<long long>(k0 / 256) * total_rows;
              tc_bulk_load(sdst, st0 + (goff + grow0) * 16, SSET_BYTES, sb);
              tc_bulk_load(sdst + TC_SSET, st1 + (goff + grow1) * 16, SSET_BYTES, sb);
            } else {
              tma_load_2d(sdst, ms0, (k0 / 32) * 2, grow0, sb);
              tma_load_2d(sdst + TC_SSET, ms1, (k0 / 32) * 2, grow1, sb);
            }
          }
          const uint32_t wi = n >> 1;
          const int ws = wi % TC_WSLOTS;
          if (!mbar_wait(wempty + 8u * ws, ((wi / TC_WSLOTS) & 1u) ^ 1u, abort_flag, args.status)) { ok = false; break; }
          fence_proxy_async_smem();
          const uint32_t wdst = smem_base + ws * TC_WSLOT;
          const uint32_t wb = wfull + 8u * ws;
          mbar_expect_tx(wb, 2 * WSET_BYTES);
          tma_load_2d(wdst, mw0, Q4 ? k0 / 2 : k0, grow0, wb);
          tma_load_2d(wdst + TC_WSET, mw1, Q4 ? k0 / 2 : k0, grow1, wb);
        }
      }
      // do not leave while copies may still land in this CTA's shared memory
      const uint32_t wn = n >> 1;
      for (uint32_t i = wn > (uint32_t)TC_WSLOTS ? wn - TC_WSLOTS : 0; i < wn; ++i)
        mbar_drain(wfull + 8u * (i % TC_WSLOTS), (i / TC_WSLOTS) & 1u, args.status);
      for (uint32_t g = gn > (uint32_t)TC_SSLOTS ? gn - TC_SSLOTS : 0; g < gn; ++g)
        mbar_drain(sfull + 8u * (g % TC_SSLOTS), (g / TC_SSLOTS) & 1u, args.status);
    }
  } else if (warp == TC_WARP_XPROD) {
    // -------------------------------------------------- TMA producer: token tiles
    if (lane == 0) {
      uint32_t n = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        int e, nt, row0, rows, ncols;
        decode(tile, e, nt, row0, rows, ncols);
        // the per-SM TMA rate is one 128-byte box row per few clocks, whether or
        // not the row is used: take the shortest box that covers the tile
        const CUtensorMap* tx = ncols <= 16 ? &tm_x16 : ncols <= 32 ? &tm_x32 : ncols <= 64 ? &tm_x64
                              : ncols <= 96 ? &tm_x96 : ncols <= 128 ? &tm_x128 : &tm_x192;
        const uint32_t xbytes = (ncols <= 16 ? 16 : ncols <= 32 ? 32 : ncols <= 64 ? 64
                               : ncols <= 96 ? 96 : ncols <= 128 ? 128 : 192) * 128;
        for (int st = 0; st < stages_per_tile; st += 2, ++n) {  // n counts slots = pairs of stages
          const int xs = n % TC_XSLOTS;
          if (!mbar_wait(xempty + 8u * xs, ((n / TC_XSLOTS) & 1u) ^ 1u, abort_flag, args.status)) { ok = false; break; }
          const uint32_t xb = xfull + 8u * xs;
          const int x0 = (((nt >> 16) & 0xff) * stages_per_tile + st) * TC_KT * 2;
          mbar_expect_tx(xb, 2 * xbytes);
          tma_load_2d(x_base + xs * TC_XSLOT, tx, x0, row0, xb);
          tma_load_2d(x_base + xs * TC_XSLOT + TC_XSUB, tx, x0 + TC_KT * 2, row0, xb);
        }
      }
      for (uint32_t i = n > (uint32_t)TC_XSLOTS ? n - TC_XSLOTS : 0; i < n; ++i)
        mbar_drain(xfull + 8u * (i % TC_XSLOTS), (i / TC_XSLOTS) & 1u, args.status);
    }
  } else if (warp == TC_WARP_MMA || warp == TC_WARP_MMA1) {
    // ------------------------------------------ MMA issuers, one per row set
    const int mset = warp - TC_WARP_MMA;
    const uint32_t acc = tmem + (mset == 0 ? TC_COL_ACC0 : TC_COL_ACC1);
    uint32_t ti = 0;
    bool ok = true;
    uint32_t xs = 0, xph = 0, as = 0, aph = 0;
    static_assert(TC_KT == 64, "tc_mma_ts_x4 issues the four K steps of a 64-k stage");
    const uint32_t desc_hi = static_cast<uint32_t>(smem_desc_sw128(0) >> 32);
    const uint32_t a_set = tmem + TC_COL_A + mset * 32;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++ti) {
      int e, nt, row0, rows, ncols;
      decode(tile, e, nt, row0, rows, ncols);
      const uint32_t idesc = make_idesc(128, ncols);
      if (!mbar_wait_warp(acc_empty_bar, (ti & 1u) ^ 1u, abort_flag, args.status)) break;
      tc_fence_after();
      for (int st = 0; st < stages_per_tile; st += HK) {
        const uint32_t ab = 8u * (2 * as + mset);
        const uint32_t sub = static_cast<uint32_t>(st) & 1u;  // half of the token slot (tiles hold an even number of stages)
        if ((sub == 0 && !mbar_wait_warp(xfull + 8u * xs, xph, abort_flag, args.status)) ||
            !mbar_wait_warp(a_ready + ab, aph, abort_flag, args.status)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t b_lo = ((x_base + xs * TC_XSLOT + sub * TC_XSUB) & 0x3FFFFu) >> 4;
        const bool last = HK == 2 || sub == 1;  // of the token slot
        if (elect_one()) {
          tc_mma_ts_x4(acc, a_set + as * (64 * HK), b_lo, desc_hi, idesc, st > 0 ? 1u : 0u);
          if constexpr (HK == 2)
            tc_mma_ts_x4(acc, a_set + as * 128 + 64, b_lo + (TC_XSUB >> 4), desc_hi, idesc, 1u);
          tc_commit(a_free + ab);
          if (last) tc_commit(xempty + 8u * xs);
        }
        __syncwarp();
        if (last) {
          if (++xs == TC_XSLOTS) { xs = 0; xph ^= 1u; }
        }
        if (++as == HSLOTS) { as = 0; aph ^= 1u; }
      }
      if (ok && elect_one()) tc_commit(acc_full_bar);
      __syncwarp();
    }
    // after a wait that ran out nobody else waits for the last MMAs
    if (elect_one()) tc_commit(mma_done + 8u * mset);
    __syncwarp();
    mbar_drain(mma_done + 8u * mset, 0, args.status);
  } else {
    // ------------------------------------- dequantise (both sets) + epilogue
    const int grp = warp >> 3;              // stage parity this warp works on
    const int set = (warp >> 2) & 1;        // row set: 0 or 1
    const int wq = warp & 3;                // TMEM lane quarter
    const int row = wq * 32 + lane;         // weight row within the set = TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(wq * 32) << 16;
    uint32_t ti = 0;
    bool ok = true;
    // ring positions of this group's next hand-over and the parities of its waits.
    // With HK = 1 a group takes its 64-k half of every weight slot, with HK = 2 every
    // second weight slot whole; hand-over slots alternate between the groups.
    uint32_t ws = HK == 2 ? grp : 0, wph = 0, ss = 0, sph = 0, as = grp, aph = 1;

    // Drains the two accumulators of a finished tile.  Each of the four
    // (group, set) warp sets takes every fourth 16-token column chunk.
    auto epilogue = [&](int nt, int row0, int rows, int ncols, uint32_t tix) -> bool {
      if (!mbar_wait_warp(acc_full_bar, tix & 1u, abort_flag, args.status)) return false;
      tc_fence_after();
      if constexpr (NMAT == 2) {
        int col = (nt & 0xffff) * args.row_tile + row;
        if (args.out_kperm) col = (col & ~7) | ((col & 3) << 1) | ((col >> 2) & 1);
        __half* obase = static_cast<__half*>(args.out) + static_cast<size_t>(row0) * args.N + col;
        const size_t ostride = static_cast<size_t>(args.N);
        const bool silu = args.act == B200MOE_ACT_SILU;
        float amax = 0.f;
        // lanes past a short row tile hold products with whatever their slot rows held:
        // neither stored nor range-checked
        const int lane_rows = row < args.row_tile ? rows : 0;
        for (int c0 = (grp * 2 + set) * 16; c0 < ncols; c0 += 64) {
#pragma unroll 1
          for (int h8 = 0; h8 < 16; h8 += 8) {
            uint32_t g[8], u[8];
            tmem_ld8(tmem + lane_addr + TC_COL_ACC0 + c0 + h8, g);
            tmem_ld8(tmem + lane_addr + TC_COL_ACC1 + c0 + h8, u);
            tmem_wait_ld();
            __half* o = obase + static_cast<size_t>(c0 + h8) * ostride;
            const int lim = lane_rows - c0 - h8;  // token rows of the segment among these eight
            if (lim >= 8) {
              if (silu) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const float v = silu_f(__uint_as_float(g[j])) * __uint_as_float(u[j]);
                  amax = fmaxf(amax, fabsf(v));
                  o[j * ostride] = to_half_sat(v);
                }
              } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const float v = gelu_erf_f(__uint_as_float(g[j])) * __uint_as_float(u[j]);
                  amax = fmaxf(amax, fabsf(v));
                  o[j * ostride] = to_half_sat(v);
                }
              }
            } else {
              // columns past the segment are products with another expert's
              // token rows: neither stored nor range-checked
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                if (j < lim) {
                  const float gv = __uint_as_float(g[j]);
                  const float v = (silu ? silu_f(gv) : gelu_erf_f(gv)) * __uint_as_float(u[j]);
                  amax = fmaxf(amax, fabsf(v));
                  o[j * ostride] = to_half_sat(v);
                }
              }
            }
          }
        }
        if (amax >= 65520.0f) atomicOr(args.status, DEV_WARN_SATURATED);
      } else {
        const int mat = MULTI ? nt >> 24 : 0;
        const size_t ostride = static_cast<size_t>(MULTI ? args.mrows[mat] : args.N);
        float* obase = (MULTI ? args.mout[mat] : static_cast<float*>(args.out)) +
                       static_cast<size_t>((nt >> 16) & 0xff) * args.P * ostride +
                       static_cast<size_t>(row0) * ostride + (nt & 0xffff) * (2 * TC_ROWS) + row;
        if (MULTI && args.ksplit == 1) {
          void* const dst = args.mdst[mat];
          const void* const res = mat == 0 ? args.residual : nullptr;
          const size_t o0 = static_cast<size_t>(row0) * ostride + (nt & 0xffff) * (2 * TC_ROWS) + row;
          for (int c0 = (grp * 2 + set) * 16; c0 < ncols; c0 += 64) {
#pragma unroll 1
            for (int h8 = 0; h8 < 16; h8 += 8) {
              uint32_t g[8], u[8];
              const int lim = rows - c0 - h8;
              const size_t i0 = o0 + static_cast<size_t>(c0 + h8) * ostride;
              // all residuals of the chunk before the first store: the compiler may not
              // move a load above a store that could hit it, and one round trip per
              // element made the drain twice as long as the products
              float r0[8], r1[8];
              if (res != nullptr) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  r0[j] = j < lim ? tc_load_residual(res, args.mdtype, i0 + j * ostride) : 0.f;
                  r1[j] = j < lim ? tc_load_residual(res, args.mdtype, i0 + j * ostride + TC_ROWS) : 0.f;
                }
              }
              tmem_ld8(tmem + lane_addr + TC_COL_ACC0 + c0 + h8, g);
              tmem_ld8(tmem + lane_addr + TC_COL_ACC1 + c0 + h8, u);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                if (j < lim) {
                  tc_store_linear(dst, args.mdtype, res != nullptr, r0[j], i0 + j * ostride, __uint_as_float(g[j]));
                  tc_store_linear(dst, args.mdtype, res != nullptr, r1[j], i0 + j * ostride + TC_ROWS, __uint_as_float(u[j]));
                }
              }
            }
          }
        } else
        for (int c0 = (grp * 2 + set) * 16; c0 < ncols; c0 += 64) {
          uint32_t g[16], u[16];
          tmem_ld16(tmem + lane_addr + TC_COL_ACC0 + c0, g);
          tmem_ld16(tmem + lane_addr + TC_COL_ACC1 + c0, u);
          tmem_wait_ld();
          float* o = obase + static_cast<size_t>(c0) * ostride;
          const int lim = rows - c0;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (j < lim) {
              o[j * ostride] = __uint_as_float(g[j]);
              o[j * ostride + TC_ROWS] = __uint_as_float(u[j]);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty_bar);
      return true;
    };

    // The epilogue of tile t runs after this warp has handed the first stage of
    // tile t+1 to its issuer (the A ring gives each group one slot, so exactly
    // one stage can be staged ahead): the wait for tile t's last MMAs and the
    // restart of the pipeline overlap.
    bool have_prev = false;
    int p_nt = 0, p_row0 = 0, p_rows = 0, p_ncols = 0;
    uint32_t p_ti = 0;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++ti) {
      int e, nt, row0, rows, ncols;
      decode(tile, e, nt, row0, rows, ncols);
      for (int sg = 0; sg < stages_per_tile / TC_SGROUP && ok; ++sg) {
        if (!mbar_wait_warp(sfull + 8u * ss, sph, abort_flag, args.status)) { ok = false; break; }
        // scales of this group's two 64-k stages of the four: Q8_0: one word (two fp16
        // block scales) per stage; Q4_K: two (scale, min) half2 pairs per stage
        uint32_t scw[2][Q4 ? 2 : 1];
        {
          const uint32_t srow = scale_base + ss * TC_SSLOT + set * TC_SSET + row * (Q4 ? 32 : 16);
          if constexpr (Q4) {
            uint32_t lo[4], hi[4];
            lds128(srow, lo);
            lds128(srow + 16, hi);
            if constexpr (HK == 2) {
#pragma unroll
              for (int i = 0; i < 4; ++i) scw[i >> 1][i & 1] = grp ? hi[i] : lo[i];
            } else {
              scw[0][0] = grp ? lo[2] : lo[0]; scw[0][1] = grp ? lo[3] : lo[1];
              scw[1][0] = grp ? hi[2] : hi[0]; scw[1][1] = grp ? hi[3] : hi[1];
            }
          } else {
            uint32_t q[4];
            lds128(srow, q);
            scw[0][0] = grp ? q[HK] : q[0];
            scw[1][0] = grp ? q[3] : q[3 - HK];
          }
        }
        fence_proxy_async_smem();  // reads done before TMA may refill the slot
        __syncwarp();
        if (lane == 0) mbar_arrive(sempty + 8u * ss);
        if (++ss == TC_SSLOTS) { ss = 0; sph ^= 1u; }
#pragma unroll
        for (int h = 0; h < 2 / HK; ++h) {
          if (!mbar_wait_warp(wfull + 8u * ws, wph, abort_flag, args.status)) { ok = false; break; }
          // this group's 64-byte (Q4_K 32-byte) pieces of its row in the slot
          constexpr int CH = Q4 ? 2 : 4;  // 16-byte chunks per 64-k stage
          const uint32_t wrow = smem_base + ws * TC_WSLOT + set * TC_WSET + row * (Q4 ? 64 : 128);
          const int swz = Q4 ? (row >> 1) & 3 : row & 7;
          uint32_t q[HK][CH][4];
#pragma unroll
          for (int j = 0; j < HK; ++j)
#pragma unroll
            for (int c = 0; c < CH; ++c)
              lds128(wrow + ((((HK == 2 ? j : grp) * CH + c) ^ swz) << 4), q[j][c]);
          fence_proxy_async_smem();  // reads done before TMA may refill the slot
          __syncwarp();
          if (lane == 0) mbar_arrive(wempty + 8u * ws);
          ws += HK;
          if (ws >= TC_WSLOTS) { ws -= TC_WSLOTS; wph ^= 1u; }
#pragma unroll
          for (int j = 0; j < HK; ++j) {
            uint32_t v[32];
            const uint32_t(&sc)[Q4 ? 2 : 1] = scw[HK == 2 ? j : h];
            if constexpr (Q4) {
#pragma unroll
              for (int c = 0; c < 2; ++c) {
                const __half2 ds = u32_as_h2(__byte_perm(sc[c], sc[c], 0x1010));
                const __half2 dm = u32_as_h2(__byte_perm(sc[c], sc[c], 0x3232));
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  dequant_q4x8(q[j][c][i], ds, dm, *reinterpret_cast<uint32_t(*)[4]>(&v[c * 16 + i * 4]));
              }
            } else {
              const __half2 s_lo = u32_as_h2(__byte_perm(sc[0], sc[0], 0x1010));
              const __half2 s_hi = u32_as_h2(__byte_perm(sc[0], sc[0], 0x3232));
#pragma unroll
              for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  dequant_q8x4(q[j][c][i], c < 2 ? s_lo : s_hi, v[c * 8 + 2 * i], v[c * 8 + 2 * i + 1]);
            }
            if (j == 0) {
              if (!mbar_wait_warp(a_free + 8u * (2 * as + set), aph, abort_flag, args.status)) { ok = false; break; }
              tc_fence_after();
            }
            tmem_st32(tmem + lane_addr + TC_COL_A + (as * HK + j) * 64 + set * 32, v);
          }
          if (!ok) break;
          tmem_wait_st();
          tc_fence_before();
          // one arrival per warp: 256 arrivals per stage on one barrier word
          // serialise in shared memory
          __syncwarp();
          if (lane == 0) mbar_arrive(a_ready + 8u * (2 * as + set));
          as += 2;
          if (as >= HSLOTS) { as -= HSLOTS; aph ^= 1u; }
          if (h == 0 && sg == 0 && have_prev) {
            have_prev = false;
            if (!epilogue(p_nt, p_row0, p_rows, p_ncols, p_ti)) { ok = false; break; }
          }
        }
      }
      if (!ok) break;
      have_prev = true;
      p_nt = nt; p_row0 = row0; p_rows = rows; p_ncols = ncols; p_ti = ti;
    }
    if (ok && have_prev) epilogue(p_nt, p_row0, p_rows, p_ncols, p_ti);
  }


  // ---- teardown: everyone is done with tensor memory before it is freed
  tc_fence_before();
  __syncthreads();
  if (warp == TC_WARP_MMA) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <int LAYOUT, int NMAT, int NMAX>
int tc_launch_n(const CUtensorMap* maps, const TcArgs& a, cudaStream_t st) {
  auto kern = tc_gemm_kernel<LAYOUT, NMAT, NMAX>;
  using G = TcCfg<NMAX>;
  static bool configured[16] = {};
  int dev = 0;
  B200_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 16 && !configured[dev]) {
    B200_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM));
    configured[dev] = true;
  }
  B200_CHECK_CUDA(launch_dependent(kern, dim3(sm_count()), dim3(TC_THREADS), G::SMEM, st, maps[0], maps[1], maps[2], maps[3], maps[4], maps[5], maps[6], maps[7], maps[8], maps[9], maps[10], maps[11], a));
  return B200MOE_OK;
}

// The kernel variant follows the token tile: <= 64, <= 128 or <= 192 rows.
template <int LAYOUT, int NMAT>
int tc_launch(const CUtensorMap* maps, const TcArgs& a, cudaStream_t st) {
  if (a.tok_tile <= 64) return tc_launch_n<LAYOUT, NMAT, 64>(maps, a, st);
  if (a.tok_tile <= 128) return tc_launch_n<LAYOUT, NMAT, 128>(maps, a, st);
  return tc_launch_n<LAYOUT, NMAT, 192>(maps, a, st);
}

// Token tile for an expected number of rows per expert: experts with few rows
// stream their weights through the narrow, deeply buffered variants.  A
// segment longer than the tile simply takes several tiles.
int tc_pick_tok_tile(int tok_tile, int pairs, int experts) {
  const int est = pairs / (experts > 0 ? experts : 1);
  if (est <= 40) return tok_tile < 64 ? tok_tile : 64;
  if (est <= 96) return tok_tile < 128 ? tok_tile : 128;
  return tok_tile;
}

// Expected token tiles over all experts when `pairs` rows fall on them evenly:
// the row count of one expert is taken as normal with the mean's variance, and
// its tiles are 1 + the number of tile boundaries it is expected to pass.
double tc_expected_token_tiles(int pairs, int experts, int tok_tile) {
  const double mean = static_cast<double>(pairs) / (experts > 0 ? experts : 1);
  const double sd = mean > 1.0 ? sqrt(mean) : 1.0;
  double tiles = 1.0;
  int b = tok_tile;
  for (; b < mean - 6.0 * sd; b += tok_tile) tiles += 1.0;  // passed for certain
  for (; b < mean + 4.0 * sd; b += tok_tile)
    tiles += 0.5 * erfc((b + 0.5 - mean) / (1.4142135623730951 * sd));
  return tiles * (pairs < experts ? pairs : experts);
}

// Rows of each weight set per gate/up tile.  The narrow token tiles stream their
// weights, so a tile's time is its rows' bytes (+ about 8 rows' worth at the boundary)
// but no less than the dequant warps take for their 128 lanes, ~620 clocks per 64-k
// stage = the bytes of 104 Q8_0 rows, and more than any 4-bit tile's bytes.  What
// counts is the sum over the waves of SMs: eight experts of 14336 rows are 896 tiles of
// 128 rows = 7 waves for 6.05 waves of work, or 1024 tiles of 112 rows = 6.92 waves of
// shorter tiles (gate/up at 128 tokens 195 -> 167 us).  Tiles of 64 rows lose even where
// they fill the waves: Q4_K, 2 tokens, ffn 16384, 7 waves of 64 rows 181 us, the
// streaming kernel 115.
// The 192-token variant is bound by its MMAs, which always work on 128 rows.
int tc_row_tile(int rows, double token_tiles, int tok_tile, bool q4) {
  if (tok_tile > 128 || q4) return TC_ROWS;
  const int sms = sm_count();
  int best = TC_ROWS;
  double best_cost = 0.0;
  for (int r = TC_ROWS; r >= 96; r -= 16) {
    if (rows % r != 0) continue;
    const double waves = ceil(token_tiles * (rows / r) / sms);
    const double cost = waves * ((r > 104 ? r : 104) + 8);
    if (r == TC_ROWS || cost < 0.98 * best_cost) { best_cost = cost; best = r; }
  }
  return best;
}

// Token-tile tensor maps with box heights 16, 32, 64, 96, 128 and 192 (maps[4..9]).
int tc_token_maps(CUtensorMap* maps, const void* x, int pairs, uint64_t row_bytes) {
  const int heights[6] = {16, 32, 64, 96, 128, 192};
  for (int i = 0; i < 6; ++i)
    if (int rc = make_tmap_2d_sw(&maps[4 + i], x, pairs, row_bytes, heights[i], 128, 128)) return rc;
  return B200MOE_OK;
}

int tc_check(const b200moe_weight_t* w, const char* name) {
  B200_REQUIRE(w->layout == B200MOE_LAYOUT_Q8_0 || w->layout == B200MOE_LAYOUT_Q4_K,
               "tensor kernel: %s must be Q8_0 or Q4_K (layout %d)", name, w->layout);
  B200_REQUIRE(w->cols % 256 == 0, "tensor kernel: %s cols (%d) must be a multiple of 256", name,
               w->cols);
  B200_REQUIRE(w->experts >= 1 && w->experts <= TC_MAX_E, "tensor kernel: %s experts out of range", name);
  const void* sc = w->layout == B200MOE_LAYOUT_Q8_0 ? w->d : w->sub;
  B200_REQUIRE(w->qs && sc && (reinterpret_cast<uintptr_t>(w->qs) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(sc) & 15) == 0,
               "tensor kernel: %s planes missing or misaligned", name);
  return B200MOE_OK;
}

int tc_weight_map(const b200moe_weight_t* w, CUtensorMap* tw, CUtensorMap* ts, int box_rows = TC_ROWS) {
  // 128-byte wide boxes of int8 with the 128-byte swizzle: box_rows x 128 k;
  // scale boxes of 8 fp16 (256 k) x box_rows, unswizzled
  const uint64_t rows = static_cast<uint64_t>(w->experts) * w->rows;
  if (w->layout == B200MOE_LAYOUT_Q4_K) {
    // nibbles: 64-byte wide boxes (128 k), 64-byte swizzle; (scale, min) pairs: 32 bytes per row
    if (int rc = make_tmap_2d_sw(tw, w->qs, rows, w->cols / 2, box_rows, 64, 64)) return rc;
    return make_tmap_2d_sw(ts, w->sub, rows, static_cast<uint64_t>(w->cols) / 32 * 4, box_rows, 32, 0);
  }
  if (int rc = make_tmap_2d_sw(tw, w->qs, rows, w->cols, box_rows, 128, 128)) return rc;
  return make_tmap_2d_sw(ts, w->d, rows, static_cast<uint64_t>(w->cols) / 32 * 2, box_rows, 16, 0);
}

}  // namespace

// Every shape condition the launchers below check, so that the automatic regime
// choice never picks the tensor kernel for a layer only the stream kernel can
// tile.  `down` selects the down projection's row rule (two 128-row sets of
// consecutive rows per tile) instead of the gate/up one (128 rows per set).
bool tc_supported(const b200moe_weight_t* w, bool down) {
  if (!(w->layout == B200MOE_LAYOUT_Q8_0 || w->layout == B200MOE_LAYOUT_Q4_K)) return false;
  if (w->cols % 256 != 0 || w->experts < 1 || w->experts > TC_MAX_E) return false;
  return w->rows % (down ? 2 * TC_ROWS : TC_ROWS) == 0;
}

int launch_tc_gate_up(const void* xs, const int32_t* seg, int pairs, int tok_tile,
                      const b200moe_weight_t* gate, const b200moe_weight_t* up, int act,
                      int out_kperm, int prefetch, void* a_out, cudaStream_t st) {
  if (int rc = tc_check(gate, "gate")) return rc;
  if (int rc = tc_check(up, "up")) return rc;
  B200_REQUIRE(gate->rows == up->rows && gate->cols == up->cols && gate->experts == up->experts &&
                   gate->layout == up->layout,
               "tensor kernel: gate and up shapes or layouts differ");
  B200_REQUIRE(gate->rows % TC_ROWS == 0, "tensor kernel: ffn (%d) must be a multiple of 128", gate->rows);
  if (pairs == 0) return B200MOE_OK;
  TcArgs a{};
  a.tok_tile = tc_pick_tok_tile(tok_tile, pairs, gate->experts);
  a.row_tile = tc_row_tile(gate->rows, tc_expected_token_tiles(pairs, gate->experts, a.tok_tile), a.tok_tile,
                           gate->layout == B200MOE_LAYOUT_Q4_K);
  CUtensorMap maps[12] = {};
  if (int rc = tc_weight_map(gate, &maps[0], &maps[2], a.row_tile)) return rc;
  if (int rc = tc_weight_map(up, &maps[1], &maps[3], a.row_tile)) return rc;
  if (int rc = tc_token_maps(maps, xs, pairs, static_cast<uint64_t>(gate->cols) * 2)) return rc;
  a.seg = seg; a.E = gate->experts; a.N = gate->rows; a.K = gate->cols;
  a.ntiles = gate->rows / a.row_tile; a.P = pairs; a.act = act;
  a.ksplit = 1;
  a.out_kperm = out_kperm;
  a.prefetch = a.tok_tile <= 128 ? prefetch : PREFETCH_NONE;
  a.out = a_out; a.status = device_status_ptr();
  a.total_rows = static_cast<long long>(gate->experts) * gate->rows;
  if (a.status == nullptr) return B200MOE_ERR_CUDA;
  if (gate->layout == B200MOE_LAYOUT_Q4_K) return tc_launch<B200MOE_LAYOUT_Q4_K, 2>(maps, a, st);
  if (gate->sub != nullptr && up->sub != nullptr) {
    a.st0 = static_cast<const uint8_t*>(gate->sub);
    a.st1 = static_cast<const uint8_t*>(up->sub);
  }
  return tc_launch<B200MOE_LAYOUT_Q8_0, 2>(maps, a, st);
}

// Writing and reading back one row of partial sums at the copy bandwidth, in 64-k stages.
static double tc_part_cost(int rows) { return rows * 8.0 / 6.5e6 / 0.4; }

int tc_down_ksplit(const b200moe_weight_t* down, int est_pairs) {
  // The long reduction is split into up to eight partitions when that fills the
  // waves of SMs better.  Cost in 64-k stages (about 0.4 us each): waves of items,
  // each its stages and about 3 for the boundary, plus writing and reading back the
  // partial sums at the copy bandwidth.  est_pairs is the expected number of rows,
  // not a bound; the number of token tiles is its expectation (195 rows per expert
  // are 1.5 tiles of 192, not 2).
  const int stages = down->cols / TC_KT;
  const int sms = sm_count();
  const int tok = tc_pick_tok_tile(TC_NTOK, est_pairs, down->experts);
  const double tiles = tc_expected_token_tiles(est_pairs, down->experts, tok) * (down->rows / (2 * TC_ROWS));
  const double part = static_cast<double>(est_pairs) * tc_part_cost(down->rows);
  int best = 1;
  double best_cost = 0.0;
  for (int ks = 1; ks <= 8; ks *= 2) {
    if (stages % (4 * ks) != 0) break;
    const double cost = ceil(tiles * ks / sms) * (stages / ks + 3) + ks * part;
    if (ks == 1 || cost < 0.98 * best_cost) { best_cost = cost; best = ks; }
  }
  return best;
}

// A split is taken only where its partial sums cost less than the last wave can save:
// ceil(x) < x + 1 in the cost above gives (ks - 1) * part < stages + 3.
size_t tc_down_extra_rows(const b200moe_weight_t* down) {
  return static_cast<size_t>((down->cols / TC_KT + 3) / tc_part_cost(down->rows)) + 1;
}

int launch_tc_down(const void* a_in, const int32_t* seg, int pairs, int tok_tile,
                   const b200moe_weight_t* down, int ksplit, int prefetch, float* d_out, cudaStream_t st) {
  if (int rc = tc_check(down, "down")) return rc;
  B200_REQUIRE(down->rows % (2 * TC_ROWS) == 0, "tensor kernel: hidden (%d) must be a multiple of 256",
               down->rows);
  if (pairs == 0) return B200MOE_OK;
  CUtensorMap maps[12] = {};
  if (int rc = tc_weight_map(down, &maps[0], &maps[2])) return rc;
  maps[1] = maps[0];
  maps[3] = maps[2];
  if (int rc = tc_token_maps(maps, a_in, pairs, static_cast<uint64_t>(down->cols) * 2)) return rc;
  TcArgs a{};
  a.seg = seg; a.E = down->experts; a.N = down->rows; a.K = down->cols;
  B200_REQUIRE(ksplit >= 1 && (down->cols / TC_KT) % (4 * ksplit) == 0, "tensor kernel: bad k split %d",
               ksplit);
  a.row_tile = TC_ROWS;
  a.ntiles = down->rows / (2 * TC_ROWS); a.tok_tile = tc_pick_tok_tile(tok_tile, pairs, down->experts); a.P = pairs; a.act = 0;
  a.ksplit = ksplit;
  a.prefetch = a.tok_tile <= 128 ? prefetch : PREFETCH_NONE;
  a.out = d_out; a.status = device_status_ptr();
  a.total_rows = static_cast<long long>(down->experts) * down->rows;
  if (a.status == nullptr) return B200MOE_ERR_CUDA;
  if (down->layout == B200MOE_LAYOUT_Q4_K) return tc_launch<B200MOE_LAYOUT_Q4_K, 1>(maps, a, st);
  if (down->sub != nullptr) a.st0 = a.st1 = static_cast<const uint8_t*>(down->sub);
  return tc_launch<B200MOE_LAYOUT_Q8_0, 1>(maps, a, st);
}

// ---- several matrices over the same rows (dense quantised linears) -----------
namespace {
// Token tile for one matrix of `row_tiles` 256-row tiles: the row count is exact, so
// the last wave can be, too.  Cost of a wave in clocks per 64-k stage: the MMAs of the
// balanced tile (4 per token), no less than the ~620 that the dequant warps take.
// 4096 rows x 16 tiles on 148 SMs: 192-row tiles are 352 items = 3 waves of 768,
// 160-row tiles 416 items = 3 waves of 640.
int tc_linear_tok_tile(int rows, int row_tiles) {
  const int narrow = tc_pick_tok_tile(TC_NTOK, rows, 1);
  if (narrow <= 128) return narrow;
  const int sms = sm_count();
  int best = TC_NTOK;
  double best_cost = 0.0;
  for (int t = TC_NTOK; t >= 128; t -= 16) {
    const int mt = (rows + t - 1) / t;
    const int n = ((rows + mt - 1) / mt + 15) & ~15;
    const int waves = (mt * row_tiles + sms - 1) / sms;
    const double cost = waves * ((4 * n > 620 ? 4 * n : 620) + 60);
    if (t == TC_NTOK || cost < 0.98 * best_cost) { best_cost = cost; best = t; }
  }
  return best;
}
}  // namespace

// k split shared by the matrices: the cost of tc_down_ksplit with their tiles together.
int tc_linear_ksplit(const b200moe_weight_t* const* w, int count, int rows) {
  int row_tiles = 0;
  long long out_rows = 0;
  for (int i = 0; i < count; ++i) { row_tiles += w[i]->rows / (2 * TC_ROWS); out_rows += w[i]->rows; }
  const int stages = w[0]->cols / TC_KT;
  const int sms = sm_count();
  const int tok = tc_linear_tok_tile(rows, row_tiles);
  const double tiles = static_cast<double>((rows + tok - 1) / tok) * row_tiles;
  const double part = rows * tc_part_cost(static_cast<int>(out_rows));
  int best = 1;
  double best_cost = 0.0;
  for (int ks = 1; ks <= 8; ks *= 2) {
    if (stages % (4 * ks) != 0) break;
    const double cost = ceil(tiles * ks / sms) * (stages / ks + 3) + ks * part;
    if (ks == 1 || cost < 0.98 * best_cost) { best_cost = cost; best = ks; }
  }
  return best;
}

// parts[i] = fp32 [ksplit, rows, w[i]->rows] partial sums of xs w[i]^T, or, with ksplit 1,
// outs[i] = the products as out_dtype (residual added to outs[0]) and parts unused;
// equal layouts and cols.  4096 rows of a 4096-wide block, one B200, us, product +
// finish kernel -> now: q + k + v 157 + 44 -> 162, output with residual 112 + 39 -> 145.
int launch_tc_linear(const void* xs, const int32_t* seg, int rows, const b200moe_weight_t* const* w, int count,
                     int ksplit, float* const* parts, void* const* outs, int out_dtype, const void* residual,
                     cudaStream_t st) {
  B200_REQUIRE(count >= 1 && count <= 3, "tensor kernel: 1..3 matrices");
  if (rows == 0) return B200MOE_OK;
  CUtensorMap maps[12] = {};
  static constexpr int WMAP[3] = {0, 1, 10}, SMAP[3] = {2, 3, 11};
  TcArgs a{};
  int row_tiles = 0;
  bool tiled_scales = true;
  for (int i = 0; i < count; ++i) {
    if (int rc = tc_check(w[i], "linear")) return rc;
    B200_REQUIRE(w[i]->experts == 1 && w[i]->layout == w[0]->layout && w[i]->cols == w[0]->cols &&
                     w[i]->rows % (2 * TC_ROWS) == 0,
                 "tensor kernel: matrices over the same rows need one layout, equal cols and rows %% 256 == 0");
    if (int rc = tc_weight_map(w[i], &maps[WMAP[i]], &maps[SMAP[i]])) return rc;
    a.mrows[i] = w[i]->rows;
    a.mtiles[i] = w[i]->rows / (2 * TC_ROWS);
    a.mout[i] = parts[i];
    a.mdst[i] = outs[i];
    a.mst[i] = static_cast<const uint8_t*>(w[i]->sub);
    row_tiles += a.mtiles[i];
    tiled_scales = tiled_scales && w[i]->sub != nullptr;
  }
  if (w[0]->layout == B200MOE_LAYOUT_Q4_K || !tiled_scales)
    for (int i = 0; i < count; ++i) a.mst[i] = nullptr;
  if (int rc = tc_token_maps(maps, xs, rows, static_cast<uint64_t>(w[0]->cols) * 2)) return rc;
  B200_REQUIRE(ksplit >= 1 && (w[0]->cols / TC_KT) % (4 * ksplit) == 0, "tensor kernel: bad k split %d", ksplit);
  a.seg = seg; a.E = count; a.K = w[0]->cols; a.P = rows; a.ksplit = ksplit;
  a.mdtype = out_dtype; a.residual = residual;
  a.row_tile = TC_ROWS;
  a.tok_tile = tc_linear_tok_tile(rows, row_tiles);
  a.status = device_status_ptr();
  if (a.status == nullptr) return B200MOE_ERR_CUDA;
  return w[0]->layout == B200MOE_LAYOUT_Q4_K ? tc_launch<B200MOE_LAYOUT_Q4_K, 3>(maps, a, st)
                                             : tc_launch<B200MOE_LAYOUT_Q8_0, 3>(maps, a, st);
}

}  // namespace b200moe
